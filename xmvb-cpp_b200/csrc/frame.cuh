// Layout and per-pair algebra of the left-string frame, shared by the forward kernels
// (spin_frame.cu) and the gradient's (gradient_frame.cu).
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "kernels.h"

namespace vbcore {

// The (hole position x particle) grid and the 8-bit particle masks hold up to eight complement
// orbitals.  A block is laid out for fr_nbmin(K) of them (a closed shell's n - K = K fits) or, for
// more, for all eight: an open shell's minority spin has n - K > K.  On the exact path the 5
// beta electrons of a 12-orbital triplet took 1895 us of the evaluation's 2290 us; with frame tables for
// them the whole evaluation takes 528 us from records and 366 us through covalent_pairs.cu.
constexpr int kFrameMaxComplement = 8;
__host__ __device__ constexpr int fr_nbmin(int K) { return K <= 4 ? K + 4 : K; }
__host__ __device__ constexpr bool fr_wide(int n, int K) { return n - K > fr_nbmin(K); }
__host__ __device__ constexpr int fr_nb(bool wide, int K) { return wide ? kFrameMaxComplement : fr_nbmin(K); }
__host__ __device__ constexpr int fr_kfs(int K) { return 8 * K + 4; }  // 8 columns per hole position + trace block
__host__ __device__ constexpr int fr_cp(int K) { return K * (K - 1) / 2; }
__host__ __device__ constexpr int fr_bp(bool wide, int K) { return fr_nb(wide, K) * (fr_nb(wide, K) - 1) / 2; }

// Layout of one left string's block (doubles; every part starts on a 2-double boundary).
struct FrameLayout {
    int rows;    // table rows: 0 = h, 1 = two-electron linear part, 2 + m = factor column m; padded to 8
    int kfs;     // table row stride
    int o_q;     // Q[bp * CP + cp]
    int o_p;     // P[b * K + c]
    int o_rowsq; // sum_c S(o, L_c)^2 for o = L_0 .. L_{K-1}, then o = Lbar_0 .. Lbar_{NB-1}
    int o_prow2; // sum_c P(b, c)^2
    int o_scal;  // det S_LL, ||Sinv||_F^2, sum_c rowsq(L_c)
    int total;
};

__host__ __device__ inline int even_up(int x) { return (x + 1) / 2 * 2; }

__host__ __device__ inline FrameLayout frame_layout(int n, int K, int R) {
    const bool wide = fr_wide(n, K);
    FrameLayout f{};
    f.rows = (R + 2 + 7) / 8 * 8;
    f.kfs = fr_kfs(K);
    int o = f.rows * f.kfs;
    f.o_q = o;
    o += even_up(fr_bp(wide, K) * fr_cp(K));
    f.o_p = o;
    o += even_up(fr_nb(wide, K) * K);
    f.o_rowsq = o;
    o += even_up(K + fr_nb(wide, K));
    f.o_prow2 = o;
    o += even_up(fr_nb(wide, K));
    f.o_scal = o;
    o += 4;
    f.total = o;
    return f;
}

__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ uint64_t occ_mask(uint64_t w, int k) {
    uint64_t m = 0;
    for (int c = 0; c < k; ++c) m |= 1ull << ((w >> (8 * c)) & 0xFFu);
    return m;
}

// One left string's block: with its electron count at compile time, or chosen per thread.
template <int K>
struct FrameView {
    const double* blk;
    const FrameLayout& F;
    __device__ static constexpr int k() { return K; }
    __device__ static constexpr int cp() { return fr_cp(K); }
    __device__ const double* p() const { return blk + F.o_p; }
    __device__ const double* q() const { return blk + F.o_q; }
    __device__ const double* rowsq() const { return blk + F.o_rowsq; }
    __device__ const double* prow2() const { return blk + F.o_prow2; }
    __device__ const double* scal() const { return blk + F.o_scal; }
};
struct FrameViewAny {
    const double* rest;  // the block from Q on
    int kk, o_p, o_rowsq, o_prow2, o_scal;
    __device__ int k() const { return kk; }
    __device__ int cp() const { return kk * (kk - 1) / 2; }
    __device__ const double* p() const { return rest + o_p; }
    __device__ const double* q() const { return rest; }
    __device__ const double* rowsq() const { return rest + o_rowsq; }
    __device__ const double* prow2() const { return rest + o_prow2; }
    __device__ const double* scal() const { return rest + o_scal; }
};

// The certificate of kernels.h for X = P[R, :] S_LL with B^-1 = A / detb, without the division:
// ||X||_F^2 from the row norms, ||X^-1||_F <= ||S_LL^-1||_F ||P[R, :]^-1||_F and
// ||P[R, :]^-1||_F^2 <= (K - E) + ||B^-1||_F^2 (1 + sum_i ||P[p_i, :]||^2).
template <int E, class View>
__device__ __forceinline__ bool frame_certificate(const View& f, const int (&hc)[E > 0 ? E : 1],
                                                  const int (&pb)[E > 0 ? E : 1], double na2, double detb) {
    const double* scal = f.scal();
    const double* rowsq = f.rowsq();
    const double* prow2 = f.prow2();
    double nx2 = scal[2], pr = 0.0;
#pragma unroll
    for (int j = 0; j < E; ++j) {
        nx2 += rowsq[f.k() + pb[j]] - rowsq[hc[j]];
        pr += prow2[pb[j]];
    }
    const double det2 = detb * detb;
    const double lhs = nx2 * scal[1] * ((double)(f.k() - E) * det2 + na2 * (1.0 + pr));
    return isfinite(lhs) && det2 > 0.0 && lhs < kCertificate2 * det2;
}

// kappa_F(S_LL)^2 below which a left string's frame is sound.  Uncertified pairs are then still evaluated
// in it, by polynomials in the entries of B (P = S[:, L] S_LL^-1 carries 0.03 kappa eps), and the gradient
// takes the string's pairs through the reverse of its tables, which loses kappa^2 eps / 50: the adjoints are
// multiplied by S_LL^-1 more than once.  Largest error of dE/dS for two nearly dependent orbitals, relative,
// against the blocks inverted one by one (6 to 8 electrons, extended precision as the reference):
//   kappa^2 = 3e3: 2e-15 against 6e-16, 1.4e4: 2e-15 against 2e-15, 2e5: 3e-13 against 3e-14, 2e7: 1e-10
//   against 5e-13, 2e9: 4e-9 against 9e-11.
// Hydrogen chains stay below 2.3e3 (14 atoms 0.7 A apart) and near-orthogonal orbitals below 60.
constexpr double kFrameCondition2 = 1.0e4;
// Pairs of the other strings take their own inverses below this kappa_F(X)^2, which lose kappa(X)^2 eps /
// 500 (1e-13 at worst), and singular values above, which lose kappa(S_LL) eps: 4e-12 instead of 9e-11 at
// kappa(S_LL)^2 = 2e9, and 3e-14 instead of 2e-8 for graded overlaps of which two are nearly dependent.
// Singular values take 58 ns a pair at seven electrons, four times an inverse (3432 strings, of which a
// quarter holds the dependent orbitals, kappa^2 = 2e5 to 2e9: 68 to 96 ms per gradient, 47 to 51 with
// inverses up to the certificate of the forward value, 134 with inverses for all strings).
constexpr double kOwnInverseCondition2 = 1.0e6;
// Strings from here on have all their pairs differentiated through singular values.
constexpr double kSingularCondition2 = 1.0e12;

__host__ __device__ constexpr int pair_slot(int x, int y) { return x < y ? y * (y - 1) / 2 + x : x * (x - 1) / 2 + y; }
// n-th element of {0, 1, ...} without i1 < i2
__host__ __device__ constexpr int nth_other(int i1, int i2, int n) {
    int r = n;
    if (r >= i1) ++r;
    if (r >= i2) ++r;
    return r;
}

// Slots of adj B: an E <= 5 pair's 25 doubles (stride 26 spreads a tile's pairs over banks).  Higher
// levels use fewer pairs per chunk with E^2 + 1 doubles per slot in the same 32 x 26 doubles of the
// warp: 16 pairs for E = 6, 7, 8 pairs for E = 8.
constexpr int kMinorsEMax = 5;
constexpr int kCompactSlot = 26;

__host__ __device__ constexpr int compact_chunk_pairs(int e) { return e <= kMinorsEMax ? 32 : (e <= 7 ? 16 : 8); }
__host__ __device__ constexpr int compact_slot(int e) { return e <= kMinorsEMax ? kCompactSlot : e * e + 1; }

}  // namespace vbcore
