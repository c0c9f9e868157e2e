// Gradient of the spin-pair records in the left string's frame (sm_100a): the reverse of
// spin_frame.cu.  Given the adjoint of every record of one string table (adj: u-vector, determinant
// and same-spin energy, see gradient.cu), the adjoints of S, h and the factor columns.
//
// A record of the pair (L, R) at excitation level E is, with B = P[p, h], A = adj B and
// D = sign det S_LL (spin_frame.cu),
//   row r:  D [ det B tr_r + sum_ij A(j, i) Table_r(p_i, h_j) ],   det = D det B,
//   energy: rows h and 2e-linear + D sum_{I, J} Q(p_I, h_J) (-1)^(I + J) m(I^c, J^c),
// so with the record's adjoint w (a_m, and a_H for the h + linear row) and a_S of its determinant
//   f = D [ det B (a_S + tr_w) + sum_ij A(j, i) tau(p_i, h_j) + a_H quad ],
//   tau = sum_r w_r Table_r,  tr_w = sum_r w_r tr_r,
// and everything the pairs of one left string contribute collapses into adjoints of that string's
// tables:  G_Table_r += w_r D A on the grid,  G_tr_r += w_r D det B,  G_Q += a_H D (-1)^(I + J) m,
// G_P(p_i, h_j) += df / dB(i, j),  G_lndet += f.  Two kernels:
//  * frame_backward_pairs<K, MT> (persistent, K + 1 warps): per round each warp takes 32 pairs of one
//    level.  tau on the FP64 tensor cores (pairs x table rows x grid); a lane per pair runs the
//    minors of spin_frame.cu forward and backward in registers (polynomials in B: blocks of any
//    rank, no division); then G_Table = sum over the round's pairs of w (D A), again on the
//    tensor cores: warp c accumulates hole position c (and G_P there), warp K the traces, for all
//    rows in registers over the whole left string, the adjoints w staged 16 pairs at a time.
//  * frame_tables_adjoint<K>: per left string, the reverse of frame_tables back to S, h and the
//    factor columns, accumulated per CTA in shared memory; frame_adjoint_reduce sums the CTAs in a
//    fixed order.
// Uncertified pairs at levels E >= 6 (1.5 % of the pairs are at these levels at K = 7) are listed for the
// exact kernel of gradient.cu; certified ones take the inverse of B.  Strings outside kFrameCondition2 are
// listed: their pairs take the pair-by-pair kernels (all the exact one outside kSingularCondition2).  When every alpha string carries one determinant (covalent singlets) and the list is spin-flip
// symmetric, the adjoint of record (u, v) is the record of the partners' beta strings times one weight:
// the rows w are then read from the records themselves, and no adjoint buffer is built or read (2.1 GB
// at K = 7, 3.8 ms).  The pair-by-pair path takes the K x K inverse of every pair with C(K, 2)^2
// shared-memory atomics, and an SVD per thread for the uncertified ones: 14 stretched hydrogen atoms
// (5.9 M pairs, 4.9 M of them uncertified), 48.7 + 170 ms and 24 ms of contractions, against 7.0 + 1.2 ms
// here and 2.9 ms for the listed pairs.  Bound by latency: eight warps per SM (255 registers, 190 KB of
// shared memory), tables re-read from shared memory for every pair tile.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "device_algebra.cuh"
#include "frame.cuh"
#include "frame_adjoint.h"
#include "internal.h"
#include "kernels.h"
#include "pair_value.cuh"

namespace vbcore {
namespace {

// pairs whose adjoint rows are staged at a time (two stages of 8 MT doubles per pair)
constexpr int stage_pairs(int MT) { return MT <= 6 ? 32 : 16; }

// Adjoint block of one left string (doubles).
struct AdjointLayout {
    int rows;  // R + 2, in record order: row m = factor column m, row R unused, row R + 1 = h + linear
    int kfs;   // row stride: the (hole position, complement) grid, then the trace
    int o_q;   // G_Q[bp * CP + cp]
    int o_p;   // G_P[b * K + c]
    int o_f;   // sum of f; 1 when the block is valid
    int total;
};

__host__ __device__ inline AdjointLayout adjoint_layout(int n, int K, int R) {
    AdjointLayout a{};
    a.rows = R + 2;
    a.kfs = fr_kfs(K);
    int o = a.rows * a.kfs;
    a.o_q = o;
    o += even_up(fr_bp(fr_wide(n, K), K) * fr_cp(K));
    a.o_p = o;
    o += even_up(fr_nb(fr_wide(n, K), K) * K);
    a.o_f = o;
    o += 2;
    a.total = o;
    return a;
}

__device__ __forceinline__ void copy_async16(void* dst, const void* src, bool present) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(present ? 16 : 0) : "memory");
}

// One pair at level E: reads tau(j, i) from ts[j E + i], writes D A(j, i) to as[j E + i] and
// df/dB(i, j) to ts[j E + i]; adds to gq (the string's G_Q) and returns f; *dd = D det B.  s: a_S + tr_w.
template <int K, int E>
__device__ __forceinline__ double backward_minors(const double* __restrict__ blk, const FrameLayout& F, unsigned desc,
                                                  double s, double aH, double* __restrict__ ts,
                                                  double* __restrict__ as, double* __restrict__ gq, double* dd) {
    constexpr int CP = fr_cp(K);
    constexpr int EE = E > 0 ? E : 1;
    constexpr int NP = E > 1 ? E * (E - 1) / 2 : 1;
    const double D = ((desc >> 16) & 1u ? -1.0 : 1.0) * blk[F.o_scal];
    int hc[EE], pb[EE];
    {
        unsigned h = desc & 0xFFu, pm = (desc >> 8) & 0xFFu;
#pragma unroll
        for (int j = 0; j < E; ++j) {
            hc[j] = __ffs(h) - 1;
            h &= h - 1;
            pb[j] = __ffs(pm) - 1;
            pm &= pm - 1;
        }
    }
    const double* P = blk + F.o_p;
    double b[EE][EE], gb[EE][EE];
#pragma unroll
    for (int i = 0; i < E; ++i)
#pragma unroll
        for (int j = 0; j < E; ++j) {
            b[i][j] = P[pb[i] * K + hc[j]];
            gb[i][j] = 0.0;
        }
    double detb = 1.0, quad = 0.0, at = 0.0;  // at = sum A tau
    if constexpr (E == 1) {
        detb = b[0][0];
        at = ts[0];
        as[0] = D;
        gb[0][0] = s;
    }
    if constexpr (E >= 2) {
        const double* Q = blk + F.o_q;
        const double scale = aH * D;
        int cp[NP];
#pragma unroll
        for (int j2 = 1; j2 < E; ++j2)
#pragma unroll
            for (int j1 = 0; j1 < j2; ++j1) cp[pair_slot(j1, j2)] = hc[j2] * (hc[j2] - 1) / 2 + hc[j1];
        // row i of the cofactors, A(j, i) = sign sum_t +- b[r][c_t] m[{j, c_t}], and its reverse
        auto cofactor_row = [&](const double (&m)[NP], double (&gm)[NP], int i, int r, bool last) {
#pragma unroll
            for (int j = 0; j < E; ++j) {
                double acc = 0.0;
#pragma unroll
                for (int t = 0; t < E - 1; ++t) {
                    const int c = t < j ? t : t + 1;
                    const double v = b[r][c] * m[pair_slot(j, c)];
                    acc = ((E - 2 + t) & 1) ? acc - v : acc + v;
                }
                if ((i + j) & 1) acc = -acc;
                const double tau = ts[j * E + i];
                at = fma(acc, tau, at);
                as[j * E + i] = D * acc;
                double ga = tau;
                if (last) {
                    detb = j == 0 ? b[i][j] * acc : fma(b[i][j], acc, detb);
                    ga = fma(s, b[i][j], ga);
                    gb[i][j] = fma(s, acc, gb[i][j]);
                }
                if ((i + j) & 1) ga = -ga;
#pragma unroll
                for (int t = 0; t < E - 1; ++t) {
                    const int c = t < j ? t : t + 1;
                    const double x = ((E - 2 + t) & 1) ? -ga : ga;
                    gb[r][c] = fma(x, m[pair_slot(j, c)], gb[r][c]);
                    gm[pair_slot(j, c)] = fma(x, b[r][c], gm[pair_slot(j, c)]);
                }
            }
        };
#pragma unroll
        for (int i2 = 1; i2 < E; ++i2)
#pragma unroll
            for (int i1 = 0; i1 < i2; ++i1) {
                const int ra = nth_other(i1, i2, 0), rb = nth_other(i1, i2, 1), rc = nth_other(i1, i2, 2);
                double m[NP], gm[NP], m2[NP], gm2[NP];
                if constexpr (E == 2) m[0] = 1.0;
                if constexpr (E == 5) {
#pragma unroll
                    for (int y = 1; y < E; ++y)
#pragma unroll
                        for (int x = 0; x < y; ++x) {
                            m2[pair_slot(x, y)] = fma(b[ra][x], b[rb][y], -b[ra][y] * b[rb][x]);
                            gm2[pair_slot(x, y)] = 0.0;
                        }
                }
                const int qrow = (pb[i2] * (pb[i2] - 1) / 2 + pb[i1]) * CP;
                double part = 0.0;
#pragma unroll
                for (int j2 = 1; j2 < E; ++j2)
#pragma unroll
                    for (int j1 = 0; j1 < j2; ++j1) {
                        const int x = nth_other(j1, j2, 0), y = nth_other(j1, j2, 1), z = nth_other(j1, j2, 2);
                        const int q = pair_slot(j1, j2);
                        if constexpr (E == 3) m[q] = b[ra][x];
                        if constexpr (E == 4) m[q] = fma(b[ra][x], b[rb][y], -b[ra][y] * b[rb][x]);
                        if constexpr (E == 5)
                            m[q] = fma(b[rc][x], m2[pair_slot(y, z)],
                                       fma(-b[rc][y], m2[pair_slot(x, z)], b[rc][z] * m2[pair_slot(x, y)]));
                        const bool neg = (i1 + i2 + j1 + j2) & 1;
                        const double v = neg ? -m[q] : m[q];
                        const double qv = Q[qrow + cp[q]];
                        part = fma(v, qv, part);
                        gm[q] = neg ? -aH * qv : aH * qv;
                        if (aH != 0.0) atomicAdd(gq + qrow + cp[q], scale * v);
                    }
                quad += part;
                if (i2 == E - 1) {
                    cofactor_row(m, gm, i1, E - 1, false);
                    if (i1 == E - 2) cofactor_row(m, gm, E - 1, E - 2, true);
                }
                // reverse of the minors
                if constexpr (E >= 3) {
#pragma unroll
                    for (int j2 = 1; j2 < E; ++j2)
#pragma unroll
                        for (int j1 = 0; j1 < j2; ++j1) {
                            const int x = nth_other(j1, j2, 0), y = nth_other(j1, j2, 1), z = nth_other(j1, j2, 2);
                            const double g = gm[pair_slot(j1, j2)];
                            if constexpr (E == 3) gb[ra][x] += g;
                            if constexpr (E == 4) {
                                gb[ra][x] = fma(g, b[rb][y], gb[ra][x]);
                                gb[rb][y] = fma(g, b[ra][x], gb[rb][y]);
                                gb[ra][y] = fma(-g, b[rb][x], gb[ra][y]);
                                gb[rb][x] = fma(-g, b[ra][y], gb[rb][x]);
                            }
                            if constexpr (E == 5) {
                                gb[rc][x] = fma(g, m2[pair_slot(y, z)], gb[rc][x]);
                                gb[rc][y] = fma(-g, m2[pair_slot(x, z)], gb[rc][y]);
                                gb[rc][z] = fma(g, m2[pair_slot(x, y)], gb[rc][z]);
                                gm2[pair_slot(y, z)] = fma(g, b[rc][x], gm2[pair_slot(y, z)]);
                                gm2[pair_slot(x, z)] = fma(-g, b[rc][y], gm2[pair_slot(x, z)]);
                                gm2[pair_slot(x, y)] = fma(g, b[rc][z], gm2[pair_slot(x, y)]);
                            }
                        }
                }
                if constexpr (E == 5) {
#pragma unroll
                    for (int y = 1; y < E; ++y)
#pragma unroll
                        for (int x = 0; x < y; ++x) {
                            const double g = gm2[pair_slot(x, y)];
                            gb[ra][x] = fma(g, b[rb][y], gb[ra][x]);
                            gb[rb][y] = fma(g, b[ra][x], gb[rb][y]);
                            gb[ra][y] = fma(-g, b[rb][x], gb[ra][y]);
                            gb[rb][x] = fma(-g, b[ra][y], gb[rb][x]);
                        }
                }
            }
    }
#pragma unroll
    for (int i = 0; i < E; ++i)
#pragma unroll
        for (int j = 0; j < E; ++j) ts[j * E + i] = D * gb[i][j];
    *dd = D * detb;
    return D * fma(detb, s, fma(aH, quad, at));
}

// The same at levels E >= 6 through W = B^-1 (Gauss-Jordan with partial pivoting), for certified pairs;
// *ok = false for the others.  With T(i, j) = tau, q = quad / det B and N = dq / dW:
//   f = D det B c,  c = s + tr(T W) + a_H q,
//   df/dB(i, j) = D det B [ W(j, i) c - (W (T + a_H N) W)(j, i) ].
// Rare (50 of 3432 pairs per string at K = 7): out of line, with its small matrices in local memory.
template <int K, int E>
__device__ __noinline__ double backward_inverse(const double* __restrict__ blk, const FrameLayout* Fp, unsigned desc,
                                                double s, double aH, double* ts, double* as, double* __restrict__ gq,
                                                double* dd, bool* ok) {
    constexpr int CP = fr_cp(K);
    const FrameLayout& F = *Fp;
    int hc[E], pb[E], lab[E];
    {
        unsigned h = desc & 0xFFu, pm = (desc >> 8) & 0xFFu;
#pragma unroll
        for (int j = 0; j < E; ++j) {
            hc[j] = __ffs(h) - 1;
            h &= h - 1;
            pb[j] = __ffs(pm) - 1;
            pm &= pm - 1;
            lab[j] = j;
        }
    }
    const double* P = blk + F.o_p;
    double x[E][E];
#pragma unroll
    for (int i = 0; i < E; ++i)
#pragma unroll
        for (int j = 0; j < E; ++j) x[i][j] = P[pb[i] * K + hc[j]];
    double detb = 1.0;
#pragma unroll
    for (int st = 0; st < E; ++st) {
        int p = st;
        double best = fabs(x[st][st]);
#pragma unroll
        for (int i = st + 1; i < E; ++i) {
            const double av = fabs(x[i][st]);
            if (av > best) {
                best = av;
                p = i;
            }
        }
#pragma unroll
        for (int i = st + 1; i < E; ++i) {
            const bool sw = (p == i);
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const double a0 = x[st][j], a1 = x[i][j];
                x[st][j] = sw ? a1 : a0;
                x[i][j] = sw ? a0 : a1;
            }
            const int l0 = lab[st], l1 = lab[i];
            lab[st] = sw ? l1 : l0;
            lab[i] = sw ? l0 : l1;
        }
        if (p != st) detb = -detb;
        const double piv = x[st][st];
        detb *= piv;
        const double ip = 1.0 / piv;
        x[st][st] = 1.0;
#pragma unroll
        for (int j = 0; j < E; ++j) x[st][j] *= ip;
#pragma unroll
        for (int i = 0; i < E; ++i) {
            if (i == st) continue;
            const double f = x[i][st];
            x[i][st] = 0.0;
#pragma unroll
            for (int j = 0; j < E; ++j) x[i][j] = fma(-f, x[st][j], x[i][j]);
        }
    }
    double na2 = 0.0;
#pragma unroll
    for (int j = 0; j < E; ++j)
#pragma unroll
        for (int q = 0; q < E; ++q) {
            as[j * E + lab[q]] = x[j][q];  // W(j, i) at as[j E + i]
            na2 = fma(detb * x[j][q], detb * x[j][q], na2);
        }
    *ok = frame_certificate<E>(FrameView<K>{blk, F}, hc, pb, na2, detb);
    *dd = 0.0;
    if (!*ok) return 0.0;
    const double D = ((desc >> 16) & 1u ? -1.0 : 1.0) * blk[F.o_scal], scale = D * detb;
    const double* Q = blk + F.o_q;
    double M[E][E];  // T + a_H N
    double c = s, q = 0.0;
#pragma unroll 1
    for (int i = 0; i < E; ++i)
#pragma unroll 1
        for (int j = 0; j < E; ++j) {
            M[i][j] = ts[j * E + i];
            c = fma(as[j * E + i], M[i][j], c);
        }
#pragma unroll 1
    for (int i2 = 1; i2 < E; ++i2)
#pragma unroll 1
        for (int i1 = 0; i1 < i2; ++i1) {
            const int qrow = (pb[i2] * (pb[i2] - 1) / 2 + pb[i1]) * CP;
#pragma unroll 1
            for (int j2 = 1; j2 < E; ++j2)
#pragma unroll 1
                for (int j1 = 0; j1 < j2; ++j1) {
                    const int at = qrow + hc[j2] * (hc[j2] - 1) / 2 + hc[j1];
                    const double w11 = as[j1 * E + i1], w12 = as[j1 * E + i2], w21 = as[j2 * E + i1], w22 = as[j2 * E + i2];
                    const double minor = fma(w11, w22, -w12 * w21), qv = Q[at], g = aH * qv;
                    q = fma(qv, minor, q);
                    M[i1][j1] = fma(g, w22, M[i1][j1]);
                    M[i2][j2] = fma(g, w11, M[i2][j2]);
                    M[i2][j1] = fma(-g, w21, M[i2][j1]);
                    M[i1][j2] = fma(-g, w12, M[i1][j2]);
                    if (aH != 0.0) atomicAdd(gq + at, scale * aH * minor);
                }
        }
    c = fma(aH, q, c);
#pragma unroll 1
    for (int j = 0; j < E; ++j) {
        double y[E];  // row j of W M
#pragma unroll 1
        for (int b = 0; b < E; ++b) {
            double acc = 0.0;
            for (int i = 0; i < E; ++i) acc = fma(as[j * E + i], M[i][b], acc);
            y[b] = acc;
        }
#pragma unroll 1
        for (int i = 0; i < E; ++i) {
            double acc = as[j * E + i] * c;
            for (int b = 0; b < E; ++b) acc = fma(-y[b], as[b * E + i], acc);
            ts[j * E + i] = scale * acc;
        }
    }
#pragma unroll 1
    for (int i = 0; i < E * E; ++i) as[i] *= scale;
    *dd = scale;
    return scale * c;
}

template <int K>
__device__ __forceinline__ double backward_dispatch(int e, const double* blk, const FrameLayout& F, unsigned desc,
                                                    double s, double aH, double* ts, double* as, double* gq,
                                                    double* dd, bool* ok) {
    *ok = true;
#define VB_BACKWARD_CASE(E_)                                                                          \
    case E_:                                                                                          \
        if constexpr (E_ <= K) {                                                                      \
            if constexpr (E_ <= kMinorsEMax)                                                          \
                return backward_minors<K, E_>(blk, F, desc, s, aH, ts, as, gq, dd);                   \
            else                                                                                      \
                return backward_inverse<K, E_>(blk, &F, desc, s, aH, ts, as, gq, dd, ok);             \
        }                                                                                             \
        break;
    switch (e) {
        VB_BACKWARD_CASE(0)
        VB_BACKWARD_CASE(1)
        VB_BACKWARD_CASE(2)
        VB_BACKWARD_CASE(3)
        VB_BACKWARD_CASE(4)
        VB_BACKWARD_CASE(5)
        VB_BACKWARD_CASE(6)
        VB_BACKWARD_CASE(7)
        VB_BACKWARD_CASE(8)
        default: break;
    }
#undef VB_BACKWARD_CASE
    *dd = 0.0;
    return 0.0;
}

// Shared memory (doubles): table rows in record order, the rest of the block, the pairs' two slots,
// their D det B and tr_w, two stages of adjoint rows; then the pairs' record indices, maps and levels.
template <int K, int MT>
struct BackwardShape {
    static constexpr int kWarps = K + 1;
    static constexpr int kThreads = 32 * kWarps;
    static constexpr int kPairs = 32 * kWarps;  // pairs per round
    static constexpr int kLdw = 8 * MT + 4;     // = 4 mod 16: fragment loads without bank conflicts
    static constexpr int kStage = stage_pairs(MT);
    static_assert(MT % 2 == 0, "staged row stride");
    __host__ __device__ static int table_rows(int R) { return (R + 2 + 3) / 4 * 4; }
    static size_t bytes(int n, int R) {
        const FrameLayout F = frame_layout(n, K, R);
        const size_t d = (size_t)table_rows(R) * fr_kfs(K) + (F.total - F.o_q) + 2 * (size_t)kPairs * kCompactSlot +
                         2 * (size_t)kPairs + 2 * (size_t)kStage * kLdw;
        return sizeof(double) * d + (size_t)kPairs * (sizeof(long long) + 3 * sizeof(unsigned)) + kPairs;
    }
};

template <int K, int MT>
__global__ void __launch_bounds__(32 * (K + 1), 1) frame_backward_pairs(FrameAdjointArgs a) {
    using Shape = BackwardShape<K, MT>;
    constexpr int KFS = fr_kfs(K), PAIRS = Shape::kPairs, LDW = Shape::kLdw;
    extern __shared__ __align__(16) double smem[];
    const int R = a.R;
    const FrameLayout F = frame_layout(a.n, K, R);
    const AdjointLayout G = adjoint_layout(a.n, K, R);
    const int trows = Shape::table_rows(R);
    double* sTab = smem;
    double* sRest = sTab + trows * KFS;
    const double* blk = sRest - F.o_q;  // parts of the block from o_q on, at their usual offsets
    double* sW = sRest + (F.total - F.o_q);  // even offsets: the staged rows start 16-byte aligned
    double* sA = sW + 2 * Shape::kStage * LDW;
    double* sT = sA + PAIRS * kCompactSlot;
    double* sD = sT + PAIRS * kCompactSlot;
    double* sTr = sD + PAIRS;
    long long* sRec = reinterpret_cast<long long*>(sTr + PAIRS);
    unsigned* sH = reinterpret_cast<unsigned*>(sRec + PAIRS);
    unsigned* sPm = sH + PAIRS;
    unsigned* sUnion = sPm + PAIRS;  // hole positions of every four pairs
    unsigned char* sE = reinterpret_cast<unsigned char*>(sUnion + PAIRS);
    __shared__ int s_task;
    __shared__ double s_f[K + 1];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gr = lane >> 2, gc = lane & 3;
    const long long N = a.n_strings;
    const bool direct = a.weight != nullptr;
    const double* const rows = direct ? a.records : a.adj;
    const long long stride = direct ? a.rec_stride : a.adj_stride;
    const int hrow = direct ? R : R + 1;      // source row that weights the h + linear table row
    const int chunks16 = (R + 2 + 1) / 2;     // 16-byte pieces of a source row
    for (;;) {
        if (tid == 0) s_task = (int)atomicAdd(a.task_counter, 1ull);
        __syncthreads();
        const int u = s_task;
        if (u >= N) break;
        int bound[K + 2];
#pragma unroll
        for (int e = 0; e < K + 2; ++e) bound[e] = __ldg(a.ebound + (long long)u * (K + 2) + e);
        const double* src = a.tables + (long long)u * F.total;
        double* out = a.out + (long long)u * G.total;
        for (int i = tid; i < trows * KFS; i += Shape::kThreads) {
            const int r = i / KFS, c = i % KFS;
            double v = 0.0;
            if (r < R) {
                v = __ldg(src + (2 + r) * KFS + c);
                if (direct && r >= a.r_pos) v = -v;
            } else if (r == hrow) {
                v = __ldg(src + c) + __ldg(src + KFS + c);
            }
            sTab[i] = v;
        }
        for (int i = tid; i < F.total - F.o_q; i += Shape::kThreads) sRest[i] = __ldg(src + F.o_q + i);
        for (int i = tid; i < G.o_p - G.o_q; i += Shape::kThreads) out[G.o_q + i] = 0.0;
        __threadfence();
        __syncthreads();
        const long long base = record_index(u, u, N);
        const double kappa2 = blk[F.o_scal + 1] * blk[F.o_scal + 2];
        const bool sound = kappa2 < kFrameCondition2, invertible = kappa2 < kSingularCondition2;
        auto list = [&](int v) {
            const unsigned long long at = atomicAdd(a.careful_count, 1ull);
            a.careful_list[at] = ((unsigned long long)u << 32) | (unsigned long long)v;
        };
        if (!sound) {
            if (!invertible)
                for (int i = tid; i < bound[K + 1]; i += Shape::kThreads) list(__ldg(a.rlist + base + i));
            if (tid == 0) {
                out[G.o_f + 1] = 0.0;
                if (invertible) a.unsound[atomicAdd(a.unsound_count, 1ull)] = u;
            }
            __syncthreads();
            continue;
        }
        int nchunks = 0;
#pragma unroll
        for (int e = 0; e <= K; ++e) nchunks += (bound[e + 1] - bound[e] + compact_chunk_pairs(e) - 1) / compact_chunk_pairs(e);
        const double weight_u = direct ? __ldg(a.weight + u) : 0.0;
        const int partner_u = direct ? __ldg(a.partner + u) : 0;
        double acc[MT][2];
#pragma unroll
        for (int m = 0; m < MT; ++m) acc[m][0] = acc[m][1] = 0.0;
        double gp = 0.0, fsum = 0.0;
        for (int c0 = 0; c0 < nchunks; c0 += Shape::kWarps) {
            // ---- a lane per pair -------------------------------------------------------------
            int e = 0, start = 0, cnt = 0, left = c0 + warp;
#pragma unroll
            for (int ee = K; ee >= 0; --ee) {
                const int cs = compact_chunk_pairs(ee), c = (bound[ee + 1] - bound[ee] + cs - 1) / cs;
                if (left >= 0 && left < c) {
                    e = ee;
                    start = bound[ee] + cs * left;
                    cnt = min(cs, bound[ee + 1] - start);
                }
                left -= c;
            }
            const bool valid = lane < cnt;
            const int pair0 = 32 * warp, pair = pair0 + lane;
            const unsigned desc = valid ? __ldg(a.rdesc + base + start + lane) : 0u;
            const int v = valid ? __ldg(a.rlist + base + start + lane) : u;
            // source row of the pair's adjoint and its weight
            long long rec = -1;
            double omega = 1.0;
            if (valid && direct) {
                const int partner = __ldg(a.partner + v);
                rec = record_index(min(partner_u, partner), max(partner_u, partner), N);
                omega = (v == u ? 2.0 : 4.0) * weight_u * __ldg(a.weight + v);
            } else if (valid) {
                rec = record_index(u, v, N);
            }
            const int slot = compact_slot(e);
            double* const as = sA + pair0 * kCompactSlot + lane * slot;
            double* const ts = sT + pair0 * kCompactSlot + lane * slot;
            unsigned hmap = 0xFFFFFFFFu, pmap = 0xFFFFFFFFu;
            {
                unsigned h = desc & 0xFFu, p = (desc >> 8) & 0xFFu;
                for (unsigned j = 0; h; ++j) {
                    hmap &= ~((0xFu ^ j) << (4 * (__ffs(h) - 1)));
                    pmap &= ~((0xFu ^ j) << (4 * (__ffs(p) - 1)));
                    h &= h - 1;
                    p &= p - 1;
                }
            }
            unsigned un = desc & 0xFFu;
            un |= __shfl_xor_sync(0xffffffffu, un, 1);
            un |= __shfl_xor_sync(0xffffffffu, un, 2);
            sRec[pair] = rec;
            sH[pair] = hmap;
            sPm[pair] = pmap;
            sE[pair] = (unsigned char)e;
            if ((lane & 3) == 0) sUnion[pair >> 2] = un;
            double aS = 0.0, aH = 0.0;
            if (valid) {
                aS = __ldg(rows + rec * stride + R);
                aH = __ldg(rows + rec * stride + R + 1);
                if (direct) {  // a record holds the determinant, then the energy
                    const double sb = aS;
                    aS = omega * fma(-a.lambda, sb, aH);
                    aH = omega * sb;
                }
            }
            // tau and tr_w, one 8-pair tile at a time; the loads of a tile's rows (48 at a time) are all
            // in flight together, the first ones issued while the tile before is multiplied
            const int tiles = (cnt + 7) / 8;
            constexpr int kBatch = 12;
            double wv[kBatch];
            auto load_rows = [&](int mt, int r0) {
                const long long rg = __shfl_sync(0xffffffffu, rec, (8 * mt + gr) & 31);
                const double* w = rows + (rg < 0 ? 0 : rg) * stride + r0 + gc;
#pragma unroll
                for (int q = 0; q < kBatch; ++q)
                    wv[q] = (rg >= 0 && r0 + 4 * q + gc < R + 2) ? __ldg(w + 4 * q) : 0.0;
            };
            if (tiles > 0) load_rows(0, 0);
#pragma unroll 1
            for (int mt = 0; mt < tiles; ++mt) {
                const int owner = 8 * mt + gr;
                const double omega_g = __shfl_sync(0xffffffffu, omega, owner);
                const unsigned hmap_g = __shfl_sync(0xffffffffu, hmap, owner);
                const unsigned pmap_g = __shfl_sync(0xffffffffu, pmap, owner);
                const unsigned uh = __reduce_or_sync(0xffffffffu, (lane >> 3) == mt ? (desc & 0xFFu) : 0u);
                double t[K][2], tr = 0.0;
#pragma unroll
                for (int c = 0; c < K; ++c) t[c][0] = t[c][1] = 0.0;
#pragma unroll 1
                for (int r0 = 0; r0 < trows; r0 += 4 * kBatch) {
                    double wc[kBatch];
#pragma unroll
                    for (int q = 0; q < kBatch; ++q) wc[q] = wv[q];
                    if (r0 + 4 * kBatch < trows)
                        load_rows(mt, r0 + 4 * kBatch);
                    else if (mt + 1 < tiles)
                        load_rows(mt + 1, 0);
#pragma unroll
                    for (int q = 0; q < kBatch; ++q) {
                        if (r0 + 4 * q >= trows) break;
                        const double* row = sTab + (r0 + 4 * q + gc) * KFS;
                        tr = fma(wc[q], row[8 * K], tr);
#pragma unroll
                        for (int c = 0; c < K; ++c)
                            if ((uh >> c) & 1u) mma_f64(t[c], wc[q], row[8 * c + gr]);
                    }
                }
                tr += __shfl_xor_sync(0xffffffffu, tr, 1);
                tr += __shfl_xor_sync(0xffffffffu, tr, 2);
                if (gc == 0) sTr[pair0 + owner] = omega_g * tr;
                double* to = sT + pair0 * kCompactSlot + owner * slot;
#pragma unroll
                for (int c = 0; c < K; ++c) {
                    const unsigned jh = (hmap_g >> (4 * c)) & 0xFu;
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        const unsigned ip = (pmap_g >> (4 * (2 * gc + x))) & 0xFu;
                        if (jh < (unsigned)e && ip < (unsigned)e) to[jh * e + ip] = omega_g * t[c][x];
                    }
                }
            }
            __syncwarp();
            double dd = 0.0;
            if (valid) {
                bool ok;
                fsum += backward_dispatch<K>(e, blk, F, desc, aS + sTr[pair], aH, ts, as, out + G.o_q, &dd, &ok);
                if (!ok) {
                    list(v);
                    sH[pair] = 0xFFFFFFFFu;  // no hole: the pair adds nothing below
                }
                if (direct && ok) {
                    // the staged rows are records: their weight goes with D adj B
                    for (int i = 0; i < e * e; ++i) as[i] *= omega;
                    dd *= omega;
                }
            }
            sD[pair] = dd;
            __syncthreads();
            // ---- adjoints of the tables ------------------------------------------------------
            const int used = min(PAIRS, 32 * (nchunks - c0));  // pairs of the warps that have a chunk
            auto stage = [&](int p0, int buf) {
                for (int i = tid; i < Shape::kStage * chunks16; i += Shape::kThreads) {
                    const int p = i / chunks16, q = i % chunks16;
                    const long long r = sRec[p0 + p];
                    copy_async16(sW + (buf * Shape::kStage + p) * LDW + 2 * q, rows + (r < 0 ? 0 : r) * stride + 2 * q, r >= 0);
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
            };
            stage(0, 0);
            for (int p0 = 0; p0 < used; p0 += Shape::kStage) {
                const int buf = (p0 / Shape::kStage) & 1;
                if (p0 + Shape::kStage < used) {
                    stage(p0 + Shape::kStage, buf ^ 1);
                    asm volatile("cp.async.wait_group 1;" ::: "memory");
                } else {
                    asm volatile("cp.async.wait_group 0;" ::: "memory");
                }
                __syncthreads();
                const double* w = sW + buf * Shape::kStage * LDW;
#pragma unroll
                for (int g4 = 0; g4 < Shape::kStage / 4; ++g4) {
                    const int p = p0 + 4 * g4 + gc;
                    double y = 0.0;
                    if (warp < K) {
                        if (!((sUnion[(p0 >> 2) + g4] >> warp) & 1u)) continue;  // no pair of the four has this hole
                        const unsigned le = sE[p];
                        const unsigned jh = (sH[p] >> (4 * warp)) & 0xFu, ip = (sPm[p] >> (4 * gr)) & 0xFu;
                        if (jh < le && ip < le) {
                            const int at = (p & ~31) * kCompactSlot + (p & 31) * compact_slot(le) + jh * le + ip;
                            y = sA[at];
                            gp += sT[at];
                        }
                    } else {
                        y = gr == 0 ? sD[p] : 0.0;
                    }
                    const double* wr = w + (4 * g4 + gc) * LDW + gr;
#pragma unroll
                    for (int m = 0; m < MT; ++m) mma_f64(acc[m], wr[8 * m], y);
                }
                __syncthreads();
            }
        }
        // ---- the string's adjoint block --------------------------------------------------------
        const int nb = a.n - K;
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const int q = 8 * m + gr, c = 2 * gc + x;
                if (q >= R + 2) continue;
                // block rows are in adjoint order: a record's determinant and energy are the other way round
                const int r = direct && q >= R ? 2 * R + 1 - q : q;
                const double v = direct && q < R && q >= a.r_pos ? -acc[m][x] : acc[m][x];
                if (warp < K)
                    out[r * KFS + 8 * warp + c] = v;
                else if (c == 0)
                    out[r * KFS + 8 * K] = v;
            }
        gp += __shfl_xor_sync(0xffffffffu, gp, 1);
        gp += __shfl_xor_sync(0xffffffffu, gp, 2);
        if (warp < K && gc == 0 && gr < nb) out[G.o_p + gr * K + warp] = gp;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) fsum += __shfl_xor_sync(0xffffffffu, fsum, o);
        if (lane == 0) s_f[warp] = fsum;
        __syncthreads();
        if (tid == 0) {
            double f = 0.0;
            for (int w = 0; w < Shape::kWarps; ++w) f += s_f[w];
            out[G.o_f] = f;
            out[G.o_f + 1] = 1.0;
        }
        __syncthreads();
    }
}

// ---- tables -> S, h, factor columns ---------------------------------------------------------------

constexpr int kAdjThreads = 256;
constexpr int kAdjSources = kAdjThreads / 64;  // sources handled at once, 64 threads (8 x 8) each
constexpr int kPad = 72;                       // 8 x 9: a staged 8 x 8 matrix

__host__ __device__ inline size_t tables_adjoint_doubles(int n, int np, int R) {
    // quadratic adjoint (64 x 64), six 8 x 8 matrices per source, S_LL^-1, P, G_lin, G_P, Acc, then the
    // CTA's sums: factor columns (np x R), S and h adjoints (n x n)
    return 64 * 64 + 6 * kAdjSources * kPad + 5 * kPad + (size_t)np * R + 2 * (size_t)n * n;
}

template <int K>
__global__ void __launch_bounds__(kAdjThreads) frame_tables_adjoint(FrameAdjointArgs a) {
    constexpr int KFS = fr_kfs(K), CP = fr_cp(K);
    extern __shared__ __align__(16) double smem[];
    const int n = a.n, R = a.R, np = n * (n + 1) / 2, nb = n - K;
    const FrameLayout F = frame_layout(n, K, R);
    const AdjointLayout G = adjoint_layout(n, K, R);
    double* sM = smem;  // [e'][e], symmetric
    double* sMat = sM + 64 * 64;
    double* sInv = sMat + 6 * kAdjSources * kPad;
    double* sP = sInv + kPad;
    double* sLin = sP + kPad;
    double* sGP = sLin + kPad;
    double* sAcc = sGP + kPad;
    double* gL = sAcc + kPad;  // [pair][m]
    double* gS = gL + (size_t)np * R;
    double* gh = gS + n * n;
    __shared__ int sL[8], sLb[8];
    __shared__ double sG[K][2 * K], sF[K];
    __shared__ double sDot[kAdjSources][2];
    const int tid = threadIdx.x, q = tid >> 6, e = tid & 63, r = e >> 3, c = e & 7, lane = tid & 31;
    double* zl = sMat + (6 * q + 0) * kPad;
    double* zb = sMat + (6 * q + 1) * kPad;  // Z rows of the complement, then Y there
    double* yl = sMat + (6 * q + 2) * kPad;
    double* vt = sMat + (6 * q + 3) * kPad;
    double* gv = sMat + (6 * q + 4) * kPad;
    double* gy = sMat + (6 * q + 5) * kPad;
    const int at = r * 9 + c;
    for (size_t i = tid; i < (size_t)np * R + 2 * (size_t)n * n; i += kAdjThreads) gL[i] = 0.0;
    for (long long u = blockIdx.x; u < a.n_strings; u += gridDim.x) {
        const double* tab = a.tables + u * F.total;
        const double* adj = a.out + u * G.total;
        if (adj[G.o_f + 1] == 0.0) continue;  // uniform: the string is not in the frame form
        __syncthreads();
        if (tid < 8) {
            const uint64_t w0 = __ldg(a.occ + 2 * u);
            sL[tid] = tid < K ? (int)((w0 >> (8 * tid)) & 0xFFu) : -1;
            const uint64_t mask = occ_mask(w0, K);
            int o = -1, seen = 0;
            for (int i = 0; i < n; ++i)
                if (!((mask >> i) & 1) && seen++ == tid) o = i;
            sLb[tid] = o;
        }
        if (tid < 64) {
            sInv[at] = 0.0;
            sP[at] = (r < nb && c < K) ? __ldg(tab + F.o_p + r * K + c) : 0.0;
            sLin[at] = (r < nb && c < K) ? adj[(R + 1) * KFS + c * 8 + r] : 0.0;
            sGP[at] = (r < nb && c < K) ? adj[G.o_p + r * K + c] : 0.0;
        }
        for (int i = tid; i < 64 * 64; i += kAdjThreads) {
            const int x = i >> 6, y = i & 63, b1 = x >> 3, c1 = x & 7, b2 = y >> 3, c2 = y & 7;
            double v = 0.0;
            if (b1 != b2 && c1 != c2 && b1 < nb && b2 < nb && c1 < K && c2 < K) {
                v = __ldcg(adj + G.o_q + pair_slot(b1, b2) * CP + pair_slot(c1, c2));
                if ((b1 < b2) != (c1 < c2)) v = -v;
            }
            sM[i] = v;
        }
        __syncthreads();
        if (tid < 32) {  // S_LL^-1 (Gauss-Jordan, as in frame_tables)
            for (int i = lane; i < K * 2 * K; i += 32) {
                const int rr = i / (2 * K), cc = i % (2 * K);
                sG[rr][cc] = cc < K ? __ldg(a.S + sL[rr] * n + sL[cc]) : (cc - K == rr ? 1.0 : 0.0);
            }
            __syncwarp();
            for (int st = 0; st < K; ++st) {
                const double inv = 1.0 / sG[st][st];
                if (lane < K) sF[lane] = sG[lane][st];
                __syncwarp();
                for (int cc = lane; cc < 2 * K; cc += 32) sG[st][cc] *= inv;
                __syncwarp();
                for (int i = lane; i < K * 2 * K; i += 32) {
                    const int rr = i / (2 * K), cc = i % (2 * K);
                    if (rr != st) sG[rr][cc] = fma(-sF[rr], sG[st][cc], sG[rr][cc]);
                }
                __syncwarp();
            }
            for (int i = lane; i < K * K; i += 32) sInv[(i / K) * 9 + i % K] = sG[i / K][K + i % K];
        }
        double gpart = 0.0, accp = 0.0;  // this thread's sums of G_P(r, c) and Acc(r, c)
        const double ge = adj[(R + 1) * KFS + 8 * K];
        const int iL = sL[r], iB = sLb[r], jL = sL[c];
        const long long pl = (iL >= 0 && jL >= 0) ? dev::pair_index(iL, jL) : -1;
        const long long pbx = (iB >= 0 && jL >= 0 && r < nb) ? dev::pair_index(iB, jL) : -1;
        for (int s0 = 0; s0 < R + 1; s0 += kAdjSources) {
            // source s: 0 = h, 1 + m = factor column m
            const int s = s0 + q;
            const bool on = s < R + 1;
            const double sg = (!on || s == 0) ? 0.0 : ((s - 1) < a.r_pos ? 1.0 : -1.0);
            const int row = s == 0 ? R + 1 : s - 1;
            double xl = 0.0, xb = 0.0, gt = 0.0, gtr = 0.0;
            if (on) {
                if (pl >= 0) xl = s == 0 ? __ldg(a.h + iL * n + jL) : __ldg(a.lf + pl * a.ld + (s - 1));
                if (pbx >= 0) xb = s == 0 ? __ldg(a.h + iB * n + jL) : __ldg(a.lf + pbx * a.ld + (s - 1));
                if (r < nb && c < K) gt = adj[row * KFS + c * 8 + r];
                gtr = adj[row * KFS + 8 * K];
            }
            __syncthreads();  // the previous sources' matrices are consumed
            zl[at] = xl;
            zb[at] = xb;
            __syncthreads();
            double y0 = 0.0, y1 = 0.0;
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                y0 = fma(zl[r * 9 + t], sInv[t * 9 + c], y0);
                y1 = fma(zb[r * 9 + t], sInv[t * 9 + c], y1);
            }
            __syncthreads();
            yl[at] = y0;
            zb[at] = y1;
            __syncthreads();
            double v = y1, tr = 0.0;
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                v = fma(-sP[r * 9 + t], yl[t * 9 + c], v);
                tr += yl[t * 9 + t];
            }
            vt[at] = v;
            double dot = sLin[at] * v;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
            if (lane == 0) sDot[q][(tid >> 5) & 1] = dot;
            __syncthreads();
            // adjoint of Vt
            double g = tr * sLin[at];
#pragma unroll
            for (int t = 0; t < 8; ++t) g = fma(-sLin[r * 9 + t], yl[c * 9 + t], g);
            double quad = 0.0;
            if (s > 0)
#pragma unroll 8
                for (int x = 0; x < 64; ++x) quad = fma(sM[x * 64 + e], vt[(x >> 3) * 9 + (x & 7)], quad);
            g = fma(sg, g + quad, gt);
            gv[at] = g;
            __syncthreads();
            // adjoint of YL, G_P
            double y = 0.0, lin = 0.0, gp = 0.0;
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                y = fma(-sP[t * 9 + r], gv[t * 9 + c], y);
                lin = fma(vt[t * 9 + r], sLin[t * 9 + c], lin);
                gp = fma(gv[r * 9 + t], yl[c * 9 + t], gp);
            }
            y = fma(-sg, fma(ge, yl[c * 9 + r], lin), y);
            if (r == c) y += fma(sg, fma(ge, tr, sDot[q][0] + sDot[q][1]), gtr);
            gpart -= gp;
            gy[at] = y;
            __syncthreads();
            double ax = 0.0, g0 = 0.0, g1 = 0.0, gb = 0.0;
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                ax = fma(yl[t * 9 + r], gy[t * 9 + c], ax);
                ax = fma(zb[t * 9 + r], gv[t * 9 + c], ax);
                g0 = fma(gy[r * 9 + t], sInv[t * 9 + c], g0);
                g1 = fma(gy[c * 9 + t], sInv[t * 9 + r], g1);
                gb = fma(gv[r * 9 + t], sInv[t * 9 + c], gb);
            }
            accp += ax;
            if (on) {
                if (s == 0) {
                    if (pl >= 0) gh[iL * n + jL] += g0;
                    if (pbx >= 0) gh[iB * n + jL] += gb;
                } else {
                    // entries (r, c) and (c, r) of the symmetric part share a packed pair
                    if (pl >= 0 && r <= c) gL[pl * R + (s - 1)] += r == c ? g0 : g0 + g1;
                    if (pbx >= 0) gL[pbx * R + (s - 1)] += gb;
                }
            }
        }
        // sums over the sources' thread groups, then S
        __syncthreads();
        sMat[q * kPad + at] = gpart;
        sMat[(kAdjSources + q) * kPad + at] = accp;
        __syncthreads();
        if (tid < 64) {
            double x = sGP[at], y = 0.0;
#pragma unroll
            for (int w = 0; w < kAdjSources; ++w) {
                x += sMat[w * kPad + at];
                y += sMat[(kAdjSources + w) * kPad + at];
            }
            sGP[at] = x;
            sAcc[at] = y;
        }
        __syncthreads();
        double acc = 0.0;
        if (tid < 64) {
            acc = sAcc[at];
#pragma unroll
            for (int t = 0; t < 8; ++t) acc = fma(sP[t * 9 + r], sGP[t * 9 + c], acc);
        }
        __syncthreads();
        if (tid < 64) sAcc[at] = acc;
        __syncthreads();
        if (tid < 64) {
            double x = adj[G.o_f] * sInv[at], y = 0.0;
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                x = fma(-sAcc[r * 9 + t], sInv[t * 9 + c], x);
                y = fma(sGP[r * 9 + t], sInv[t * 9 + c], y);
            }
            if (pl >= 0) gS[iL * n + jL] += x;
            if (pbx >= 0) gS[iB * n + jL] += y;
        }
    }
    __syncthreads();
    double* part = a.partial + (size_t)blockIdx.x * ((size_t)np * R + 2 * (size_t)n * n);
    for (size_t i = tid; i < (size_t)np * R + 2 * (size_t)n * n; i += kAdjThreads) part[i] = gL[i];
}

// gL[q ld + m], gS and gh += the CTAs' sums, in CTA order.
__global__ void frame_adjoint_reduce(const double* __restrict__ partial, int parts, int n, int np, int R, int ld,
                                     double* __restrict__ gL, double* __restrict__ gS, double* __restrict__ gh) {
    const int size = np * R + 2 * n * n;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < size; i += gridDim.x * blockDim.x) {
        double acc = 0.0;
#pragma unroll 8
        for (int b = 0; b < parts; ++b) acc += __ldg(partial + (size_t)b * size + i);
        if (i < np * R)
            gL[(size_t)(i / R) * ld + i % R] += acc;
        else if (i < np * R + n * n)
            gS[i - np * R] += acc;
        else
            gh[i - np * R - n * n] += acc;
    }
}

// M tiles of the table adjoint: 8 MT >= R + 2 (6: R <= 46; 14: R <= 110, K = 6 and 7 only; 18: R <= 142)
template <int K>
int m_tiles(int R) {
    if (R + 2 <= 48) return 6;
    if ((K == 6 || K == 7) && R + 2 <= 112) return 14;
    return R + 2 <= 144 ? 18 : 0;
}

constexpr size_t kSmemLimit = 224 * 1024;

template <int K>
bool supported(int n, int R) {
    const int mt = m_tiles<K>(R);
    if (mt == 0 || R < 1) return false;
    size_t pairs = mt == 6 ? BackwardShape<K, 6>::bytes(n, R) : BackwardShape<K, 18>::bytes(n, R);
    if constexpr (K == 6 || K == 7)
        if (mt == 14) pairs = BackwardShape<K, 14>::bytes(n, R);
    return pairs <= kSmemLimit && sizeof(double) * tables_adjoint_doubles(n, n * (n + 1) / 2, R) <= kSmemLimit;
}

template <int K, int MT>
cudaError_t launch_pairs(const FrameAdjointArgs& a, int sms, cudaStream_t s) {
    const size_t smem = BackwardShape<K, MT>::bytes(a.n, a.R);
    const auto kernel = frame_backward_pairs<K, MT>;
    cudaError_t err = allow_dynamic_smem((const void*)kernel, smem);
    int per_sm = 1;
    if (err == cudaSuccess)
        err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, BackwardShape<K, MT>::kThreads, smem);
    if (err != cudaSuccess) return err;
    const int grid = (int)(a.n_strings < (long long)sms * per_sm ? a.n_strings : (long long)sms * (per_sm > 0 ? per_sm : 1));
    kernel<<<grid, BackwardShape<K, MT>::kThreads, smem, s>>>(a);
    return cudaGetLastError();
}

template <int K>
cudaError_t launch(const FrameAdjointArgs& a, cudaStream_t s) {
    int dev = 0, sms = 148;
    cudaError_t err = cudaGetDevice(&dev);
    if (err == cudaSuccess) err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (err != cudaSuccess) return err;
    switch (m_tiles<K>(a.R)) {
        case 6: err = launch_pairs<K, 6>(a, sms, s); break;
        case 14:
            if constexpr (K == 6 || K == 7) err = launch_pairs<K, 14>(a, sms, s);
            break;
        case 18: err = launch_pairs<K, 18>(a, sms, s); break;
        default: return cudaErrorInvalidValue;
    }
    if (err != cudaSuccess) return err;
    const int np = a.n * (a.n + 1) / 2;
    const size_t smem = sizeof(double) * tables_adjoint_doubles(a.n, np, a.R);
    err = allow_dynamic_smem((const void*)frame_tables_adjoint<K>, smem);
    if (err != cudaSuccess) return err;
    const int grid = a.n_strings < kAdjointMaxParts ? a.n_strings : kAdjointMaxParts;
    frame_tables_adjoint<K><<<grid, kAdjThreads, smem, s>>>(a);
    err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    const int size = np * a.R + 2 * a.n * a.n;
    frame_adjoint_reduce<<<(size + 127) / 128, 128, 0, s>>>(a.partial, grid, a.n, np, a.R, a.ld, a.gL, a.gS, a.gh);
    return cudaGetLastError();
}

}  // namespace

size_t frame_adjoint_block_doubles(int n, int k, int R) { return (size_t)adjoint_layout(n, k, R).total; }

bool frame_adjoint_supported(int n, int k, int R) {
    if (!frame_spin_supported(n, k, R)) return false;
    switch (k) {
        case 1: return supported<1>(n, R);
        case 2: return supported<2>(n, R);
        case 3: return supported<3>(n, R);
        case 4: return supported<4>(n, R);
        case 5: return supported<5>(n, R);
        case 6: return supported<6>(n, R);
        case 7: return supported<7>(n, R);
        case 8: return supported<8>(n, R);
        default: return false;
    }
}

cudaError_t launch_frame_adjoint(const FrameAdjointArgs& a, cudaStream_t s) {
    switch (a.k) {
        case 1: return launch<1>(a, s);
        case 2: return launch<2>(a, s);
        case 3: return launch<3>(a, s);
        case 4: return launch<4>(a, s);
        case 5: return launch<5>(a, s);
        case 6: return launch<6>(a, s);
        case 7: return launch<7>(a, s);
        case 8: return launch<8>(a, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace vbcore
