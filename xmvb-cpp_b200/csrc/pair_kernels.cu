// Determinant-pair kernels for sm_100a.
//
//  * prepare_tables: the unpacked pair kernel K[p][q] = (p|q) over packed orbital pairs and the
//    antisymmetrized same-spin table Gamma[(i<k)][(j<l)] = (ij|kl) - (il|kj) used by the
//    same-spin two-electron sum (hamiltonian.cpp:83-123 sums exactly these differences).
//  * factor_pair_registers, factor_pair_kernel: pivoted LDL^T of the pair kernel, K = sum_m sigma_m l_m l_m^T.
//  * the register-resident spin-pair path lives in spin_frame.cu (left-string frame kernels); a
//    block is accepted there only under the conditioning certificate (kCertificate2): then the
//    last pivot of a complete-pivoting LU is at least 1 / ||X^{-1}||_F and the first at most
//    ||X||_F, so their ratio stays far above 1e-12 and the reference's FullPivLU would also find
//    full rank (overlap.cpp:60-71).  Other blocks are evaluated there by polynomials at excitation levels
//    up to 5 when the left string's frame is sound, or appended to a list for the exact kernel.
//  * spin_pairs_exact<KM>: complete-pivoting LU / Jacobi SVD with the reference semantics
//    (device_algebra.cuh) for listed blocks, one thread per block, local arrays bounded by KM.
//  * determinant pairs of covalent lists: covalent_pairs.cu, without records.
//  * full_pairs_kernel: one thread per determinant pair (d <= e) of a band of columns:
//    S = S_a S_b, H = H_a S_b + H_b S_a + sum_m sigma_m u_a[m] u_b[m] (evaluator.cpp:95-148,
//    354-384 with the opposite-spin term in factored form), folded over the spin-flip orbit.
//  * block_pairs_kernel: the same for lists ordered by blocks of alpha x beta strings, as products of
//    the blocks' records on the FP64 tensor cores.
#include <cuda_runtime.h>
#include <limits.h>
#include <math.h>

#include <algorithm>
#include <stdint.h>

#include <string>

#include "autotune.h"
#include "device_algebra.cuh"
#include "frame.cuh"
#include "internal.h"
#include "kernels.h"
#include "pair_value.cuh"

namespace vbcore {
namespace {

constexpr double kThreshold = 1.0e-12;
// Relative pivot cut of the pair-kernel factorization.  Once the numerical rank is exhausted the
// Schur complement holds rounding noise of about (steps) * eps * max|K_pp|, so a cut of 8 np eps
// (at least 1e-15) ends the factorization there instead of emitting columns of noise.
double factor_tolerance(int np) { return fmax(1.0e-15, 8.0 * np * 2.220446049250313e-16); }
constexpr int kSms = 148;

__device__ __forceinline__ int occ_byte(const uint64_t* row, int i) {
    const uint64_t w = row[i >> 3];
    return (int)((w >> (8 * (i & 7))) & 0xFFu);
}

__global__ void prepare_tables_kernel(int n, const double* __restrict__ eri, double* __restrict__ gamma,
                                      double* __restrict__ kfull) {
    const int np = n * (n + 1) / 2;
    const int gd = n * (n - 1) / 2;
    const long long total_k = (long long)np * np;
    const long long total_g = (long long)gd * gd;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total_k + total_g; t += stride) {
        if (t < total_k) {
            const long long p = t / np, q = t % np;
            const long long hi = p > q ? p : q, lo = p > q ? q : p;
            kfull[t] = eri[hi * (hi + 1) / 2 + lo];
        } else {
            const long long g = t - total_k;
            const int row = (int)(g / gd), col = (int)(g % gd);
            // row = anti_index(i, kk) with i < kk; col = anti_index(j, l) with j < l
            int kk = (int)floor((1.0 + sqrt(1.0 + 8.0 * row)) * 0.5);
            while (kk * (kk - 1) / 2 > row) --kk;
            while ((kk + 1) * kk / 2 <= row) ++kk;
            const int i = row - kk * (kk - 1) / 2;
            int l = (int)floor((1.0 + sqrt(1.0 + 8.0 * col)) * 0.5);
            while (l * (l - 1) / 2 > col) --l;
            while ((l + 1) * l / 2 <= col) ++l;
            const int j = col - l * (l - 1) / 2;
            gamma[g] = dev::eri_packed(eri, i, j, kk, l) - dev::eri_packed(eri, i, l, kk, j);
        }
    }
}

// Pivoted LDL^T of the unpacked pair kernel with diagonal (complete) pivoting, K = sum_m sigma_m l_m l_m^T.
// Stops when the largest remaining |diagonal| falls to rel_tol times the largest initial one; the dropped
// remainder then perturbs any opposite-spin energy by at most rel_tol * max|K_pp| * ||p_a||_1 ||p_b||_1.
// Columns are emitted positive-sign first.
//
// factor_pair_registers (np <= 32 B): one CTA of W warps, right-looking, the Schur complement in
// registers: entry (i, j) with i = W a + warp and j = 32 b + lane in s[a][b].  Per pivot the warp that
// owns row p scales it into shared memory, one barrier, and every thread updates its entries.  Each warp
// keeps all diagonals (dg[b], updated from the same row) and finds the next pivot by itself, by integer
// reductions over the high and low words of |diagonal|: no second barrier and no published maxima.  Bound
// by the chain pivot search - rsqrt - row - barrier - update, one per factor column: 24 us for 36 columns
// of 78 rows (n = 12) and 10 us for 18 of 21 (n = 6).  The left-looking form below, which gathers m products
// per row, publishes warp maxima and compares them in every thread, took 66 us at n = 12, and a one-warp
// form that read K from global memory in every step 22 us at n = 6.
template <int W, int B>
__global__ void __launch_bounds__(32 * W) factor_pair_registers(int np, const double* __restrict__ kfull,
                                                                int* __restrict__ signs, double* __restrict__ lf, int ld,
                                                                int* __restrict__ meta, double rel_tol) {
    constexpr int A = 32 * B / W;
    extern __shared__ double L[];  // column m of the factor at L[m np ..]
    __shared__ double s_row[2][32 * B];
    __shared__ int s_sign[32 * B], s_slot[32 * B];
    const unsigned full = 0xffffffffu;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    double s[A][B], dg[B];
    unsigned used = 0;  // bit b: row 32 b + lane is a pivot already (or past the end)
#pragma unroll
    for (int a = 0; a < A; ++a)
#pragma unroll
        for (int b = 0; b < B; ++b) {
            const int i = W * a + warp, j = 32 * b + lane;
            s[a][b] = i < np && j < np ? __ldg(kfull + (long long)i * np + j) : 0.0;
        }
#pragma unroll
    for (int b = 0; b < B; ++b) {
        const int j = 32 * b + lane;
        dg[b] = j < np ? __ldg(kfull + (long long)j * np + j) : 0.0;
        if (j >= np) used |= 1u << b;
    }
    // largest |diagonal| of the rows left, the smallest index on ties; *p = -1 when there is none
    auto search = [&](int* p, double* piv) {
        double best = -1.0, bd = 0.0;
        int bi = INT_MAX;
#pragma unroll
        for (int b = 0; b < B; ++b)
            if (!((used >> b) & 1u) && fabs(dg[b]) > best) {
                best = fabs(dg[b]);
                bd = dg[b];
                bi = 32 * b + lane;
            }
        // every lane takes part in every reduction
        bool in = bi != INT_MAX;
        const unsigned hi = in ? (unsigned)__double2hiint(best) : 0u;
        const unsigned top = __reduce_max_sync(full, hi);
        in = in && hi == top;
        const unsigned lo = in ? (unsigned)__double2loint(best) : 0u;
        const unsigned low = __reduce_max_sync(full, lo);
        in = in && lo == low;
        const int at = __reduce_min_sync(full, in ? bi : INT_MAX);
        *piv = __shfl_sync(full, bd, at & 31);
        *p = at == INT_MAX ? -1 : at;
    };
    int p;
    double piv;
    search(&p, &piv);
    const double cut = rel_tol * fabs(piv);
    int m = 0;
    for (; m < np; ++m) {
        if (p < 0 || !(fabs(piv) > cut) || piv == 0.0) break;
        const double inv = rsqrt(fabs(piv));
        const double sgn = piv > 0.0 ? 1.0 : -1.0;
        double* row = s_row[m & 1];
        if (warp == p % W) {
            const int ap = p / W;
#pragma unroll
            for (int b = 0; b < B; ++b) {
                double v = 0.0;
#pragma unroll
                for (int a = 0; a < A; ++a) v = a == ap ? s[a][b] : v;
                v = (used >> b) & 1u ? 0.0 : v * inv;
                const int j = 32 * b + lane;
                row[j] = v;
                if (j < np) L[m * np + j] = v;
            }
        }
        if (lane == (p & 31)) used |= 1u << (p >> 5);
        if (tid == 0) {
            s_sign[m] = (int)sgn;
            signs[m] = (int)sgn;
        }
        __syncthreads();
        double lj[B];
#pragma unroll
        for (int b = 0; b < B; ++b) {
            lj[b] = row[32 * b + lane];
            dg[b] = fma(-sgn * lj[b], lj[b], dg[b]);
        }
#pragma unroll
        for (int a = 0; a < A; ++a) {
            const double li = -sgn * row[W * a + warp];
#pragma unroll
            for (int b = 0; b < B; ++b) s[a][b] = fma(li, lj[b], s[a][b]);
        }
        search(&p, &piv);
    }
    // slots: the columns with positive sign first
    if (warp == 0) {
        int pos = 0;
        for (int c0 = 0; c0 < m; c0 += 32) pos += __popc(__ballot_sync(full, c0 + lane < m && s_sign[c0 + lane] > 0));
        int ip = 0, in = pos;
        for (int c0 = 0; c0 < m; c0 += 32) {
            const bool here = c0 + lane < m, plus = here && s_sign[c0 + lane] > 0;
            const unsigned bp = __ballot_sync(full, plus), bn = __ballot_sync(full, here && !plus);
            const unsigned below = (1u << lane) - 1u;
            if (here) s_slot[plus ? ip + __popc(bp & below) : in + __popc(bn & below)] = c0 + lane;
            ip += __popc(bp);
            in += __popc(bn);
        }
        if (lane == 0) {
            meta[0] = pos;
            meta[1] = m - pos;
        }
    }
    __syncthreads();
    for (int q = warp; q < np; q += W)
        for (int slot = lane; slot < ld; slot += 32)
            lf[(long long)q * ld + slot] = slot < m ? L[s_slot[slot] * np + q] : 0.0;
}

// Larger pair kernels, one CTA, left-looking.  Thread t owns rows t, t + nt, ... (at most kFactorRows) and
// keeps their diagonal in registers.  Step m: with the pivot p and its value known, every owned row forms
// its entry of the Schur-complement column, K[i, p] - sum_{m' < m} sigma_m' l_m'[p] l_m'[i], scales it
// into l_m[i] and updates its diagonal; each warp then reduces its rows' largest |diagonal| and
// one barrier publishes the warp results, from which every thread picks the next pivot.
// The columns l_m (l_m[i] at [m np + i]) live in `cols`.  `work_g` is not used.
constexpr int kFactorRows = 4;

__global__ void __launch_bounds__(1024) factor_pair_kernel(int np, const double* __restrict__ kfull,
                                                           double* __restrict__ work_g, double* __restrict__ cols,
                                                           int* __restrict__ signs, double* __restrict__ lf, int ld,
                                                           int* __restrict__ meta, double rel_tol) {
    (void)work_g;
    extern __shared__ double fsm[];
    double* sig = fsm;                                        // np
    int* slot_col = reinterpret_cast<int*>(sig + np);         // np (+1 pad)
    const double* K = kfull;
    double* L = cols;
    __shared__ double red_v[2][32], red_d[2][32];
    __shared__ int red_i[2][32];
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarps = nt >> 5;
    double dg[kFactorRows];
    bool used[kFactorRows];
#pragma unroll
    for (int r = 0; r < kFactorRows; ++r) {
        const int i = tid + r * nt;
        dg[r] = i < np ? __ldg(kfull + (long long)i * np + i) : 0.0;
        used[r] = i >= np;
    }
    // publishes this thread's best unused row to the warp slots of buffer b (largest |diagonal|,
    // smallest index on ties)
    auto publish = [&](int b) {
        double best = -1.0, bd = 0.0;
        int bi = -1;
#pragma unroll
        for (int r = 0; r < kFactorRows; ++r)
            if (!used[r] && fabs(dg[r]) > best) {
                best = fabs(dg[r]);
                bd = dg[r];
                bi = tid + r * nt;
            }
        for (int o = 16; o > 0; o >>= 1) {
            const double ov = __shfl_xor_sync(0xffffffffu, best, o);
            const double od = __shfl_xor_sync(0xffffffffu, bd, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi >= 0 && (bi < 0 || oi < bi))) {
                best = ov;
                bd = od;
                bi = oi;
            }
        }
        if (lane == 0) {
            red_v[b][warp] = best;
            red_d[b][warp] = bd;
            red_i[b][warp] = bi;
        }
    };
    auto pick = [&](int b, int* p, double* piv) {
        double best = -1.0, bd = 0.0;
        int bi = -1;
        for (int w = 0; w < nwarps; ++w) {
            const double ov = red_v[b][w];
            const int oi = red_i[b][w];
            if (ov > best || (ov == best && oi >= 0 && (bi < 0 || oi < bi))) {
                best = ov;
                bd = red_d[b][w];
                bi = oi;
            }
        }
        *p = bi;
        *piv = bd;
    };
    publish(0);
    __syncthreads();
    int p;
    double piv;
    pick(0, &p, &piv);
    const double cut = rel_tol * fmax(fabs(piv), 0.0);
    int m = 0;
    for (; m < np; ++m) {
        if (p < 0 || !(fabs(piv) > cut) || piv == 0.0) break;
        const double inv = rsqrt(fabs(piv));
        const double sgn = piv > 0.0 ? 1.0 : -1.0;
        double* lm = L + (long long)m * np;
#pragma unroll
        for (int r = 0; r < kFactorRows; ++r) {
            const int i = tid + r * nt;
            if (i >= np) continue;
            double v = 0.0;
            if (!used[r]) {
                double acc0 = K[(long long)p * np + i], acc1 = 0.0, acc2 = 0.0, acc3 = 0.0;
                int q = 0;
                for (; q + 3 < m; q += 4) {
                    const double* l0 = L + (long long)q * np;
                    acc0 = fma(-sig[q] * l0[p], l0[i], acc0);
                    acc1 = fma(-sig[q + 1] * l0[np + p], l0[np + i], acc1);
                    acc2 = fma(-sig[q + 2] * l0[2 * np + p], l0[2 * np + i], acc2);
                    acc3 = fma(-sig[q + 3] * l0[3 * np + p], l0[3 * np + i], acc3);
                }
                for (; q < m; ++q) acc0 = fma(-sig[q] * L[(long long)q * np + p], L[(long long)q * np + i], acc0);
                v = ((acc0 + acc1) + (acc2 + acc3)) * inv;
                if (i == p)
                    used[r] = true;
                else
                    dg[r] = fma(-sgn * v, v, dg[r]);
            }
            lm[i] = v;
        }
        if (tid == 0) {
            sig[m] = sgn;
            signs[m] = (int)sgn;
        }
        publish((m + 1) & 1);
        __syncthreads();
        pick((m + 1) & 1, &p, &piv);
    }
    if (tid == 0) {
        int pos = 0;
        for (int c = 0; c < m; ++c) pos += sig[c] > 0.0 ? 1 : 0;
        int ip = 0, in = pos;
        for (int c = 0; c < m; ++c) slot_col[sig[c] > 0.0 ? ip++ : in++] = c;
        meta[0] = pos;
        meta[1] = m - pos;
    }
    __syncthreads();
    for (int q = warp; q < np; q += nwarps)
        for (int slot = lane; slot < ld; slot += 32)
            lf[(long long)q * ld + slot] = slot < m ? L[(long long)slot_col[slot] * np + q] : 0.0;
}

// Listed blocks (or all blocks): one thread per block resolves it by the exact path; its first
// cofactors A go to the lane's shared slot (k^2 doubles).  The warp then treats its 32 blocks one
// at a time: the u-vectors of the records with the factor columns split over lanes, and, for
// full-rank blocks with k > 3, the regular two-electron sum (A11 A22 - A12 A21) / det
// (hamiltonian.cpp:83-123) with its C(k,2)^2 terms split over lanes, which keeps a block's
// latency short when only a few blocks are listed.  Rank-deficient blocks and k <= 3 are summed
// by their own thread: nullity 1 in the expanded form of the wedge second cofactors
//   parity prod sv * sum_{s<k-1} (u_s ^ u_n)(v_s ^ v_n) / sv_s            (contractions.cpp:937-963)
//   = Y(r1,c1) zu(r2) zv(c2) - Y(r1,c2) zu(r2) zv(c1) - Y(r2,c1) zu(r1) zv(c2) + Y(r2,c2) zu(r1) zv(c1),
// Y = parity sum_{s<k-1} u_s v_s^T prod_{l<k-1, l != s} sv_l; nullity 2 and k <= 3 by
// second_cofactor; nullity >= 3 is zero.  Dynamic shared memory: 32 k^2 doubles per warp.
template <int KM, int KC>  // KC > 0: electrons per string fixed at compile time (== KM)
__global__ void __launch_bounds__(64) spin_pairs_exact(SpinTableArgs a) {
    extern __shared__ double slots[];
    const long long count = a.all_careful ? a.n_pairs : (long long)(*a.careful_count);
    const int lane = threadIdx.x & 31;
    const int k = KC > 0 ? KC : a.k, kk = k * k, gd = a.gamma_dim;
    const int cp = k * (k - 1) / 2;
    double* wslot = slots + (size_t)(threadIdx.x >> 5) * 32 * kk;
    double* cof = wslot + (size_t)lane * kk;
    const long long N = a.n_strings;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    // blocks per warp: 32 (one per lane) when there are enough, fewer so that a short list
    // spreads over as many warps as it has blocks
    long long chunk = (count + nwarps - 1) / nwarps;
    chunk = chunk < 1 ? 1 : (chunk > 32 ? 32 : chunk);
    for (long long base = warp * chunk; base < count; base += nwarps * chunk) {
        const long long idx = base + lane;
        long long u = 0, v = 0;
        const bool valid = lane < chunk && idx < count;
        double det = 0.0, h1 = 0.0, h2 = 0.0;
        int nullity = 3;
        bool regular = false;  // two-electron sum done by the warp
        if (valid) {
            if (a.all_careful) {
                const double b = 2.0 * (double)N + 1.0;
                long long uu = (long long)floor((b - sqrt(fmax(b * b - 8.0 * (double)idx, 0.0))) * 0.5);
                if (uu < 0) uu = 0;
                if (uu > N - 1) uu = N - 1;
                while (uu > 0 && uu * N - uu * (uu - 1) / 2 > idx) --uu;
                while (uu + 1 < N && (uu + 1) * N - (uu + 1) * uu / 2 <= idx) ++uu;
                u = uu;
                v = u + (idx - (u * N - u * (u - 1) / 2));
            } else {
                const unsigned long long w = a.careful_list[idx];
                u = (long long)(w >> 32);
                v = (long long)(w & 0xffffffffull);
            }
            int L[KM], R[KM];
            for (int c = 0; c < k; ++c) {
                L[c] = occ_byte(a.occ + 2 * u, c);
                R[c] = occ_byte(a.occ + 2 * v, c);
            }
            double x[KM * KM];
            for (int c = 0; c < k; ++c)
                for (int r = 0; r < k; ++r) x[c * k + r] = __ldg(a.S + R[r] * a.n + L[c]);
            dev::ResolutionT<KM> res;
            dev::resolve_exact<KM>(k, x, kThreshold, &res);
            dev::first_cofactor<KM>(res, cof);
            det = res.det;
            nullity = res.nullity;
            regular = res.nullity == 0 && k > 3;
            if (res.nullity < 3) {
                if (res.nullity <= 1)
                    for (int c = 0; c < k; ++c)
                        for (int r = 0; r < k; ++r) h1 = fma(__ldg(a.h + L[c] * a.n + R[r]), cof[c * k + r], h1);
                if (!regular) {
                    const bool rank1 = res.nullity == 1 && k > 3;
                    double Y[KM * KM], zu[KM], zv[KM];
                    if (rank1) {
                        const int ni = k - 1;
                        double w[KM];
                        for (int s2 = 0; s2 < ni; ++s2) {
                            double p = res.parity;
                            for (int l = 0; l < ni; ++l)
                                if (l != s2) p *= res.sv[l];
                            w[s2] = p;
                        }
                        for (int r = 0; r < k; ++r) {
                            zu[r] = res.u[ni * k + r];
                            zv[r] = res.v[ni * k + r];
                            for (int c = 0; c < k; ++c) {
                                double acc = 0.0;
                                for (int s2 = 0; s2 < ni; ++s2) acc = fma(res.u[s2 * k + r] * w[s2], res.v[s2 * k + c], acc);
                                Y[r * k + c] = acc;
                            }
                        }
                    }
                    for (int r2 = 1; r2 < k; ++r2)
                        for (int r1 = 0; r1 < r2; ++r1) {
                            const double* grow = a.gamma + (long long)dev::anti_index(R[r1], R[r2]) * gd;
                            double part = 0.0;
                            for (int c2 = 1; c2 < k; ++c2)
                                for (int c1 = 0; c1 < c2; ++c1) {
                                    const double g = __ldg(grow + dev::anti_index(L[c1], L[c2]));
                                    const double m2 = rank1 ? Y[r1 * k + c1] * zu[r2] * zv[c2] - Y[r1 * k + c2] * zu[r2] * zv[c1] -
                                                                  Y[r2 * k + c1] * zu[r1] * zv[c2] + Y[r2 * k + c2] * zu[r1] * zv[c1]
                                                            : dev::second_cofactor<KM>(res, r1, r2, c1, c2);
                                    part = fma(g, m2, part);
                                }
                            h2 += part;
                        }
                }
            }
            if (res.nullity > 1)
                for (int i = 0; i < kk; ++i) cof[i] = 0.0;
        }
        __syncwarp();
        for (int j = 0; j < chunk; ++j) {
            const long long jdx = base + j;
            if (jdx >= count) break;
            const long long uj = __shfl_sync(0xffffffffu, u, j), vj = __shfl_sync(0xffffffffu, v, j);
            const uint64_t* ol = a.occ + 2 * uj;
            const uint64_t* orr = a.occ + 2 * vj;
            const double* cj = wslot + (size_t)j * kk;
            // regular two-electron sum of block j, terms split over lanes: gamma[(R r1, R r2)][(L c1, L c2)]
            // is (r1 c1 | r2 c2) - (r1 c2 | r2 c1)
            if (__shfl_sync(0xffffffffu, (int)regular, j)) {
                double part = 0.0;
                if constexpr (KC > 0) {
                    // k fixed: every lane's terms unrolled, occupations from registers, loads batched
                    constexpr int CPK = KC * (KC - 1) / 2;
                    constexpr int PER = (CPK * CPK + 31) / 32;
                    const uint64_t wl = __ldg(ol), wr = __ldg(orr);
#pragma unroll 2
                    for (int t = 0; t < PER; ++t) {
                        const int q = lane + 32 * t;
                        if (q < CPK * CPK) {
                            const int rp = q / CPK, cq = q % CPK;
                            int r2 = 1;
                            while ((r2 + 1) * r2 / 2 <= rp) ++r2;
                            const int r1 = rp - r2 * (r2 - 1) / 2;
                            int c2 = 1;
                            while ((c2 + 1) * c2 / 2 <= cq) ++c2;
                            const int c1 = cq - c2 * (c2 - 1) / 2;
                            const int R1 = (int)((wr >> (8 * r1)) & 0xFFu), R2 = (int)((wr >> (8 * r2)) & 0xFFu);
                            const int L1 = (int)((wl >> (8 * c1)) & 0xFFu), L2 = (int)((wl >> (8 * c2)) & 0xFFu);
                            const double g = __ldg(a.gamma + (long long)dev::anti_index(R1, R2) * gd + dev::anti_index(L1, L2));
                            part = fma(g, cj[c1 * KC + r1] * cj[c2 * KC + r2] - cj[c2 * KC + r1] * cj[c1 * KC + r2], part);
                        }
                    }
                } else {
                    for (int q = lane; q < cp * cp; q += 32) {
                        const int rp = q / cp, cq = q % cp;
                        int r2 = 1;
                        while ((r2 + 1) * r2 / 2 <= rp) ++r2;
                        const int r1 = rp - r2 * (r2 - 1) / 2;
                        int c2 = 1;
                        while ((c2 + 1) * c2 / 2 <= cq) ++c2;
                        const int c1 = cq - c2 * (c2 - 1) / 2;
                        const double g = __ldg(a.gamma + (long long)dev::anti_index(occ_byte(orr, r1), occ_byte(orr, r2)) * gd +
                                               dev::anti_index(occ_byte(ol, c1), occ_byte(ol, c2)));
                        part = fma(g, cj[c1 * k + r1] * cj[c2 * k + r2] - cj[c2 * k + r1] * cj[c1 * k + r2], part);
                    }
                }
                for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
                if (lane == j) h2 = part / det;
            }
            // u-vectors: u_m = sum_{c,r} A(r,c) l_m[pair(R_r, L_c)]
            double* rec = a.records + record_index(uj, vj, N) * (long long)a.rec_stride;
            if constexpr (KC > 0) {
                // k fixed: the k^2 factor-row loads of a column issued together
                const uint64_t wl = __ldg(ol), wr = __ldg(orr);
                for (int m = lane; m < a.R; m += 32) {
                    double acc = 0.0;
#pragma unroll 1
                    for (int c = 0; c < KC; ++c) {
                        const int lc = (int)((wl >> (8 * c)) & 0xFFu);
                        double v[KC];
#pragma unroll
                        for (int r = 0; r < KC; ++r)
                            v[r] = __ldg(a.lf + (long long)dev::pair_index((int)((wr >> (8 * r)) & 0xFFu), lc) * a.ld + m);
#pragma unroll
                        for (int r = 0; r < KC; ++r) acc = fma(cj[c * KC + r], v[r], acc);
                    }
                    rec[m] = acc;
                }
            } else {
                for (int m = lane; m < a.R; m += 32) {
                    double acc = 0.0;
                    for (int c = 0; c < k; ++c) {
                        const int lc = occ_byte(ol, c);
                        for (int r = 0; r < k; ++r) {
                            const double cv = cj[c * k + r];
                            if (cv != 0.0)
                                acc = fma(cv, __ldg(a.lf + (long long)dev::pair_index(occ_byte(orr, r), lc) * a.ld + m),
                                          acc);
                        }
                    }
                    rec[m] = acc;
                }
            }
        }
        if (valid) {
            double* rec = a.records + record_index(u, v, N) * (long long)a.rec_stride;
            rec[a.R + 0] = det;
            rec[a.R + 1] = nullity < 3 ? h1 + h2 : 0.0;
            rec[a.R + 2] = nullity < 3 ? h1 : 0.0;
            rec[a.R + 3] = (double)nullity;
        }
        __syncwarp();
    }
}

__device__ __forceinline__ void band_decode(long long t, long long e0, long long e1, long long* d, long long* e) {
    const long long B = e1 - e0;
    const long long rect = e0 * B;
    if (t < rect) {
        *d = t / B;
        *e = e0 + t % B;
        return;
    }
    const long long tp = t - rect;
    const double b2 = 2.0 * (double)B + 1.0;
    long long i = (long long)floor((b2 - sqrt(fmax(b2 * b2 - 8.0 * (double)tp, 0.0))) * 0.5);
    if (i < 0) i = 0;
    if (i > B - 1) i = B - 1;
    while (i > 0 && i * B - i * (i - 1) / 2 > tp) --i;
    while (i + 1 < B && (i + 1) * B - (i + 1) * i / 2 <= tp) ++i;
    *d = e0 + i;
    *e = *d + (tp - (i * B - i * (i - 1) / 2));
}

// Weight of the upper-triangle pair (d <= e) in H_d = U' + U'^T: 1/2 on the diagonal, and,
// with a spin-flip permutation, the unordered pairs {d, e} and {flip d, flip e} (same H_de and,
// for structures whose coefficients are flip-invariant, the same coefficient products) fold
// onto one representative with twice the weight; the other member gets weight 0.
__device__ __forceinline__ double pair_weight(const int* flip, long long d, long long e) {
    const double w = (d == e) ? 0.5 : 1.0;
    if (!flip) return w;
    const long long fd = __ldg(flip + d), fe = __ldg(flip + e);
    const long long d2 = fd < fe ? fd : fe, e2 = fd < fe ? fe : fd;
    if (d < d2 || (d == d2 && e < e2)) return 2.0 * w;
    if (d == d2 && e == e2) return w;
    return 0.0;
}

__global__ void __launch_bounds__(512) full_pairs_kernel(FullPairArgs a) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < a.n_items; t += stride) {
        long long d, e;
        band_decode(t, a.e0, a.e1, &d, &e);
        const double w = pair_weight(a.flip, d, e);
        double H = 0.0, S = 0.0;
        if (w != 0.0) {
            pair_value(a, d, e, &H, &S);
            H *= w;
            S *= w;
        }
        const long long o = d * a.ldb + (e - a.e0);
        a.Hb[o] = H;
        a.Sb[o] = S;
    }
}

// Determinant pairs by blocks (BlockPairArgs): one CTA per block pair (g <= h).  With the alpha records
// of the string pairs (i, j), i in g and j in h, as rows and the beta records of (k, l) as columns,
//   H[(i, k), (j, l)] = sum_m sigma_m u_a[ij][m] u_b[kl][m] + H_a[ij] S_b[kl] + S_a[ij] H_b[kl]
// is one (up to 64) x (up to 64) x (R + 2) product on the FP64 tensor cores, and S the outer product of
// the determinants: every record is read once per block pair and used by 7 x 7 determinant pairs (n =
// 12, singly ionic), where one thread per pair gathers two records (640 bytes) for R multiply-adds.
// The records arrive by cp.async, all in flight together (a warp per record, one after the other, left
// the loads' latency exposed: 35 ms).  Each of the eight warps owns M tiles w and w + 4 (w = 0 .. 3) and
// half of the N tiles; H goes through shared memory so that band rows are written in runs of a block's determinants.  Both
// members of a spin-flip orbit are evaluated: blocks do not map to blocks under the flip.  Bound by the
// product (1.7 ms at the tensor cores' rate for 34,188 determinants) and the band it writes (9.3 GB, 1.4 ms);
// takes 8.7 to 9.0 ms there (10.7 with record addresses and determinant cells divided out per element, four
// warps and four barriers), the gather form 27.3 ms.  A block pair is 2.4 us of loads, products and stores
// one after the other on 3 CTAs per SM; a second record buffer with one CTA per SM: 11.7 ms.
constexpr int kBlockWarps = 8;
constexpr int kBlockEdge = 8;                        // strings per block and spin
constexpr int kBlockCells = kBlockEdge * kBlockEdge;

__host__ __device__ inline int block_k(int R) { return (R + 2 + 3) / 4 * 4; }
// record stride in shared memory: 4 or 12 mod 16 doubles (conflict-free fragment loads)
__host__ __device__ inline int block_ld(int R) { return block_k(R) % 8 == 4 ? block_k(R) : block_k(R) + 4; }
__host__ __device__ inline int block_rows(int rows) { return (rows + 7) / 8 * 8; }
inline size_t block_pairs_smem(int rows_a, int rows_b, int dets, int R) {
    return sizeof(double) * ((size_t)(block_rows(rows_a) + block_rows(rows_b)) * block_ld(R) + (size_t)dets * (dets + 1));
}

__global__ void __launch_bounds__(32 * kBlockWarps, 3) block_pairs_kernel(BlockPairArgs a) {
    extern __shared__ __align__(16) double bsm[];
    const int R = a.f.R, KD = block_k(R), LD = block_ld(R), r_pos = a.f.r_pos;
    double* sA = bsm;                                    // [ij][record]
    double* sB = sA + block_rows(a.max_a) * LD;          // [kl][record]
    double* sH = sB + block_rows(a.max_b) * LD;          // [determinant of g][determinant of h]
    const int OUT = a.max_dets + 1;
    __shared__ __align__(16) BlockStrings s_desc[2][2];
    __shared__ unsigned char s_i[2][kBlockCells], s_k[2][kBlockCells];  // determinant -> its strings
    // first cells of block g and of block h of record row ij (alpha) and of record column kl (beta)
    __shared__ unsigned char s_row[2][kBlockCells], s_col[2][kBlockCells];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gr = lane >> 2, gc = lane & 3;
    const int chunks = (R + 3) / 2;  // 16-byte pieces of a record up to the energy
    // block pairs of the band: a rectangle (g < h0) and a triangle
    const long long nh = a.h1 - a.h0, rect = nh * a.h0, total = rect + nh * (nh + 1) / 2;
    auto decode = [&](unsigned t, int* g, int* h) {
        if (t < (unsigned)rect) {
            *g = (int)(t / (unsigned)nh);
            *h = a.h0 + (int)(t - (unsigned)*g * (unsigned)nh);
            return;
        }
        const int q = (int)(t - (unsigned)rect);
        int y = (int)((sqrtf(8.0f * (float)q + 1.0f) - 1.0f) * 0.5f);
        while (y * (y + 1) / 2 > q) --y;
        while ((y + 1) * (y + 2) / 2 <= q) ++y;
        *h = a.h0 + y;
        *g = a.h0 + (q - y * (y + 1) / 2);
    };
    constexpr int kWords = sizeof(BlockStrings) / 4;  // one word per thread of the first two warps
    static_assert(kWords == 32 && 2 * kBlockCells <= 32 * kBlockWarps, "a descriptor per warp, a cell per thread");
    auto descriptor_word = [&](int g, int h) {
        return __ldg(reinterpret_cast<const unsigned*>(a.strings + (tid < kWords ? g : h)) + tid % kWords);
    };
    // a warp copies the records warp, warp + 8, ... of a block pair: lane q addresses the q-th of them
    auto load_records = [&](const BlockStrings* desc) {
        const int wa = desc[1].n_alpha, wb = desc[1].n_beta;
        const int rows_a = desc[0].n_alpha * wa, rows = rows_a + desc[0].n_beta * wb;
        const double* rec = nullptr;
        const int r = warp + kBlockWarps * lane;
        if (r < rows) {
            const bool beta = r >= rows_a;
            const int q = beta ? r - rows_a : r, w = beta ? wb : wa;
            const int qi = q / w, qj = q - qi * w;
            const int u = beta ? desc[0].beta[qi] : desc[0].alpha[qi];
            const int v = beta ? desc[1].beta[qj] : desc[1].alpha[qj];
            const long long at = record_index(min(u, v), max(u, v), beta ? a.f.Nb : a.f.Na);
            rec = beta ? a.f.rec_b + at * a.f.stride_b : a.f.rec_a + at * a.f.stride_a;
        }
        for (int it = 0, y = warp; y < rows; ++it, y += kBlockWarps) {
            const double* src =
                reinterpret_cast<const double*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(rec), it));
            const unsigned dst = (unsigned)__cvta_generic_to_shared(y < rows_a ? sA + y * LD : sB + (y - rows_a) * LD);
            for (int piece = lane; piece < chunks; piece += 32)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * piece), "l"(src + 2 * piece) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // fragment tiles of this warp: M tiles wm and wm + 4, N tiles wn to wn + 3
    const int wm = warp & 3, wn = 4 * (warp >> 2);
    int g = 0, h = 0, g1 = 0, h1 = 0;  // blocks of this pair and of the next
    unsigned word = 0;                 // this thread's word of the pair after next
    long long t = blockIdx.x;
    if (t < total) {
        decode(t, &g, &h);
        if (tid < 2 * kWords) reinterpret_cast<unsigned*>(s_desc[0])[tid] = descriptor_word(g, h);
        if (t + gridDim.x < total) {
            decode(t + gridDim.x, &g1, &h1);
            if (tid < 2 * kWords) word = descriptor_word(g1, h1);
        }
    }
    __syncthreads();
    for (int parity = 0; t < total; t += gridDim.x, parity ^= 1) {
        const int d0 = __ldg(a.first + g), nd = __ldg(a.first + g + 1) - d0;
        const int e0 = __ldg(a.first + h), ne = __ldg(a.first + h + 1) - e0;
        const bool diagonal = g == h, more = t + gridDim.x < total;
        const BlockStrings* desc = s_desc[parity];
        __syncthreads();  // the previous pair's shared data is consumed
        load_records(desc);
        if (tid < 2 * kWords && more) reinterpret_cast<unsigned*>(s_desc[parity ^ 1])[tid] = word;
        const int wa = desc[1].n_alpha, wb = desc[1].n_beta;
        const int rows_a = desc[0].n_alpha * wa, rows_b = desc[0].n_beta * wb;
        if (tid < 2 * kBlockCells) {
            const int which = tid / kBlockCells, cell = tid % kBlockCells;
            const unsigned char at = desc[which].cell[cell];
            if (at != 0xFF) {
                s_i[which][at] = (unsigned char)(cell / kBlockEdge);
                s_k[which][at] = (unsigned char)(cell % kBlockEdge);
            }
        } else if (tid < 4 * kBlockCells) {
            const bool beta = tid >= 3 * kBlockCells;
            const int q = tid % kBlockCells, w = beta ? wb : wa, qi = q / w;
            if (q < (beta ? rows_b : rows_a)) {
                (beta ? s_col[0] : s_row[0])[q] = (unsigned char)(beta ? qi : kBlockEdge * qi);
                (beta ? s_col[1] : s_row[1])[q] = (unsigned char)(beta ? q - qi * w : kBlockEdge * (q - qi * w));
            }
        }
        g = g1;
        h = h1;
        if (t + 2 * (long long)gridDim.x < total) {
            decode(t + 2 * (long long)gridDim.x, &g1, &h1);
            if (tid < 2 * kWords) word = descriptor_word(g1, h1);
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        const int mt = (rows_a + 7) / 8, nt = (rows_b + 7) / 8 - wn;
        if (wm < mt && nt > 0) {
            double acc[2][4][2];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
            const bool two = wm + 4 < mt;
            const double* pa = sA + (8 * wm + gr) * LD;
            const double* pa2 = pa + (two ? 32 * LD : 0);
            const double* pb = sB + (8 * wn + gr) * LD;
            // sign of the factor columns from r_pos on
            auto signed_value = [](double x, bool negative) {
                return __hiloint2double(__double2hiint(x) ^ (negative ? 0x80000000 : 0), __double2loint(x));
            };
            auto products = [&](double a0, double a1, int kb, bool on) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (j >= nt) break;
                    const double b = on ? pb[8 * j * LD + kb] : 0.0;
                    mma_f64(acc[0][j], a0, b);
                    if (two) mma_f64(acc[1][j], a1, b);
                }
            };
            int k = 0;
#pragma unroll 2
            for (; k + 4 <= R; k += 4) {
                const bool negative = k + gc >= r_pos;
                products(signed_value(pa[k + gc], negative), signed_value(pa2[k + gc], negative), k + gc, true);
            }
            for (; k < KD; k += 4) {
                // the remaining factor columns, then H_a S_b and S_a H_b (a record holds [.. | S | H])
                const int m = k + gc;
                const bool on = m < R + 2, negative = m < R && m >= r_pos;
                const int ma = m < R ? m : (on ? 2 * R + 1 - m : 0);
                products(on ? signed_value(pa[ma], negative) : 0.0, on ? signed_value(pa2[ma], negative) : 0.0, on ? m : 0, on);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int r = 8 * (wm + 4 * i) + gr;
                if (r >= rows_a) continue;
                const unsigned char* cg = desc[0].cell + s_row[0][r];
                const unsigned char* ch = desc[1].cell + s_row[1][r];
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        const int c = 8 * (wn + j) + 2 * gc + x;
                        if (c >= rows_b) continue;
                        const unsigned d = cg[s_col[0][c]], e = ch[s_col[1][c]];
                        if (d != 0xFF && e != 0xFF) sH[d * OUT + e] = acc[i][j][x];
                    }
            }
        }
        __syncthreads();
        for (int d = warp; d < nd; d += kBlockWarps) {
            const int i = s_i[0][d] * wa, k = s_k[0][d] * wb;
            double* H = a.f.Hb + (d0 + d) * a.f.ldb + (e0 - a.f.e0);
            double* S = a.f.Sb + (d0 + d) * a.f.ldb + (e0 - a.f.e0);
#pragma unroll 2
            for (int e = lane; e < ne; e += 32) {
                if (diagonal && e < d) continue;
                const double w = diagonal && e == d ? 0.5 : 1.0;
                const double sa = sA[(i + s_i[1][e]) * LD + R], sb = sB[(k + s_k[1][e]) * LD + R];
                H[e] = w * sH[d * OUT + e];
                S[e] = w * (sa * sb);
            }
        }
    }
}

// Listed determinant pairs (d, e) in any order.
__global__ void listed_pairs_kernel(FullPairArgs a, long long n_pairs, const long long* __restrict__ pairs,
                                    double* __restrict__ h_out, double* __restrict__ s_out) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n_pairs;
         t += (long long)gridDim.x * blockDim.x) {
        double H, S;
        pair_value(a, pairs[2 * t], pairs[2 * t + 1], &H, &S);
        h_out[t] = H;
        s_out[t] = S;
    }
}

__global__ void resolve_blocks_kernel(int k, long long batch, const double* __restrict__ blocks, double* det,
                                      int* nullity, double* cof_out) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < batch;
         t += (long long)gridDim.x * blockDim.x) {
        dev::Resolution res;
        dev::resolve_exact(k, blocks + t * k * k, kThreshold, &res);
        double cof[dev::KMAX * dev::KMAX];
        dev::first_cofactor(res, cof);
        det[t] = res.det;
        nullity[t] = res.nullity;
        if (cof_out)
            for (int i = 0; i < k * k; ++i) cof_out[t * k * k + i] = res.nullity <= 1 ? cof[i] : 0.0;
    }
}

__global__ void same_spin_list_kernel(int n, int k, long long batch, const int* __restrict__ occ_left,
                                      const int* __restrict__ occ_right, const double* __restrict__ S,
                                      const double* __restrict__ h, const double* __restrict__ eri, double* scalars,
                                      double* cof_out) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < batch;
         t += (long long)gridDim.x * blockDim.x) {
        int L[dev::KMAX], R[dev::KMAX];
        for (int i = 0; i < k; ++i) {
            L[i] = occ_left[t * k + i];
            R[i] = occ_right[t * k + i];
        }
        double x[dev::KMAX * dev::KMAX];
        for (int c = 0; c < k; ++c)
            for (int r = 0; r < k; ++r) x[c * k + r] = S[L[c] * n + R[r]];
        dev::Resolution res;
        dev::resolve_exact(k, x, kThreshold, &res);
        double cof[dev::KMAX * dev::KMAX];
        dev::first_cofactor(res, cof);
        double h1 = 0.0, htot = 0.0;
        if (k > 0 && res.nullity < 3) htot = dev::same_spin_exact(n, k, L, R, res, cof, h, eri, &h1);
        scalars[4 * t + 0] = res.det;
        scalars[4 * t + 1] = h1;
        scalars[4 * t + 2] = htot;
        scalars[4 * t + 3] = (double)res.nullity;
        if (cof_out)
            for (int i = 0; i < k * k; ++i) cof_out[t * k * k + i] = res.nullity <= 1 ? cof[i] : 0.0;
    }
}

}  // namespace

cudaError_t launch_factor_pair_kernel(int np, const double* kfull, double* work, double* cols, int* signs, double* lf,
                                      int ld, int* meta, cudaStream_t stream) {
    const double tol = factor_tolerance(np);
    // up to 152 rows (16 orbitals) the columns fit shared memory and the Schur complement registers
    const size_t columns = sizeof(double) * (size_t)np * np;
    auto registers = [&](auto kernel, int warps) {
        const cudaError_t err = allow_dynamic_smem((const void*)kernel, columns);
        if (err != cudaSuccess) return err;
        kernel<<<1, 32 * warps, columns, stream>>>(np, kfull, signs, lf, ld, meta, tol);
        return cudaGetLastError();
    };
    if (np <= 32) return registers(factor_pair_registers<4, 1>, 4);
    if (np <= 64) return registers(factor_pair_registers<8, 2>, 8);
    if (np <= 96) return registers(factor_pair_registers<16, 3>, 16);
    if (np <= 128) return registers(factor_pair_registers<16, 4>, 16);
    if (np <= 152) return registers(factor_pair_registers<16, 5>, 16);
    int threads = (np + 31) / 32 * 32;
    threads = threads > 1024 ? 1024 : threads;
    if (np > threads * kFactorRows) return cudaErrorInvalidValue;
    const size_t smem = sizeof(double) * ((size_t)np + (np + 2) / 2);
    cudaError_t err = allow_dynamic_smem((const void*)factor_pair_kernel, (int)smem);
    if (err != cudaSuccess) return err;
    factor_pair_kernel<<<1, threads, smem, stream>>>(np, kfull, work, cols, signs, lf, ld, meta, tol);
    return cudaGetLastError();
}

cudaError_t launch_prepare_tables(int n, const double* eri, double* gamma, double* kfull, cudaStream_t stream) {
    const long long np = (long long)n * (n + 1) / 2, gd = (long long)n * (n - 1) / 2;
    long long total = np * np + gd * gd;
    long long blocks = (total + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    if (blocks < 1) blocks = 1;
    prepare_tables_kernel<<<(unsigned)blocks, 256, 0, stream>>>(n, eri, gamma, kfull);
    return cudaGetLastError();
}

size_t exact_stack_bytes() {
    size_t m = 0;
    cudaFuncAttributes fa{};
    if (cudaFuncGetAttributes(&fa, spin_pairs_exact<8, 0>) == cudaSuccess) m = std::max(m, fa.localSizeBytes);
    if (cudaFuncGetAttributes(&fa, spin_pairs_exact<7, 7>) == cudaSuccess) m = std::max(m, fa.localSizeBytes);
    return m;
}

cudaError_t preload_spin_pair_kernels() {
    // cudaFuncGetAttributes loads a function that lazy module loading has not loaded yet
    const void* fns[] = {(const void*)prepare_tables_kernel, (const void*)factor_pair_kernel,
                         (const void*)factor_pair_registers<4, 1>, (const void*)factor_pair_registers<8, 2>,
                         (const void*)factor_pair_registers<16, 3>, (const void*)factor_pair_registers<16, 4>,
                         (const void*)factor_pair_registers<16, 5>,
                         (const void*)spin_pairs_exact<7, 7>, (const void*)spin_pairs_exact<8, 0>,
                         (const void*)spin_pairs_exact<dev::KMAX, 0>};
    for (const void* f : fns) {
        cudaFuncAttributes fa{};
        const cudaError_t err = cudaFuncGetAttributes(&fa, f);
        if (err != cudaSuccess) return err;
    }
    return preload_frame_kernels();
}

cudaError_t launch_spin_tables(const SpinTableArgs& a, double* tables, cudaStream_t stream, int* launches) {
    if (a.n_pairs <= 0 || a.k <= 0 || a.all_careful || !frame_spin_supported(a.n, a.k, a.R)) return cudaSuccess;
    ++*launches;
    return launch_frame_tables(a, tables, stream);
}

cudaError_t launch_spin_pairs(const SpinTableArgs& a, double* tables, cudaStream_t stream, int* launches) {
    if (a.n_pairs <= 0 || a.k <= 0) return cudaSuccess;
    cudaError_t err = cudaSuccess;
    const bool fast_ok = !a.all_careful && frame_spin_supported(a.n, a.k, a.R);
    if (fast_ok) {
        // the pair-to-warp schedule (warps per CTA) is chosen by the autotuner per shape; the
        // listed-pair counter and the task counter are restored before every timed launch
        const std::string key = "spin_pairs_frame k=" + std::to_string(a.k) + " n=" + std::to_string(a.n) +
                                " R=" + std::to_string(a.R) + " N=" + std::to_string(a.n_strings);
        const int tuned = autotune_run(
            key, frame_pair_variants(a.n, a.k, a.R), stream, [&](int v) { return launch_frame_pairs(a, tables, stream, v); },
            [&]() {
                // the counters of listed and uncertified pairs and the task counter
                cudaError_t e = cudaMemsetAsync(a.careful_count, 0, sizeof(unsigned long long), stream);
                if (e == cudaSuccess && a.uncertified)
                    e = cudaMemsetAsync(a.uncertified, 0, sizeof(unsigned long long), stream);
                if (e == cudaSuccess) e = cudaMemsetAsync(a.task_counter, 0, sizeof(unsigned long long), stream);
                return e;
            },
            &err);
        (void)tuned;
        if (err != cudaSuccess) return err;
        ++*launches;
    }
    return cudaSuccess;
}

cudaError_t launch_spin_pairs_exact(const SpinTableArgs& a, cudaStream_t stream, int* launches) {
    if (a.n_pairs <= 0 || a.k <= 0) return cudaSuccess;
    cudaError_t err = cudaSuccess;
    const bool fast_ok = !a.all_careful && frame_spin_supported(a.n, a.k, a.R);
    SpinTableArgs b = a;
    b.all_careful = fast_ok ? 0 : 1;
    auto exact = a.k == 7 ? spin_pairs_exact<7, 7> : (a.k <= 8 ? spin_pairs_exact<8, 0> : spin_pairs_exact<dev::KMAX, 0>);
    const size_t slot_bytes = sizeof(double) * 64 * (size_t)a.k * a.k;  // two warps
    if (slot_bytes > 48 * 1024) {
        err = allow_dynamic_smem((const void*)exact, (int)slot_bytes);
        if (err != cudaSuccess) return err;
    }
    // at most one warp per pair of the table: the list is usually empty, and a full grid of CTAs that only
    // read its length takes 6 us
    const long long grid = (a.n_pairs + 1) / 2;
    exact<<<(unsigned)(grid < kSms * 8 ? grid : kSms * 8), 64, slot_bytes, stream>>>(b);
    ++*launches;
    return cudaGetLastError();
}

cudaError_t launch_full_pairs(const FullPairArgs& a, cudaStream_t stream, int* launches) {
    if (a.n_items <= 0) return cudaSuccess;
    // launch variants (block size, CTAs per SM), chosen by the autotuner per band shape
    constexpr int kVariants = 4;
    constexpr int threads[kVariants] = {256, 128, 256, 512};
    constexpr int per_sm[kVariants] = {16, 16, 8, 4};
    const std::string key = "full_pairs_kernel R=" + std::to_string(a.R) + " ndet=" + std::to_string(a.n_det) +
                            " items=" + std::to_string(a.n_items) + " flip=" + std::to_string(a.flip ? 1 : 0);
    cudaError_t err = cudaSuccess;
    autotune_run(
        key, kVariants, stream,
        [&](int v) {
            long long blocks = (a.n_items + threads[v] - 1) / threads[v];
            if (blocks > (long long)kSms * per_sm[v]) blocks = (long long)kSms * per_sm[v];
            full_pairs_kernel<<<(unsigned)blocks, threads[v], 0, stream>>>(a);
            return cudaGetLastError();
        },
        {}, &err);
    ++*launches;
    return err;
}

bool block_pairs_supported(int max_a, int max_b, int max_dets, int R) {
    // of the 227 KB a CTA may have, the kernel's static arrays take one
    return block_pairs_smem(max_a, max_b, max_dets, R) <= 226 * 1024;
}

cudaError_t launch_block_pairs(const BlockPairArgs& a, cudaStream_t stream, int* launches) {
    const long long nh = a.h1 - a.h0, total = nh * a.h0 + nh * (nh + 1) / 2;
    if (total <= 0) return cudaSuccess;
    const size_t smem = block_pairs_smem(a.max_a, a.max_b, a.max_dets, a.f.R);
    const auto kernel = block_pairs_kernel;
    cudaError_t err = allow_dynamic_smem((const void*)kernel, smem);
    if (err != cudaSuccess) return err;
    int per_sm = 1;
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 32 * kBlockWarps, smem);
    if (err != cudaSuccess) return err;
    // launch variants (CTAs per SM: as many as fit, or one less), chosen by the autotuner per list on a band
    // that fills the chip sixteen times over (the first bands of a large list are too short to tell: tuned
    // there, 34,188 determinants took 10.3 ms instead of 8.7)
    if (per_sm < 1) per_sm = 1;
    const int fewer = per_sm > 1 ? per_sm - 1 : 1;
    auto launch = [&](int v) {
        const long long grid = (long long)kSms * (v ? fewer : per_sm);
        kernel<<<(unsigned)(total < grid ? total : grid), 32 * kBlockWarps, smem, stream>>>(a);
        return cudaGetLastError();
    };
    ++*launches;
    if (total < 16ll * kSms * per_sm) return launch(0);
    autotune_run("full_pairs_kernel (blocks) R=" + std::to_string(a.f.R) + " ndet=" + std::to_string(a.f.n_det), 2, stream,
                 launch, {}, &err);
    return err;
}

cudaError_t launch_listed_pairs(const FullPairArgs& a, long long n_pairs, const long long* pairs, double* h_out,
                                double* s_out, cudaStream_t stream) {
    if (n_pairs <= 0) return cudaSuccess;
    long long blocks = (n_pairs + 127) / 128;
    if (blocks > kSms * 16) blocks = kSms * 16;
    listed_pairs_kernel<<<(unsigned)blocks, 128, 0, stream>>>(a, n_pairs, pairs, h_out, s_out);
    return cudaGetLastError();
}

cudaError_t launch_resolve_blocks(int k, long long batch, const double* blocks, double* det, int* nullity, double* cof,
                                  cudaStream_t stream) {
    if (batch <= 0) return cudaSuccess;
    long long g = (batch + 63) / 64;
    if (g > kSms * 8) g = kSms * 8;
    resolve_blocks_kernel<<<(unsigned)g, 64, 0, stream>>>(k, batch, blocks, det, nullity, cof);
    return cudaGetLastError();
}

cudaError_t launch_same_spin_list(int n, int k, long long batch, const int* occ_left, const int* occ_right,
                                  const double* S, const double* h, const double* eri, double* scalars, double* cof,
                                  cudaStream_t stream) {
    if (batch <= 0) return cudaSuccess;
    long long g = (batch + 63) / 64;
    if (g > kSms * 8) g = kSms * 8;
    same_spin_list_kernel<<<(unsigned)g, 64, 0, stream>>>(n, k, batch, occ_left, occ_right, S, h, eri, scalars, cof);
    return cudaGetLastError();
}

}  // namespace vbcore
