// Lowest root of the dense structure problem H c = E S c by a generalized Davidson iteration
// on the device (the selected-root path of solve_structure_problem,
// src/vbscf/derivatives/gradient/active_space/evaluator.cpp:466-560, and
// GeneralizedEigensolver::solve_davidson, src/linalg/eigensolver.hpp:194-198, here on the
// materialized H and S).  For structure spaces too large for the dense all-root solver.
//
// Per iteration, with one read-back: a pass over H and S computes H t and S t of the newest
// direction t (the HBM-bound step: 16 n^2 bytes) after its second orthogonalization; the images
// kernel adds up the partial sums and forms every dot product with the basis; the host extends
// the projected problem (dimension <= kMaxSubspace) by the new row in O(k^2) and takes its lowest
// pair from a Householder tridiagonal form; the Ritz kernel appends the scaled column, forms the
// Ritz vector, its images, the residual r = H x - theta S x, the correction t = r / (theta S_ii -
// H_ii) and the dot products of the first S-orthogonalization; the orthogonalization kernel
// applies them and forms those of the second.  The convergence norms of an iteration are read
// with the next one's dot products.  A full basis restarts from its 12 lowest Ritz vectors (thick
// restart).  Converged when ||r||_2 <= tol (||H x|| + |theta| ||S x||) (a backward-error
// criterion, attainable whatever the conditioning of S).  The diagonal preconditioner is weak on
// strongly coupled structure matrices, so after 24 iterations the Ritz value seeds a shift sigma
// below the lowest root (lowered until H - sigma S = U^T U is positive definite) and the
// correction becomes t = U^-1 U^-T r: the basis then grows along the Krylov space of the
// shift-inverted operator, whose lowest root is well separated.
//
// What bounds it: below n of about 1000 the launches, read-backs and the projected problem.  With
// a launch per vector operation, five read-backs per iteration and a cyclic Jacobi of the whole
// projected problem (1.8 ms at dimension 48), the 294 structures of eight orbitals took 8.2 ms per
// energy and gradient; 2.8 ms this way.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "internal.h"

namespace vbcore {
namespace {

constexpr int kMaxSubspace = 48;
constexpr int kKeep = 12;  // Ritz vectors kept at a restart
constexpr int kDiagonalPhase = 24;  // iterations with the diagonal preconditioner
constexpr int kSplits = 64;  // most column ranges of the matrix-vector partial sums
constexpr int kRows = 64;    // rows per CTA of the vector kernels
constexpr int kVecThreads = 256;
constexpr int kVecWarps = kVecThreads / 32;
constexpr int kDotsMax = 2 * (kMaxSubspace + 1) + 3;  // dot products one kernel forms

// Column ranges of the matrix-vector passes: enough CTAs (256 rows each) to fill the GPU several
// times, at least eight columns per range (n = 294: 36 ranges of 9; n = 5676: 64 of 89)
int gemv_splits(int n) { return std::max(1, std::min(kSplits, n / 8)); }

struct Coefficients {
    double v[kMaxSubspace];
};

// y_h = H x, y_s = S x (column-major n x n), partial sums over column ranges, where x = t - V c is
// formed by each CTA for its own columns (c == nullptr: x = t) and stored to x_out by the first row
// of CTAs.
__global__ void __launch_bounds__(256) gemv2_partial_kernel(const double* __restrict__ H, const double* __restrict__ S,
                                                            int n, const double* __restrict__ t,
                                                            const double* __restrict__ V, int k,
                                                            const double* __restrict__ c, double* __restrict__ x_out,
                                                            double* __restrict__ part_h, double* __restrict__ part_s) {
    __shared__ double sx[256], sc[kMaxSubspace];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int split = blockIdx.y;
    const int chunk = (n + gridDim.y - 1) / gridDim.y;
    const int j0 = split * chunk, j1 = min(n, j0 + chunk);
    if (c && threadIdx.x < k) sc[threadIdx.x] = c[threadIdx.x];
    double ah = 0.0, as = 0.0;
    for (int jc = j0; jc < j1; jc += 256) {
        const int cnt = min(256, j1 - jc);
        __syncthreads();
        if ((int)threadIdx.x < cnt) {
            const int j = jc + threadIdx.x;
            double v = t[j];
            if (c)
#pragma unroll 8
                for (int q = 0; q < k; ++q) v = fma(-__ldg(V + j + (long long)q * n), sc[q], v);
            sx[threadIdx.x] = v;
            if (blockIdx.x == 0) x_out[j] = v;
        }
        __syncthreads();
        if (i < n) {
            const double* h = H + i + (long long)jc * n;
            const double* s = S + i + (long long)jc * n;
#pragma unroll 8
            for (int j = 0; j < cnt; ++j) {
                ah = fma(__ldg(h + (long long)j * n), sx[j], ah);
                as = fma(__ldg(s + (long long)j * n), sx[j], as);
            }
        }
    }
    if (i < n) {
        part_h[(long long)split * n + i] = ah;
        part_s[(long long)split * n + i] = as;
    }
}

// Sum over rows of the CTA's tile, for count dot products (values by dot(c, row)): partial sums to
// partial[block][c]; the last CTA to finish adds them up in block order into out.
template <class Dot>
__device__ __forceinline__ void block_dots(int n, int count, const Dot& dot, double* __restrict__ partial,
                                           double* __restrict__ out, unsigned* __restrict__ counter) {
    __shared__ bool s_last;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r0 = blockIdx.x * kRows;
#pragma unroll 2
    for (int c = warp; c < count; c += kVecWarps) {
        double acc = 0.0;
#pragma unroll
        for (int h = 0; h < kRows / 32; ++h)
            if (r0 + lane + 32 * h < n) acc += dot(c, lane + 32 * h);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) partial[(long long)blockIdx.x * kDotsMax + c] = acc;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(counter, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int c = threadIdx.x; c < count; c += blockDim.x) {
        double acc = 0.0;
#pragma unroll 8
        for (int b = 0; b < (int)gridDim.x; ++b) acc += __ldcg(partial + (long long)b * kDotsMax + c);
        out[c] = acc;
    }
    if (threadIdx.x == 0) *counter = 0;
}

// s_out[m][row] = sum_c A_m[row + c n] coef(c) for the CTA's rows and M matrices, the columns split
// over the CTA's thread groups and added up in group order.
template <int M, class Coef>
__device__ __forceinline__ void block_combine(int n, int k, const double* const (&A)[M], const Coef& coef,
                                              double (*s_part)[kVecThreads], double (*s_out)[kRows]) {
    constexpr int G = kVecThreads / kRows;
    const int row = threadIdx.x % kRows, g = threadIdx.x / kRows;
    const int i = blockIdx.x * kRows + row;
    double acc[M];
#pragma unroll
    for (int m = 0; m < M; ++m) acc[m] = 0.0;
    if (i < n)
#pragma unroll 4
        for (int c = g; c < k; c += G)
#pragma unroll
            for (int m = 0; m < M; ++m) acc[m] = fma(A[m][i + (long long)c * n], coef(c), acc[m]);
#pragma unroll
    for (int m = 0; m < M; ++m) s_part[m][threadIdx.x] = acc[m];
    __syncthreads();
    for (int e = threadIdx.x; e < M * kRows; e += kVecThreads) {
        const int m = e / kRows, r = e % kRows;
        double v = 0.0;
#pragma unroll
        for (int q = 0; q < G; ++q) v += s_part[m][q * kRows + r];
        s_out[m][r] = v;
    }
    __syncthreads();
}

// H t and S t from the partial sums, and out = [V^T H t (k), t^T H t, V^T S t (k), t^T S t].
__global__ void __launch_bounds__(kVecThreads) images_kernel(int n, int k, int splits, const double* __restrict__ ph,
                                                             const double* __restrict__ ps,
                                                             const double* __restrict__ V,
                                                             const double* __restrict__ t, double* __restrict__ ht,
                                                             double* __restrict__ st, double* __restrict__ partial,
                                                             double* __restrict__ out, unsigned* counter) {
    __shared__ double s_part[2][kVecThreads], s_img[2][kRows];
    const double* const parts[2] = {ph, ps};
    block_combine<2>(n, splits, parts, [](int) { return 1.0; }, s_part, s_img);
    const int r0 = blockIdx.x * kRows;
    if (threadIdx.x < kRows && r0 + (int)threadIdx.x < n) {
        ht[r0 + threadIdx.x] = s_img[0][threadIdx.x];
        st[r0 + threadIdx.x] = s_img[1][threadIdx.x];
    }
    block_dots(n, 2 * (k + 1), [&](int c, int row) {
        const int m = c > k, q = m ? c - k - 1 : c;
        const double v = q < k ? V[r0 + row + (long long)q * n] : t[r0 + row];
        return v * s_img[m][row];
    }, partial, out, counter);
}

// The Ritz pair of the extended basis: column k - 1 of V, HV and SV becomes scale times t and its
// images; x, H x, S x = the combinations by y; r = H x - theta S x; and (diagonal) the corrections
// t_out = r / (theta S_ii - H_ii).  out = [|H x|^2, |S x|^2, |r|^2, then (diagonal) (S V)^T t_out].
__global__ void __launch_bounds__(kVecThreads) ritz_kernel(int n, int k, Coefficients y, double scale, double theta,
                                                           bool diagonal, double* V, double* HV, double* SV,
                                                           const double* __restrict__ t, const double* __restrict__ ht,
                                                           const double* __restrict__ st,
                                                           const double* __restrict__ hd, const double* __restrict__ sd,
                                                           double* __restrict__ x, double* __restrict__ r,
                                                           double* __restrict__ t_out, double* __restrict__ partial,
                                                           double* __restrict__ out, unsigned* counter) {
    __shared__ double s_part[3][kVecThreads], s_img[3][kRows], s_y[kMaxSubspace], s_r[kRows], s_t[kRows];
    const int r0 = blockIdx.x * kRows, row = threadIdx.x;
    if (threadIdx.x < kMaxSubspace) s_y[threadIdx.x] = y.v[threadIdx.x];
    if (row < kRows && r0 + row < n) {
        const long long at = r0 + row + (long long)(k - 1) * n;
        V[at] = scale * t[r0 + row];
        HV[at] = scale * ht[r0 + row];
        SV[at] = scale * st[r0 + row];
    }
    __syncthreads();
    const double* const images[3] = {V, HV, SV};
    block_combine<3>(n, k, images, [&](int c) { return s_y[c]; }, s_part, s_img);
    if (row < kRows) {
        double ri = 0.0, ti = 0.0;
        if (r0 + row < n) {
            ri = s_img[1][row] - theta * s_img[2][row];
            double den = theta * sd[r0 + row] - hd[r0 + row];
            if (fabs(den) < 1.0e-8) den = den < 0.0 ? -1.0e-8 : 1.0e-8;
            ti = ri / den;
            x[r0 + row] = s_img[0][row];
            r[r0 + row] = ri;
            if (diagonal) t_out[r0 + row] = ti;
        }
        s_r[row] = ri;
        s_t[row] = ti;
    }
    __syncthreads();
    block_dots(n, 3 + (diagonal ? k : 0), [&](int c, int q) {
        if (c == 0) return s_img[1][q] * s_img[1][q];
        if (c == 1) return s_img[2][q] * s_img[2][q];
        if (c == 2) return s_r[q] * s_r[q];
        return SV[r0 + q + (long long)(c - 3) * n] * s_t[q];
    }, partial, out, counter);
}

// t (or, with part, the sum of its column-range partial sums) minus V c (c != nullptr), in place,
// and out = (S V)^T t.
__global__ void __launch_bounds__(kVecThreads) orthogonalize_kernel(int n, int k, const double* __restrict__ V,
                                                                    const double* __restrict__ SV,
                                                                    const double* __restrict__ part, int splits,
                                                                    const double* __restrict__ c, double* t,
                                                                    double* __restrict__ partial,
                                                                    double* __restrict__ out, unsigned* counter) {
    __shared__ double s_part[1][kVecThreads], s_sum[1][kRows], s_t[kRows], s_c[kMaxSubspace];
    const int r0 = blockIdx.x * kRows, row = threadIdx.x;
    if (part) {
        const double* const parts[1] = {part};
        block_combine<1>(n, splits, parts, [](int) { return 1.0; }, s_part, s_sum);
        if (row < kRows) s_t[row] = s_sum[0][row];
    } else if (row < kRows) {
        s_t[row] = r0 + row < n ? t[r0 + row] : 0.0;
    }
    if (c) {
        if (threadIdx.x < k) s_c[threadIdx.x] = c[threadIdx.x];
        __syncthreads();
        const double* const basis[1] = {V};
        block_combine<1>(n, k, basis, [&](int q) { return s_c[q]; }, s_part, s_sum);
        if (row < kRows) s_t[row] -= s_sum[0][row];
    }
    if (row < kRows && r0 + row < n) t[r0 + row] = s_t[row];
    __syncthreads();
    block_dots(n, k, [&](int q, int rw) { return SV[r0 + rw + (long long)q * n] * s_t[rw]; }, partial, out, counter);
}

// Thick restart: out[m][j] = sum_c A_m[:, c] coef[c + j k] for the basis and its two images
// (blockIdx.y = j + keep m; out column-major, the images' blocks keep columns apart).
__global__ void restart_kernel(int n, int k, int keep, const double* __restrict__ V, long long image_step,
                               const double* __restrict__ coef, double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int j = blockIdx.y % keep, m = blockIdx.y / keep;
    const double* A = V + m * image_step + i;
    double acc = 0.0;
#pragma unroll 8
    for (int c = 0; c < k; ++c) acc = fma(A[(long long)c * n], __ldg(coef + c + j * k), acc);
    out[i + (long long)blockIdx.y * n] = acc;
}

__global__ void diag_kernel(int n, const double* __restrict__ H, const double* __restrict__ S, double* hd, double* sd) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    hd[i] = H[i + (long long)i * n];
    sd[i] = S[i + (long long)i * n];
}

// t = the unit vector of the row with the smallest H_ii / S_ii (the first of equals), one CTA.
__global__ void __launch_bounds__(1024) start_kernel(int n, const double* __restrict__ hd, const double* __restrict__ sd,
                                                     double* __restrict__ t) {
    __shared__ double s_v[32];
    __shared__ int s_i[32];
    double best = 0.0;
    int bi = -1;
    auto take = [&](double v, int i) {
        if (i >= 0 && (bi < 0 || v < best || (v == best && i < bi))) {
            best = v;
            bi = i;
        }
    };
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double v = hd[i] / sd[i];
        if (v == v || (i == 0)) take(v == v ? v : INFINITY, i);
        t[i] = 0.0;
    }
    auto warp_best = [&]() {
        for (int o = 16; o > 0; o >>= 1) {
            const double v = __shfl_xor_sync(0xffffffffu, best, o);
            const int i = __shfl_xor_sync(0xffffffffu, bi, o);
            take(v, i);
        }
    };
    warp_best();
    if ((threadIdx.x & 31) == 0) {
        s_v[threadIdx.x >> 5] = best;
        s_i[threadIdx.x >> 5] = bi;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        best = s_v[threadIdx.x];
        bi = s_i[threadIdx.x];
        warp_best();
        if (threadIdx.x == 0) t[bi] = 1.0;
    }
}

// y = A^T x for upper-triangular A (one warp per column, coalesced down the column's rows <= col)
__global__ void __launch_bounds__(256) gemv_t_kernel(const double* __restrict__ A, int n, const double* __restrict__ x,
                                                     double* __restrict__ y) {
    const int col = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (col >= n) return;
    const double* a = A + (long long)col * n;
    double acc = 0.0;
    for (int i = lane; i <= col; i += 32) acc = fma(__ldg(a + i), __ldg(x + i), acc);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) y[col] = acc;
}

// y = A x for upper-triangular A, column-split partial sums (same scheme as gemv2; row i reads
// only its columns j >= i)
__global__ void __launch_bounds__(256) gemv_partial_kernel(const double* __restrict__ A, int n,
                                                           const double* __restrict__ x, double* __restrict__ part) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int split = blockIdx.y;
    const int chunk = (n + gridDim.y - 1) / gridDim.y;
    const int j0 = split * chunk, j1 = min(n, j0 + chunk);
    if (i >= n) return;
    double acc = 0.0;
#pragma unroll 8
    for (int j = max(j0, i); j < j1; ++j) acc = fma(__ldg(A + i + (long long)j * n), __ldg(x + j), acc);
    part[(long long)split * n + i] = acc;
}

// M = H - sigma S
__global__ void shift_kernel(long long count, const double* __restrict__ H, const double* __restrict__ S, double sigma,
                             double* __restrict__ M) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < count; e += (long long)gridDim.x * blockDim.x)
        M[e] = H[e] - sigma * S[e];
}

// ---- projected problem (host) -----------------------------------------------------------------

// The two lowest eigenvalues and the lowest eigenvector of a symmetric k x k matrix: Householder
// tridiagonal form, bisection on Sturm counts, inverse iteration, transformed back.  About 0.07 ms
// at k = 48 (a cyclic Jacobi of the whole spectrum takes 1.8 ms there, 0.2 ms at k = 24).
struct LowestPair {
    std::vector<double> a, d, e, tau, w, u;  // u: reflector j in column j (k x k)
    std::vector<double> q;
    double theta[2] = {0.0, 0.0};

    void solve(int k, const std::vector<double>& m, int ld) {
        a.resize((size_t)k * k);
        for (int j = 0; j < k; ++j)
            for (int i = 0; i < k; ++i) a[i + (size_t)j * k] = m[i + (size_t)j * ld];
        d.assign(k, 0.0);
        e.assign(k, 0.0);
        tau.assign(k, 0.0);
        w.assign(k, 0.0);
        u.assign((size_t)k * k, 0.0);
        // column j: reflector I - tau v v^T on rows j + 1 .. k - 1 takes the column to e[j] e_{j+1}
        for (int j = 0; j + 2 < k; ++j) {
            double* col = &a[(size_t)j * k];
            double* v = &u[(size_t)j * k];
            double norm2 = 0.0;
            for (int i = j + 2; i < k; ++i) norm2 += col[i] * col[i];
            d[j] = col[j];
            if (norm2 == 0.0) {
                e[j] = col[j + 1];
                continue;
            }
            const double norm = std::sqrt(norm2 + col[j + 1] * col[j + 1]);
            const double beta = col[j + 1] > 0.0 ? -norm : norm;
            for (int i = j + 1; i < k; ++i) v[i] = col[i];
            v[j + 1] -= beta;
            tau[j] = 2.0 / (norm2 + v[j + 1] * v[j + 1]);
            e[j] = beta;
            // rank-two update of the trailing block: w = tau (A v - (tau v^T A v / 2) v)
            for (int i = j + 1; i < k; ++i) w[i] = 0.0;
            for (int c = j + 1; c < k; ++c) {
                const double* ac = &a[(size_t)c * k];
                const double vc = v[c];
                for (int i = j + 1; i < k; ++i) w[i] += ac[i] * vc;
            }
            double vav = 0.0;
            for (int i = j + 1; i < k; ++i) vav += v[i] * w[i];
            const double half = 0.5 * tau[j] * vav;
            for (int i = j + 1; i < k; ++i) w[i] = tau[j] * (w[i] - half * v[i]);
            for (int c = j + 1; c < k; ++c) {
                double* ac = &a[(size_t)c * k];
                const double vc = v[c], wc = w[c];
                for (int i = j + 1; i < k; ++i) ac[i] -= v[i] * wc + w[i] * vc;
            }
        }
        for (int j = std::max(0, k - 2); j < k; ++j) d[j] = a[j + (size_t)j * k];
        if (k > 1) e[k - 2] = a[(k - 1) + (size_t)(k - 2) * k];
        values(k);
        vector(k);
        for (int c = k - 3; c >= 0; --c) {
            if (tau[c] == 0.0) continue;
            const double* v = &u[(size_t)c * k];
            double dot = 0.0;
            for (int i = c + 1; i < k; ++i) dot += v[i] * q[i];
            dot *= tau[c];
            for (int i = c + 1; i < k; ++i) q[i] -= dot * v[i];
        }
        // Rayleigh quotient: the root to second order in the vector's rounding
        double rq = 0.0, qq = 0.0;
        for (int j = 0; j < k; ++j) {
            double acc = 0.0;
            for (int i = 0; i < k; ++i) acc += m[i + (size_t)j * ld] * q[i];
            rq += acc * q[j];
            qq += q[j] * q[j];
        }
        theta[0] = rq / qq;
    }

  private:
    std::vector<double> lu_d, lu_e, lu_f, lu_l;
    std::vector<char> swapped;
    double bound = 0.0;  // of the spectrum's magnitude (Gershgorin)

    void values(int k) {
        double lo = d[0], hi = d[0];
        for (int i = 0; i < k; ++i) {
            const double off = (i > 0 ? std::fabs(e[i - 1]) : 0.0) + (i + 1 < k ? std::fabs(e[i]) : 0.0);
            lo = std::min(lo, d[i] - off);
            hi = std::max(hi, d[i] + off);
        }
        bound = std::max(std::fabs(lo), std::fabs(hi));
        const double floor = std::max(bound, 1e-300) * 1.0e-290;
        // eigenvalues below x: negative pivots of T - x I
        auto below = [&](double x) {
            int count = 0;
            double p = d[0] - x;
            for (int i = 0;;) {
                if (p < 0.0) ++count;
                if (++i == k) return count;
                if (std::fabs(p) < floor) p = p < 0.0 ? -floor : floor;
                p = d[i] - x - e[i - 1] * e[i - 1] / p;
            }
        };
        for (int j = 0; j < std::min(k, 2); ++j) {
            double a0 = lo, a1 = hi;
            for (int iter = 0; iter < 64; ++iter) {
                const double mid = 0.5 * (a0 + a1);
                if (!(mid > a0 && mid < a1)) break;
                (below(mid) > j ? a1 : a0) = mid;
                if (a1 - a0 <= 1.1e-16 * bound) break;
            }
            theta[j] = 0.5 * (a0 + a1);
            lo = a0;
        }
    }

    // lowest eigenvector of the tridiagonal matrix by inverse iteration (LU with row exchanges)
    void vector(int k) {
        q.assign(k, 0.0);
        lu_d.assign(k, 0.0);
        lu_e.assign(k, 0.0);
        lu_f.assign(k, 0.0);
        lu_l.assign(k, 0.0);
        swapped.assign(k, 0);
        const double tiny = std::max(bound, 1e-280) * 2.2e-16;
        auto away = [&](double v) { return std::fabs(v) < tiny ? (v < 0.0 ? -tiny : tiny) : v; };
        double cur_d = d[0] - theta[0], cur_e = k > 1 ? e[0] : 0.0;
        for (int i = 0; i + 1 < k; ++i) {
            const double sub = e[i], nd = d[i + 1] - theta[0], ne = i + 2 < k ? e[i + 1] : 0.0;
            if (std::fabs(cur_d) >= std::fabs(sub)) {
                cur_d = away(cur_d);
                lu_d[i] = cur_d;
                lu_e[i] = cur_e;
                lu_l[i] = sub / cur_d;
                cur_d = nd - lu_l[i] * cur_e;
                cur_e = ne;
            } else {
                swapped[i] = 1;
                lu_d[i] = sub;
                lu_e[i] = nd;
                lu_f[i] = ne;
                lu_l[i] = cur_d / sub;
                cur_d = cur_e - lu_l[i] * nd;
                cur_e = -lu_l[i] * ne;
            }
        }
        lu_d[k - 1] = away(cur_d);
        for (int i = 0; i < k; ++i) q[i] = 1.0 + 0.01 * ((i * 7) % 11);
        for (int pass = 0; pass < 3; ++pass) {
            if (pass > 0)
                for (int i = 0; i + 1 < k; ++i) {
                    if (swapped[i]) std::swap(q[i], q[i + 1]);
                    q[i + 1] -= lu_l[i] * q[i];
                }
            for (int i = k - 1; i >= 0; --i) {
                double v = q[i];
                if (i + 1 < k) v -= lu_e[i] * q[i + 1];
                if (i + 2 < k) v -= lu_f[i] * q[i + 2];
                q[i] = v / lu_d[i];
            }
            double big = 0.0, norm = 0.0;
            for (int i = 0; i < k; ++i) big = std::max(big, std::fabs(q[i]));
            for (int i = 0; i < k; ++i) norm += (q[i] / big) * (q[i] / big);
            norm = std::sqrt(norm) * big;
            for (int i = 0; i < k; ++i) q[i] /= norm;
        }
    }
};

// All eigenvalues (ascending) and eigenvectors (columns of V) of a symmetric k x k matrix by cyclic
// Jacobi, for the thick restart.
void symmetric_eigs(int k, std::vector<double> M, std::vector<double>* theta, std::vector<double>* vectors) {
    std::vector<double> V(k * k, 0.0);
    for (int i = 0; i < k; ++i) V[i + i * k] = 1.0;
    for (int sweep = 0; sweep < 100; ++sweep) {
        double off = 0.0, tot = 0.0;
        for (int i = 0; i < k; ++i)
            for (int j = 0; j < k; ++j) (i == j ? tot : off) += M[i + j * k] * M[i + j * k];
        if (off <= 1e-26 * (tot + off) || off == 0.0) break;
        for (int p = 0; p < k; ++p)
            for (int q = p + 1; q < k; ++q) {
                const double apq = M[p + q * k];
                if (apq == 0.0) continue;
                const double tau = (M[q + q * k] - M[p + p * k]) / (2.0 * apq);
                const double t = (tau >= 0 ? 1.0 : -1.0) / (std::fabs(tau) + std::hypot(1.0, tau));
                const double c = 1.0 / std::sqrt(1.0 + t * t), s = t * c;
                for (int r = 0; r < k; ++r) {
                    const double mp = M[r + p * k], mq = M[r + q * k];
                    M[r + p * k] = c * mp - s * mq;
                    M[r + q * k] = s * mp + c * mq;
                }
                for (int r = 0; r < k; ++r) {
                    const double mp = M[p + r * k], mq = M[q + r * k];
                    M[p + r * k] = c * mp - s * mq;
                    M[q + r * k] = s * mp + c * mq;
                }
                for (int r = 0; r < k; ++r) {
                    const double vp = V[r + p * k], vq = V[r + q * k];
                    V[r + p * k] = c * vp - s * vq;
                    V[r + q * k] = s * vp + c * vq;
                }
            }
    }
    std::vector<int> order(k);
    for (int i = 0; i < k; ++i) order[i] = i;
    std::sort(order.begin(), order.end(), [&](int a, int b) { return M[a + a * k] < M[b + b * k]; });
    theta->resize(k);
    vectors->resize((size_t)k * k);
    for (int j = 0; j < k; ++j) {
        (*theta)[j] = M[order[j] + order[j] * k];
        std::copy(&V[(size_t)order[j] * k], &V[(size_t)order[j] * k] + k, &(*vectors)[(size_t)j * k]);
    }
}

// The projected problem A y = theta B y in the basis that orthonormalizes B, extended a row at a
// time: B = L L^T, C = L^-1 (rows: the orthonormal vectors in basis coefficients), M = C A C^T.
struct Projected {
    int k = 0;
    std::vector<double> C, M;  // kMaxSubspace x kMaxSubspace
    LowestPair pair;

    Projected() : C(kMaxSubspace * kMaxSubspace, 0.0), M(kMaxSubspace * kMaxSubspace, 0.0) {}
    double& c(int i, int j) { return C[i * kMaxSubspace + j]; }  // row i
    double& m(int i, int j) { return M[i * kMaxSubspace + j]; }

    // a[i], b[i] (i < k), a[k], b[k]: products of the new vector with the basis and itself
    bool append(const double* a, const double* b) {
        double at[kMaxSubspace], bt[kMaxSubspace];
        for (int i = 0; i < k; ++i) {
            double x = 0.0, y = 0.0;
            for (int j = 0; j <= i; ++j) {
                x += c(i, j) * a[j];
                y += c(i, j) * b[j];
            }
            at[i] = x;
            bt[i] = y;
        }
        double rho2 = b[k], mkk = a[k];
        for (int i = 0; i < k; ++i) rho2 -= bt[i] * bt[i];
        if (!(rho2 > 0.0)) return false;
        const double inv = 1.0 / std::sqrt(rho2);
        for (int j = 0; j < k; ++j) {
            double x = 0.0, mb = 0.0;
            for (int i = j; i < k; ++i) x -= bt[i] * c(i, j);
            for (int i = 0; i < k; ++i) mb += m(j, i) * bt[i];
            c(k, j) = x * inv;
            m(k, j) = m(j, k) = (at[j] - mb) * inv;
            mkk += bt[j] * (mb - 2.0 * at[j]);
        }
        c(k, k) = inv;
        m(k, k) = mkk * inv * inv;
        ++k;
        return true;
    }

    // coefficient vector y = C^T q of a vector in the orthonormal basis
    void to_basis(const double* q, double* y) {
        for (int p = 0; p < k; ++p) y[p] = 0.0;
        for (int i = 0; i < k; ++i)
            for (int p = 0; p <= i; ++p) y[p] += c(i, p) * q[i];
    }

    // the lowest pair (and, in pair.theta[1], the second root)
    double lowest(double* y) {
        pair.solve(k, M, kMaxSubspace);
        to_basis(pair.q.data(), y);
        return pair.theta[0];
    }

    // the `keep` lowest roots and their coefficient vectors (columns of y, k x keep)
    void lowest_many(int keep, std::vector<double>* theta, std::vector<double>* y) {
        std::vector<double> A((size_t)k * k), q;
        for (int j = 0; j < k; ++j)
            for (int i = 0; i < k; ++i) A[i + (size_t)j * k] = m(i, j);
        symmetric_eigs(k, std::move(A), theta, &q);
        y->resize((size_t)k * keep);
        for (int j = 0; j < keep; ++j) to_basis(&q[(size_t)j * k], &(*y)[(size_t)j * k]);
    }

    void restart(int keep, const std::vector<double>& theta) {
        k = keep;
        for (int i = 0; i < keep; ++i)
            for (int j = 0; j < keep; ++j) {
                c(i, j) = i == j ? 1.0 : 0.0;
                m(i, j) = i == j ? theta[i] : 0.0;
            }
    }
};

}  // namespace
}  // namespace vbcore

using namespace vbcore;

extern "C" vb_status vb_lowest_root(vb_context* ctx, const double* H, const double* S, int n, int mem_space,
                                    double tolerance, int max_iterations, double* eigenvalue, double* eigenvector,
                                    int* iterations) {
    if (!ctx) return VB_ERR_INVALID;
    if (n < 1 || !H || !S || !eigenvalue || !eigenvector)
        return set_error(ctx, VB_ERR_INVALID, "vb_lowest_root: bad arguments");
    if (mem_space != VB_MEM_HOST && mem_space != VB_MEM_DEVICE) return set_error(ctx, VB_ERR_INVALID, "bad memory space");
    cudaSetDevice(ctx->device);
    cudaStream_t s = ctx->stream;
    const size_t m2 = sizeof(double) * (size_t)n * n, v1 = sizeof(double) * n;
    const bool host = mem_space == VB_MEM_HOST;
    const int kmax = std::min(kMaxSubspace, n);
    const int splits = gemv_splits(n);
    const int blocks = (n + kRows - 1) / kRows;
    // (the partial dot products' room also takes the coefficients of a thick restart)
    const size_t partials = std::max<size_t>((size_t)blocks * kDotsMax, (size_t)kMaxSubspace * kKeep);
    // workspace: [H S (host mode)] V HV SV (n x kmax) parts (2 x splits x n) vectors (8 n), per-CTA
    // dot products, their sums (images, Ritz, orthogonalization) and the CTA counter
    const size_t ws_doubles = (host ? 2 * (size_t)n * n : 0) + 3 * (size_t)n * kmax + 2 * (size_t)splits * n +
                              8 * (size_t)n + partials + 3 * kDotsMax + 2 + 3 * (size_t)kKeep * n;
    DeviceBuffer ws;
    vb_status st = ws.allocate(ctx, sizeof(double) * ws_doubles);
    if (st != VB_OK) return st;
    double* base = ws.as<double>();
    const double* dH = H;
    const double* dS = S;
    cudaError_t err = cudaSuccess;
    if (host) {
        err = cudaMemcpyAsync(base, H, m2, cudaMemcpyHostToDevice, s);
        if (err == cudaSuccess) err = cudaMemcpyAsync(base + (size_t)n * n, S, m2, cudaMemcpyHostToDevice, s);
        dH = base;
        dS = base + (size_t)n * n;
        base += 2 * (size_t)n * n;
    }
    auto take = [&](size_t count) {
        double* at = base;
        base += count;
        return at;
    };
    double* V = take((size_t)n * kmax);
    double* HV = take((size_t)n * kmax);
    double* SV = take((size_t)n * kmax);
    double* ph = take((size_t)splits * n);
    double* ps = take((size_t)splits * n);
    double* hd = take(n);
    double* sd = take(n);
    double* x = take(n);
    double* r = take(n);
    double* t = take(n);    // correction before its second orthogonalization
    double* t2 = take(n);   // and after it
    double* ht = take(n);   // H t2, S t2
    double* stv = take(n);
    double* partial = take(partials);
    // sums: [images (2 k + 2) | Ritz norms (3) and first pass (k)] read back together, second pass
    double* sums = take(2 * kDotsMax);
    double* ritz_out = sums + kDotsMax;
    double* second = take(kDotsMax);
    unsigned* counter = reinterpret_cast<unsigned*>(take(2));
    double* restart = take(3 * (size_t)kKeep * n);
    double* back = static_cast<double*>(context_pinned(ctx, &st));
    if (!back) return st;
    const int tb = 256, nb = (n + tb - 1) / tb;
    auto check = [&](const char* what) -> vb_status {
        if (err == cudaSuccess) err = cudaGetLastError();
        if (err != cudaSuccess) return cuda_error(ctx, err, what);
        return VB_OK;
    };
    // sums (images and Ritz parts) to the host
    auto read_back = [&]() -> vb_status {
        if (err == cudaSuccess)
            err = cudaMemcpyAsync(back, sums, sizeof(double) * 2 * kDotsMax, cudaMemcpyDeviceToHost, s);
        if (err == cudaSuccess) err = cudaStreamSynchronize(s);
        return check("vb_lowest_root");
    };
    const double* norms = back + kDotsMax;
    if (err == cudaSuccess) err = cudaMemsetAsync(counter, 0, sizeof(unsigned), s);
    diag_kernel<<<nb, tb, 0, s>>>(n, dH, dS, hd, sd);
    start_kernel<<<1, 1024, 0, s>>>(n, hd, sd, t);
    int k = 0;
    Projected proj;
    double theta = 0.0, scale = 1.0;
    std::vector<double> y, ritz;  // ritz: lowest Ritz value of every iteration
    bool converged = false;
    DeviceBuffer mbuf, uibuf;
    double* Ui = nullptr;
    int it = 0;  // Ritz pairs formed
    auto is_converged = [&]() {
        return std::sqrt(norms[2]) <= tolerance * (std::sqrt(norms[0]) + std::fabs(theta) * std::sqrt(norms[1]));
    };
    for (;;) {
        // images of the new direction and its products with the basis
        gemv2_partial_kernel<<<dim3(nb, splits), tb, 0, s>>>(dH, dS, n, t, V, k, k > 0 ? second : nullptr, t2, ph, ps);
        images_kernel<<<blocks, kVecThreads, 0, s>>>(n, k, splits, ph, ps, V, t2, ht, stv, partial, sums, counter);
        if ((st = read_back()) != VB_OK) return st;
        if (it > 0 && is_converged()) {
            converged = true;
            break;
        }
        if (it >= max_iterations) break;
        const double norm2 = back[2 * k + 1];  // t^T S t
        if (it > 0 && !(norm2 > 1e-28)) break;  // no new direction
        const double inv = 1.0 / std::sqrt(norm2);
        double a[kMaxSubspace + 1], b[kMaxSubspace + 1];
        for (int i = 0; i < k; ++i) {
            a[i] = back[i] * inv;
            b[i] = back[k + 1 + i] * inv;
        }
        a[k] = back[k] * inv * inv;
        b[k] = norm2 * inv * inv;
        if (!proj.append(a, b))
            return set_error(ctx, VB_ERR_NUMERIC, "vb_lowest_root: projected overlap is not positive definite");
        ++k;
        Coefficients yc{};
        theta = proj.lowest(yc.v);
        ritz.push_back(theta);
        scale = std::max(1.0, std::fabs(theta));
        ritz_kernel<<<blocks, kVecThreads, 0, s>>>(n, k, yc, inv, theta, Ui == nullptr, V, HV, SV, t2, ht, stv, hd, sd, x,
                                                   r, t, partial, ritz_out, counter);
        ++it;
        const bool new_shift = !Ui && it >= kDiagonalPhase;
        if (new_shift || k == kmax) {
            if ((st = read_back()) != VB_OK) return st;
            if (is_converged()) {
                converged = true;
                break;
            }
        }
        if (new_shift) {
            // switch to the shift-invert preconditioner (H - sigma S)^-1 with sigma below the
            // lowest root: the factorization only holds (positive definite) there
            // shift below the root: by default from the residual, which overstates the distance to
            // the root by orders of magnitude on non-orthogonal structures (a shift far below it
            // leaves a weak preconditioner); when the Ritz values of the last eight iterations
            // decrease at a slowing rate, the root is estimated by Aitken's delta-squared
            // extrapolation of theta_{it-8}, theta_{it-4}, theta_it and the shift is 1.5 times the
            // estimated distance plus a tenth of the Ritz gap.  A shift that proves to lie above the
            // root fails the factorization and is widened below.
            double delta = std::max(1.0e-2 * scale, 10.0 * std::sqrt(norms[2]));
            const size_t nr = ritz.size();
            if (nr > 8) {
                const double d1 = ritz[nr - 5] - ritz[nr - 9], d2 = ritz[nr - 1] - ritz[nr - 5];
                if (d1 < 0.0 && d2 < 0.0 && d2 > d1) {
                    const double below = d2 * d2 / (d2 - d1);  // theta - estimated root
                    const double gap = k > 1 ? proj.pair.theta[1] - theta : 0.0;
                    delta = 1.5 * below + std::max(0.1 * gap, 1.0e-4 * scale);
                }
            }
            if ((st = mbuf.allocate(ctx, m2)) != VB_OK) return st;
            if ((st = uibuf.allocate(ctx, m2)) != VB_OK) return st;
            int info = 1;
            for (int attempt = 0; attempt < 16 && info != 0; ++attempt) {
                const long long count = (long long)n * n;
                shift_kernel<<<(unsigned)std::min<long long>(4096, (count + 255) / 256), 256, 0, s>>>(
                    count, dH, dS, theta - delta, mbuf.as<double>());
                if ((st = check("vb_lowest_root")) != VB_OK) return st;
                if ((st = factor_inverse_device(ctx, mbuf.as<double>(), n, uibuf.as<double>(), &info)) != VB_OK)
                    return st;
                if (info != 0) delta *= 4.0;
            }
            if (info != 0) return set_error(ctx, VB_ERR_NUMERIC, "vb_lowest_root: no positive-definite shift found");
            Ui = uibuf.as<double>();
        }
        if (Ui) {
            // t = U^-1 U^-T r, its column-range sums added up below
            gemv_t_kernel<<<(n * 32 + 255) / 256, 256, 0, s>>>(Ui, n, r, ht);
            gemv_partial_kernel<<<dim3(nb, splits), tb, 0, s>>>(Ui, n, ht, ph);
        }
        bool first_pass = !Ui;  // the Ritz kernel formed the first pass's products
        if (k == kmax) {
            // thick restart: the kKeep lowest Ritz vectors (S-orthonormal) and their images
            const int keep = std::min(kKeep, k);
            std::vector<double> kept;
            proj.lowest_many(keep, &kept, &y);
            err = cudaMemcpyAsync(partial, y.data(), sizeof(double) * k * keep, cudaMemcpyHostToDevice, s);
            restart_kernel<<<dim3(nb, 3 * keep), tb, 0, s>>>(n, k, keep, V, (long long)n * kmax, partial, restart);
            double* const into[3] = {V, HV, SV};
            for (int m = 0; m < 3 && err == cudaSuccess; ++m)
                err = cudaMemcpyAsync(into[m], restart + (size_t)m * keep * n, v1 * keep, cudaMemcpyDeviceToDevice, s);
            if ((st = check("vb_lowest_root")) != VB_OK) return st;
            proj.restart(keep, kept);
            k = keep;
            first_pass = false;
        }
        // S-orthogonalize the correction t against the basis, twice: V^T S t = (S V)^T t (S is
        // symmetric), so the coefficients come from the stored images S V without a pass over S.
        // The second pass is applied where the next pass over H and S reads t.
        if (!first_pass)
            orthogonalize_kernel<<<blocks, kVecThreads, 0, s>>>(n, k, V, SV, Ui ? ph : nullptr, splits, nullptr, t,
                                                                partial, ritz_out + 3, counter);
        orthogonalize_kernel<<<blocks, kVecThreads, 0, s>>>(n, k, V, SV, nullptr, 0, ritz_out + 3, t, partial, second,
                                                            counter);
        if ((st = check("vb_lowest_root")) != VB_OK) return st;
    }
    if (iterations) *iterations = converged ? it - 1 : it;
    *eigenvalue = theta;
    if (host)
        err = cudaMemcpyAsync(eigenvector, x, v1, cudaMemcpyDeviceToHost, s);
    else
        err = cudaMemcpyAsync(eigenvector, x, v1, cudaMemcpyDeviceToDevice, s);
    if (err == cudaSuccess) err = cudaStreamSynchronize(s);
    if (err != cudaSuccess) return cuda_error(ctx, err, "vb_lowest_root");
    if (!converged) return set_error(ctx, VB_ERR_NUMERIC, "vb_lowest_root: no convergence within the iteration limit");
    return VB_OK;
}
