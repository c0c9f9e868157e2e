// All roots of a generalized problem of moderate size (33 <= n <= 160) through a tridiagonal form:
// the dense solver's path between the one-warp Jacobi (n <= 32) and the cooperative block Jacobi.
//
//   S = U^T U and U^-1                      blocked Cholesky (cholesky_blocked.cu)
//   A = U^-T H U^-1                         td_product (16 x 16 tiles, one warp each, FP64 tensor cores)
//   A = P T P^T, T tridiagonal              td_reduce (four CTAs, the matrix in registers)
//   T z = lambda z, x = P z                 td_vectors (one warp per root: 32-way section of the
//                                           spectrum on Sturm counts, inverse iteration, reflectors)
//   close roots                             td_clusters (modified Gram-Schmidt inside clusters)
//   X <- X (3 I - X^T X) / 2, C = U^-1 X    td_product
// The last step takes vectors that inverse iteration left orthogonal to eps ||T|| / gap, at most
// 1e-9 outside clusters, to rounding (the Newton step toward the nearest orthogonal matrix).
// Whatever is not settled (a cluster whose vectors do not separate) is reported and solved by Jacobi.
//
// What bounds it: chains (n reflectors, 11 sections, two triangular solves), not work: 9 n^3 is
// 20 MFLOP at n = 132.  The block Jacobi took eight sweeps of nine rounds with two grid barriers
// and a 32 x 32 inner sweep each: 3.23 ms at n = 132 against 0.64 ms here (reduction 0.22, vectors
// 0.17, Cholesky and inverse 0.13).
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math.h>

#include "eigh_tridiagonal.h"
#include "internal.h"

namespace vbcore {
namespace {

constexpr int kMaxN = kTridiagonalMax;  // 160
constexpr int kCols = kMaxN / 32;       // columns per lane (5)
constexpr int kReduceCtas = 4, kReduceWarps = 8;  // 32 warps in the cluster, five rows each
constexpr double kClusterGap = 1.0e-5;       // of ||T||: closer roots are orthogonalized explicitly

__device__ __forceinline__ void mma_8x8x4(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One exchange of a sum over lanes of several values: each lane keeps H of its first 2 H, added to its
// partner's.
template <int H>
__device__ __forceinline__ void halve(double (&p)[kCols], bool up, int o) {
#pragma unroll
    for (int i = 0; i < H; ++i) {
        const double keep = up ? p[i + H] : p[i], send = up ? p[i] : p[i + H];
        p[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
}

// 16 x 16 tiles of C = op(A) op(B), one warp per CTA (all n x n, column-major):
//   0: T = H Ui           (H from its upper triangle, Ui upper)
//   1: A = Ui^T T         (tiles on or above the diagonal, mirrored)
//   2: G = X^T X          (likewise); status bit 1 when |G - I| > 0.1 somewhere
//   3: Y = X (3 I - G) / 2
//   4: C = Ui Y
// 3 and 4 only when everything is settled: C may lie over H or S, which Jacobi then still needs.
template <int MODE>
__global__ void __launch_bounds__(32) td_product(int n, const double* __restrict__ A, const double* __restrict__ B,
                                                 double* __restrict__ C, int* __restrict__ status) {
    const int lane = threadIdx.x, gr = lane >> 2, gc = lane & 3;
    const int r0 = 16 * blockIdx.x, c0 = 16 * blockIdx.y;
    constexpr bool kMirror = MODE == 1 || MODE == 2;
    if (MODE >= 3 && *status != 0) return;
    if (kMirror && r0 > c0) return;
    const long long ld = n;
    auto a_elem = [&](int r, int k) -> double {
        if (r >= n || k >= n) return 0.0;
        if (MODE == 0) return r <= k ? __ldg(A + r + k * ld) : __ldg(A + k + r * ld);
        if (MODE == 1) return k <= r ? __ldg(A + k + r * ld) : 0.0;
        if (MODE == 2) return __ldg(A + k + r * ld);
        if (MODE == 3) return __ldg(A + r + k * ld);
        return r <= k ? __ldg(A + r + k * ld) : 0.0;
    };
    auto b_elem = [&](int k, int c) -> double {
        if (c >= n || k >= n) return 0.0;
        if (MODE == 0) return k <= c ? __ldg(B + k + c * ld) : 0.0;
        if (MODE == 3) {
            const double g = -0.5 * __ldg(B + k + c * ld);
            return k == c ? 1.5 + g : g;
        }
        return __ldg(B + k + c * ld);
    };
    // k range the triangular operand leaves
    const int kb = MODE == 4 ? r0 : 0;
    const int ke = MODE == 0 ? min(n, c0 + 16) : (MODE == 1 ? min(n, r0 + 16) : n);
    double acc[2][2][2] = {};
    for (int k0 = kb; k0 < ke; k0 += 16) {
        double a[4][2], b[4][2];
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                a[q][i] = a_elem(r0 + 8 * i + gr, k0 + 4 * q + gc);
                b[q][i] = b_elem(k0 + 4 * q + gc, c0 + 8 * i + gr);
            }
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) mma_8x8x4(acc[i][j], a[q][i], b[q][j]);
    }
    bool far = false;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = r0 + 8 * i + gr, c = c0 + 8 * j + 2 * gc + h;
                if (r >= n || c >= n) continue;
                const double v = acc[i][j][h];
                if (kMirror && r > c) continue;
                C[r + c * ld] = v;
                if (kMirror && r < c) C[c + r * ld] = v;
                if (MODE == 2 && !(fabs(v - (r == c ? 1.0 : 0.0)) <= 0.1)) far = true;
            }
    if (MODE == 2 && far) atomicOr(status, 2);
}

// Householder reduction by a cluster of four CTAs.  Warp q of the cluster's 32 holds rows q + 32 i, lane
// l columns l + 32 j of the full symmetric matrix in registers.  Step s: the reflector I - tau v v^T
// that takes row s to e[s] e_{s+1}; every warp forms v and the scalars itself (from the same values in
// the same order), p = A v and the next row before its update go to all four CTAs' shared memory,
// one cluster barrier, then A -= v w^T + w v^T with w = tau p - (tau^2 v^T p / 2) v, and every warp
// updates the next row for itself.  The matrix is scaled by a power of two to a largest element in [1, 2)
// (squares neither overflow nor vanish at any scale of H); diag and off are left scaled, the exponent goes
// to tau[n].  Bound by the chain of n steps (barrier, two warp sums, a square
// root, two divisions): 222 us at n = 132, 555 us in one CTA of 20 warps, where the matrix spilled.
__global__ void __cluster_dims__(kReduceCtas, 1, 1) __launch_bounds__(32 * kReduceWarps, 1)
    td_reduce(int n, const double* __restrict__ A, double* __restrict__ diag, double* __restrict__ off,
              double* __restrict__ tau_out, double* __restrict__ V) {
    __shared__ double s_p[2][kMaxN], s_row[2][kMaxN];  // alternating by step: one barrier is enough
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int lane = threadIdx.x & 31, rank = (int)cluster.block_rank();
    const int base = rank * kReduceWarps + (threadIdx.x >> 5);  // this warp's first row, the lane of its columns
    double a[kCols][kCols];
#pragma unroll
    for (int i = 0; i < kCols; ++i)
#pragma unroll
        for (int j = 0; j < kCols; ++j) {
            const int r = base + 32 * i, c = lane + 32 * j;
            a[i][j] = (r < n && c < n) ? __ldg(A + r + (long long)c * n) : 0.0;
        }
    double x[kCols];  // row s
#pragma unroll
    for (int j = 0; j < kCols; ++j) x[j] = lane + 32 * j < n ? __ldg(A + (long long)(lane + 32 * j) * n) : 0.0;
    double big = 0.0;
#pragma unroll
    for (int i = 0; i < kCols; ++i)
#pragma unroll
        for (int j = 0; j < kCols; ++j) big = fmax(big, fabs(a[i][j]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
    __shared__ double s_big[kReduceWarps];
    if (lane == 0) s_big[threadIdx.x >> 5] = big;
    cluster.sync();  // no CTA addresses another one's shared memory before that one runs
    for (int i = lane; i < kReduceCtas * kReduceWarps; i += 32)
        big = fmax(big, cluster.map_shared_rank(s_big, i / kReduceWarps)[i % kReduceWarps]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
    const int exponent = big > 0.0 && isfinite(big) ? ilogb(big) : 0;
#pragma unroll
    for (int j = 0; j < kCols; ++j) {
        x[j] = scalbn(x[j], -exponent);
#pragma unroll
        for (int i = 0; i < kCols; ++i) a[i][j] = scalbn(a[i][j], -exponent);
    }
    if (base == 0 && lane == 0) tau_out[n] = (double)exponent;
    // one of five registers, without a dynamic index
    auto pick = [](int q, double y0, double y1, double y2, double y3, double y4) {
        return q < 2 ? (q == 0 ? y0 : y1) : (q == 2 ? y2 : (q == 3 ? y3 : y4));
    };
    // element c of a vector spread over lanes and registers
    auto element = [&](const double (&v)[kCols], int c) {
        return __shfl_sync(0xffffffffu, pick(c >> 5, v[0], v[1], v[2], v[3], v[4]), c & 31);
    };
    for (int s = 0; s + 2 < n; ++s) {
        double v[kCols], part = 0.0;
#pragma unroll
        for (int j = 0; j < kCols; ++j) {
            const int c = lane + 32 * j;
            v[j] = c > s ? x[j] : 0.0;
            if (c > s + 1) part = fma(v[j], v[j], part);
        }
        const double norm2 = warp_sum(part);
        const double x1 = element(x, s + 1);
        double beta = x1, tau = 0.0;
        if (norm2 > 0.0) {
            const double norm = sqrt(fma(x1, x1, norm2));
            beta = x1 > 0.0 ? -norm : norm;
            const double v1 = x1 - beta;
            tau = 2.0 / fma(v1, v1, norm2);
#pragma unroll
            for (int j = 0; j < kCols; ++j)
                if (lane + 32 * j == s + 1) v[j] = v1;
        }
        if (base == 0) {
#pragma unroll
            for (int j = 0; j < kCols; ++j) {
                if (lane + 32 * j < n) V[(long long)s * n + lane + 32 * j] = v[j];
                if (lane + 32 * j == s) {
                    diag[s] = x[j];
                    off[s] = beta;
                    tau_out[s] = tau;
                }
            }
        }
        // p = A v for this warp's rows: four by halving exchanges, the fifth by a plain sum
        double p[kCols];
#pragma unroll
        for (int i = 0; i < kCols; ++i) {
            double acc = 0.0;
#pragma unroll
            for (int j = 0; j < kCols; ++j) acc = fma(a[i][j], v[j], acc);
            p[i] = base + 32 * i > s ? acc : 0.0;
        }
        static_assert(kCols == 5, "two halving exchanges and one sum");
        halve<2>(p, lane & 16, 16);
        halve<1>(p, lane & 8, 8);
        double p03 = p[0];
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) p03 += __shfl_xor_sync(0xffffffffu, p03, o);
        const double p4 = warp_sum(p[4]);
        const int buf = s & 1, to = lane & 7;
        if (to < kReduceCtas) {  // eight lanes hold each sum: one per destination
            double* peer = cluster.map_shared_rank(s_p[buf], to);
            peer[base + 32 * (((lane >> 4) & 1) * 2 + ((lane >> 3) & 1))] = p03;
            if (lane < 8) peer[base + 128] = p4;
        }
        if (base == ((s + 1) & 31)) {
#pragma unroll
            for (int j = 0; j < kCols; ++j) {
                const double y = pick((s + 1) >> 5, a[0][j], a[1][j], a[2][j], a[3][j], a[4][j]);
#pragma unroll
                for (int t = 0; t < kReduceCtas; ++t) cluster.map_shared_rank(s_row[buf], t)[lane + 32 * j] = y;
            }
        }
        cluster.sync();
        double w[kCols], dot = 0.0;
#pragma unroll
        for (int j = 0; j < kCols; ++j) {
            w[j] = s_p[buf][lane + 32 * j];
            dot = fma(w[j], v[j], dot);
        }
        const double half = 0.5 * tau * tau * warp_sum(dot);
#pragma unroll
        for (int j = 0; j < kCols; ++j) w[j] = fma(tau, w[j], -half * v[j]);
#pragma unroll
        for (int i = 0; i < kCols; ++i) {
            if (base + 32 * i <= s || base + 32 * i >= n) continue;
            const double vr = __shfl_sync(0xffffffffu, v[i], base), wr = __shfl_sync(0xffffffffu, w[i], base);
#pragma unroll
            for (int j = 0; j < kCols; ++j) a[i][j] = fma(-vr, w[j], fma(-wr, v[j], a[i][j]));
        }
        const double v1 = element(v, s + 1), w1 = element(w, s + 1);
#pragma unroll
        for (int j = 0; j < kCols; ++j) x[j] = fma(-v1, w[j], fma(-w1, v[j], s_row[buf][lane + 32 * j]));
    }
    // the last 2 x 2 block
#pragma unroll
    for (int j = 0; j < kCols; ++j) {
        const int c = lane + 32 * j;
        if (base == 0 && c == n - 2) diag[c] = x[j];
        if (base == 0 && c == n - 1) off[n - 2] = x[j];
#pragma unroll
        for (int i = 0; i < kCols; ++i)
            if (base + 32 * i == n - 1 && c == n - 1) diag[c] = a[i][j];
    }
    cluster.sync();  // no CTA leaves while another may still write to its shared memory
}

// Root blockIdx.x (ascending) and its vector, one warp.  The spectrum (Gershgorin interval, scaled to
// norm 1) is cut into 33 by 32 Sturm counts per round: the sequence p_i = (d_i - x) p_{i-1} -
// e_{i-1}^2 p_{i-2} is the exact one of a matrix with relative perturbations eps in d_i - x and
// e^2, so the counts are as good as those of the quotient form without its divisions.  Then two
// inverse iterations (lane 0; LU with row exchanges) and the reflectors, last to first.
__global__ void __launch_bounds__(32) td_vectors(int n, const double* __restrict__ diag, const double* __restrict__ off,
                                                 const double* __restrict__ tau, const double* __restrict__ V,
                                                 double* __restrict__ values, double* __restrict__ X,
                                                 double* __restrict__ norm_out) {
    __shared__ double sd[kMaxN], se[kMaxN], se2[kMaxN], sx[kMaxN];
    __shared__ double ud[kMaxN], ue[kMaxN], uf[kMaxN], ul[kMaxN];
    __shared__ unsigned char sw[kMaxN];
    const int lane = threadIdx.x, j = blockIdx.x;
    double lo = INFINITY, hi = -INFINITY;
    for (int i = lane; i < n; i += 32) {
        const double d = __ldg(diag + i), e0 = i > 0 ? fabs(__ldg(off + i - 1)) : 0.0;
        const double e1 = i + 1 < n ? fabs(__ldg(off + i)) : 0.0;
        lo = fmin(lo, d - (e0 + e1));
        hi = fmax(hi, d + (e0 + e1));
        sd[i] = d;
        se[i] = i + 1 < n ? __ldg(off + i) : 0.0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    const double norm = fmax(fmax(fabs(lo), fabs(hi)), 1e-280);
    const int exponent = (int)__ldg(tau + n);
    const double inv = 1.0 / norm;
    for (int i = lane; i < n; i += 32) {
        sd[i] *= inv;
        se[i] *= inv;
        se2[i] = se[i] * se[i];
    }
    __syncwarp();
    lo = lo * inv - 4e-16;
    hi = hi * inv + 4e-16;
    for (int round = 0; round < 13 && hi - lo > 2.3e-16; ++round) {
        const double width = hi - lo;
        const double x = fma(width, (double)(lane + 1) / 33.0, lo);
        // eigenvalues below x: sign changes of the sequence
        // (a zero becomes a tiny value of the sign opposite to its predecessor's: a relative change
        // of 1e-25 in d - x)
        double p0 = 1.0, p1 = sd[0] - x;
        if (p1 == 0.0) p1 = -1e-25;
        bool neg = p1 < 0.0;
        int count = neg ? 1 : 0;
        for (int i = 1; i < n; ++i) {
            double p = fma(sd[i] - x, p1, -se2[i - 1] * p0);
            if (p == 0.0) p = -1e-25 * p1;
            const bool s = p < 0.0;
            count += s != neg;
            neg = s;
            p0 = p1;
            p1 = p;
            if ((i & 7) == 7) {
                // keep the pair within range (its scale is free)
                const double big = fmax(fabs(p0), fabs(p1));
                if (big < 1e-100) {
                    p0 *= 1e150;
                    p1 *= 1e150;
                } else if (big > 1e100) {
                    p0 *= 1e-150;
                    p1 *= 1e-150;
                }
            }
        }
        const int below = __popc(__ballot_sync(0xffffffffu, count <= j));  // sections left of the root
        const double a = below == 0 ? lo : __shfl_sync(0xffffffffu, x, below > 0 ? below - 1 : 0);
        const double b = below == 32 ? hi : __shfl_sync(0xffffffffu, x, below < 32 ? below : 31);
        lo = a;
        hi = b;
    }
    const double lambda = 0.5 * (lo + hi);
    if (lane == 0) {
        values[j] = scalbn(lambda * norm, exponent);
        if (j == 0) *norm_out = scalbn(norm, exponent);
        const double tiny = 2.3e-16;
        auto away = [&](double v) { return fabs(v) < tiny ? (v < 0.0 ? -tiny : tiny) : v; };
        double cd = sd[0] - lambda, ce = se[0];
        for (int i = 0; i + 1 < n; ++i) {
            const double sub = se[i], nd = sd[i + 1] - lambda, ne = i + 2 < n ? se[i + 1] : 0.0;
            if (fabs(cd) >= fabs(sub)) {
                cd = away(cd);
                const double r = 1.0 / cd, l = sub * r;
                ud[i] = r;
                ue[i] = ce;
                uf[i] = 0.0;
                ul[i] = l;
                sw[i] = 0;
                cd = fma(-l, ce, nd);
                ce = ne;
            } else {
                const double r = 1.0 / sub, l = cd * r;
                ud[i] = r;
                ue[i] = nd;
                uf[i] = ne;
                ul[i] = l;
                sw[i] = 1;
                cd = fma(-l, nd, ce);
                ce = -l * ne;
            }
        }
        ud[n - 1] = 1.0 / away(cd);
        // start vector: entries in [0.5, 1.5], different for every root
        unsigned seed = 2654435761u * (unsigned)(j + 1);
        for (int i = 0; i < n; ++i) {
            seed = seed * 1664525u + 1013904223u;
            sx[i] = 0.5 + (double)(seed >> 8) * (1.0 / 16777216.0);
        }
        for (int pass = 0; pass < 3; ++pass) {
            if (pass > 0) {
                double x0 = sx[0];
                for (int i = 0; i + 1 < n; ++i) {
                    double x1 = sx[i + 1];
                    if (sw[i]) {
                        const double t = x0;
                        x0 = x1;
                        x1 = t;
                    }
                    sx[i] = x0;
                    x0 = fma(-ul[i], x0, x1);
                }
                sx[n - 1] = x0;
            }
            double y1 = 0.0, y2 = 0.0, big = 0.0;
            for (int i = n - 1; i >= 0; --i) {
                double v = sx[i];
                if (i + 1 < n) v = fma(-ue[i], y1, v);
                if (i + 2 < n) v = fma(-uf[i], y2, v);
                v *= ud[i];
                sx[i] = v;
                y2 = y1;
                y1 = v;
                big = fmax(big, fabs(v));
            }
            // keep the range for the next solve; the direction is all that counts
            const double r = 1.0 / big;
            for (int i = 0; i < n; ++i) sx[i] *= r;
        }
    }
    __syncwarp();
    double x[kCols], part = 0.0;
#pragma unroll
    for (int q = 0; q < kCols; ++q) {
        const int i = lane + 32 * q;
        x[q] = i < n ? sx[i] : 0.0;
        part = fma(x[q], x[q], part);
    }
    const double scale = 1.0 / sqrt(warp_sum(part));
#pragma unroll
    for (int q = 0; q < kCols; ++q) x[q] *= scale;
    double v[kCols], t = 0.0;
    auto load = [&](int s) {
#pragma unroll
        for (int q = 0; q < kCols; ++q) v[q] = lane + 32 * q < n ? __ldg(V + (long long)s * n + lane + 32 * q) : 0.0;
        t = __ldg(tau + s);
    };
    if (n > 2) load(n - 3);
    for (int s = n - 3; s >= 0; --s) {
        double u[kCols], dot = 0.0;
        const double ts = t;
#pragma unroll
        for (int q = 0; q < kCols; ++q) {
            u[q] = v[q];
            dot = fma(u[q], x[q], dot);
        }
        if (s > 0) load(s - 1);
        const double f = ts * warp_sum(dot);
#pragma unroll
        for (int q = 0; q < kCols; ++q) x[q] = fma(-f, u[q], x[q]);
    }
#pragma unroll
    for (int q = 0; q < kCols; ++q)
        if (lane + 32 * q < n) X[(long long)j * n + lane + 32 * q] = x[q];
}

// Modified Gram-Schmidt (twice) inside every run of roots closer than kClusterGap ||T||.  One CTA;
// status bit 0 when a vector nearly lies in the span of its predecessors.
__global__ void __launch_bounds__(1024) td_clusters(int n, const double* __restrict__ values,
                                                    const double* __restrict__ norm, double* __restrict__ X,
                                                    int* __restrict__ status) {
    __shared__ double red[32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const double gap = kClusterGap * *norm;
    auto block_dot = [&](double v) {
        v = warp_sum(v);
        __syncthreads();
        if (lane == 0) red[warp] = v;
        __syncthreads();
        double s = 0.0;
        for (int w = 0; w < (n + 31) / 32; ++w) s += red[w];
        return s;
    };
    int first = 0;
    for (int j = 1; j < n; ++j) {
        if (__ldg(values + j) - __ldg(values + j - 1) > gap) {
            first = j;
            continue;
        }
        double x = tid < n ? X[(long long)j * n + tid] : 0.0;
        for (int pass = 0; pass < 2; ++pass)
            for (int i = first; i < j; ++i) {
                const double y = tid < n ? X[(long long)i * n + tid] : 0.0;
                x = fma(-block_dot(x * y), y, x);
            }
        const double len2 = block_dot(x * x);
        if (!(len2 > 1e-6) && tid == 0) atomicOr(status, 1);
        if (tid < n) X[(long long)j * n + tid] = x * (1.0 / sqrt(len2));
        __syncthreads();
    }
}

}  // namespace

size_t tridiagonal_workspace_doubles(int n) { return 4 * (size_t)n * n + 4 * (size_t)n + 4; }

cudaError_t tridiagonal_eigh(const double* H, const double* Ui, int n, double* values, double* vectors, double* work,
                             int* status_host, cudaStream_t s) {
    const size_t m2 = (size_t)n * n;
    double* T = work;
    double* A = T + m2;
    double* V = A + m2;
    double* X = V + m2;
    double* diag = X + m2;
    double* off = diag + n;
    double* tau = off + n;
    double* norm = tau + 2 * n;
    int* status = reinterpret_cast<int*>(norm + 1);
    cudaError_t err = cudaMemsetAsync(status, 0, sizeof(int), s);
    if (err != cudaSuccess) return err;
    const dim3 tiles((n + 15) / 16, (n + 15) / 16);
    td_product<0><<<tiles, 32, 0, s>>>(n, H, Ui, T, status);
    td_product<1><<<tiles, 32, 0, s>>>(n, Ui, T, A, status);
    td_reduce<<<kReduceCtas, 32 * kReduceWarps, 0, s>>>(n, A, diag, off, tau, V);
    td_vectors<<<n, 32, 0, s>>>(n, diag, off, tau, V, values, X, norm);
    td_clusters<<<1, (n + 31) / 32 * 32, 0, s>>>(n, values, norm, X, status);
    td_product<2><<<tiles, 32, 0, s>>>(n, X, X, T, status);
    td_product<3><<<tiles, 32, 0, s>>>(n, X, T, A, status);
    td_product<4><<<tiles, 32, 0, s>>>(n, Ui, A, vectors, status);
    err = cudaGetLastError();
    if (err == cudaSuccess) err = cudaMemcpyAsync(status_host, status, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (err == cudaSuccess) err = cudaStreamSynchronize(s);
    return err;
}

}  // namespace vbcore
