// Blocked FP64 Cholesky factorization and triangular inverse on the FP64 tensor cores, as
// stream-ordered launches with no grid barrier (vb_metric_cholesky and the Davidson shift-invert
// preconditioner above the one-CTA size).
//
// Factorization M = U^T U (upper triangle of M read; Eigen::LLT / LAPACK dpotrf semantics: the
// first non-positive or non-finite pivot stops it with info = its order), right-looking over
// 64-column panels:
//   1. bc_panel_kernel (one CTA): the previous panel's update of the diagonal block, its Cholesky
//      factor and the inverse of that triangular block, in shared memory;
//   2. bc_panel_row_kernel: the previous panel's update of the row block A_12, then
//      U_12 = U_11^-T A_12;
//   3. bc_trailing_kernel: A_22 -= U_12^T U_12 over the upper 64 x 64 tiles from the row block after
//      the next one on.
// The chain of 1 and 2 bounds the factorization (n = 2048: 32 panels, 1.88 ms before the panel's
// pivots moved into one warp and the next panel's updates into these two kernels, 1.31 ms after it,
// 1.16 ms with the row kernel launched beside the panel kernel: its update needs earlier panels only); it
// runs on a high-priority auxiliary stream while the trailing updates run one panel behind it on
// the caller's stream.
// Inverse U^-1 (optional): the panel kernels leave U_JJ^-1 on the diagonal blocks; then for block
// sizes b = 64, 128, ... consecutive diagonal blocks are paired,
//   [[A, B], [0, C]]^-1 = [[A^-1, -A^-1 B C^-1], [0, C^-1]],
// every pair of a level at once: T = B C^-1 (bc_level_kernel<0>), then X = -A^-1 T
// (bc_level_kernel<1>).
// Products: 64 x 64 output tiles per CTA, 32-deep k-steps staged through shared memory (double
// buffered, the next step's loads in registers while the current one is multiplied), mma.sync
// m8n8k4 FP64.  Every launch first reads the status word and returns when a panel has failed.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

#include "internal.h"

namespace vbcore {
namespace {

constexpr int kNB = 64;         // panel width and output tile edge
constexpr int kKS = 32;         // k-step of a tile product
constexpr int kThreadsB = 256;  // eight warps: 16 x 32 of the output tile each
constexpr int kStrideKC = 36;   // [x][k] staging (k contiguous): 36 = 4 mod 16 doubles
constexpr int kStrideXC = 72;   // [k][x] staging (x contiguous): 72 = 8 mod 16 doubles
constexpr int kTileDoubles = kNB * kStrideKC;  // == kKS * kStrideXC
constexpr size_t kProductSmem = 4 * kTileDoubles * sizeof(double);

static_assert(kNB * kStrideKC == kKS * kStrideXC, "both staging layouts fill one tile buffer");

// Operand of a tile product: element (x, k) (x = row of A or column of B) at p[k + x ld] when the
// operand is k-contiguous, else at p[x + k ld]; x < xn and k < kn are read, the rest is zero.
struct Opnd {
    const double* p;
    long long ld;
    int xn, kn;
};

template <bool KC>
__device__ __forceinline__ void load_regs(const Opnd& o, int x0, int k0, double (&r)[8]) {
    const int t = threadIdx.x;
    if (KC) {
        const int k = k0 + (t & 31);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int x = x0 + (t >> 5) + 8 * i;
            r[i] = (x < o.xn && k < o.kn) ? o.p[k + (long long)x * o.ld] : 0.0;
        }
    } else {
        const int x = x0 + (t & 63);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int k = k0 + (t >> 6) + 4 * i;
            r[i] = (x < o.xn && k < o.kn) ? o.p[x + (long long)k * o.ld] : 0.0;
        }
    }
}

template <bool KC>
__device__ __forceinline__ void store_tile(double* s, const double (&r)[8]) {
    const int t = threadIdx.x;
    if (KC) {
        const int k = t & 31;
#pragma unroll
        for (int i = 0; i < 8; ++i) s[((t >> 5) + 8 * i) * kStrideKC + k] = r[i];
    } else {
        const int x = t & 63;
#pragma unroll
        for (int i = 0; i < 8; ++i) s[((t >> 6) + 4 * i) * kStrideXC + x] = r[i];
    }
}

template <bool KC>
__device__ __forceinline__ double frag(const double* s, int x, int k) {
    return KC ? s[x * kStrideKC + k] : s[k * kStrideXC + x];
}

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// acc += sum_{k in [kb, ke)} A(xa + r, k) B(k, xb + c) for the CTA's 64 x 64 output tile: warp w
// holds rows 16 (w % 4) .. + 15 and columns 32 (w / 4) .. + 31 as 2 x 4 fragments, lane element
// (row 8 i + lane / 4, column 8 j + 2 (lane % 4) + h) in acc[i][j][h].  kb < ke is uniform.
template <bool AKC, bool BKC>
__device__ void tile_product(Opnd A, Opnd B, int xa, int xb, int kb, int ke, double* smem,
                             double (&acc)[2][4][2]) {
    A.kn = min(A.kn, ke);
    B.kn = min(B.kn, ke);
    // buffers: A in [0, 2) and B in [2, 4) tile slots, alternating by k-step
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gr = lane >> 2, gc = lane & 3;
    const int wm = (warp & 3) * 16, wn = (warp >> 2) * 32;
    double ra[8], rb[8];
    load_regs<AKC>(A, xa, kb, ra);
    load_regs<BKC>(B, xb, kb, rb);
    store_tile<AKC>(smem, ra);
    store_tile<BKC>(smem + 2 * kTileDoubles, rb);
    __syncthreads();
    int buf = 0;
    for (int k0 = kb; k0 < ke; k0 += kKS) {
        const bool more = k0 + kKS < ke;
        if (more) {
            load_regs<AKC>(A, xa, k0 + kKS, ra);
            load_regs<BKC>(B, xb, k0 + kKS, rb);
        }
        const double* a = smem + buf * kTileDoubles;
        const double* b = smem + (2 + buf) * kTileDoubles;
#pragma unroll
        for (int kk = 0; kk < kKS; kk += 4) {
            double af[2], bf[4];
#pragma unroll
            for (int i = 0; i < 2; ++i) af[i] = frag<AKC>(a, wm + 8 * i + gr, kk + gc);
#pragma unroll
            for (int j = 0; j < 4; ++j) bf[j] = frag<BKC>(b, wn + 8 * j + gr, kk + gc);
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) dmma(acc[i][j], af[i], bf[j]);
        }
        if (more) {
            store_tile<AKC>(smem + (buf ^ 1) * kTileDoubles, ra);
            store_tile<BKC>(smem + (2 + (buf ^ 1)) * kTileDoubles, rb);
        }
        __syncthreads();
        buf ^= 1;
    }
}

// Output element (row, column) within the tile of acc[i][j][h].
__device__ __forceinline__ int out_row(int i) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    return (warp & 3) * 16 + 8 * i + (lane >> 2);
}
__device__ __forceinline__ int out_col(int j, int h) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    return (warp >> 2) * 32 + 8 * j + 2 * (lane & 3) + h;
}

__device__ __forceinline__ bool failed(const int* status) { return *(const volatile int*)status != 0; }

__global__ void bc_init_kernel(const double* __restrict__ M, double* __restrict__ U, int n) {
    const long long total = (long long)n * n;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const long long r = e % n, c = e / n;
        U[e] = r <= c ? M[e] : 0.0;
    }
}

// Panel j0: Cholesky of the (updated) 64 x 64 diagonal block and the inverse of its factor, one CTA;
// rows beyond the matrix are padded with the identity.  The serial chain of 64 pivots bounds it, so
// the chain runs inside one warp without barriers: 16 x 16 blocks, each factored and inverted by
// warp 0 in registers (panel_factor16: lane (h, c) holds rows 8 h .. 8 h + 7 of column c, the pivot
// row travels by shuffles), while the other warps still apply the previous block's rank-16 update;
// then U_12 = U_11^-T A_12 on the tensor cores.  Two barriers per 16 pivots.  The 64 x 64 inverse
// pairs the 16 x 16 ones (and then the 32 x 32 ones) as bc_level_kernel does.  n = 2048: 41 us a
// panel when every pivot was published through shared memory to 256 threads (64 + 64 barriers).
// Shared layout: column-major, stride 68 = 4 mod 16 doubles, so that the fragments of both operand
// orders load without bank conflicts.  Writes U_JJ into U, its inverse into Ub (64 x 64,
// column-major) and, when Ui is given, onto Ui's diagonal block.
constexpr int kPL = kNB + 4;  // column stride of the panel's shared blocks
constexpr int kPT = 36;       // column stride of the 32 x 32 scratch of the inverse
constexpr int kPW = kThreadsB / 32;
constexpr size_t kPanelSmem = sizeof(double) * (2 * kNB * kPL + 32 * kPT);

// Warp 0: the 16 x 16 block at sA (column-major, stride kPL; upper triangle) becomes its Cholesky
// factor (zeros below), sX its inverse.  Returns the order of the first failing pivot, 0 when there
// is none.  Entries below the diagonal carry values that no later step reads.
__device__ __forceinline__ int panel_factor16(double* sA, double* sX) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, h = lane >> 4, c = lane & 15;
    double v[8], mine = 1.0;
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = sA[c * kPL + 8 * h + i];
    int bad = 0;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const int src = (k >> 3) * 16, kk = k & 7;  // the lanes and register that hold row k
        const double p = __shfl_sync(full, v[kk], src + k);
        if (bad == 0 && (!(p > 0.0) || !isfinite(p))) bad = k + 1;  // the same decision in every lane
        if (c == k) mine = p;
        const double inv = 1.0 / p;
        const double x = __shfl_sync(full, v[kk], src + c);
        const double f = c > k ? x * inv : 0.0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (8 + i <= k) continue;  // no row left in either half
            const double q = __shfl_sync(full, v[kk], src + 8 * h + i);
            v[i] = fma(8 * h + i > k ? -q : 0.0, f, v[i]);
        }
    }
    if (bad) return bad;
    // rows scaled by 1 / sqrt(pivot); lane c holds pivot c
    const double d = sqrt(mine), di = 1.0 / d;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = 8 * h + i;
        const double dr = __shfl_sync(full, di, r);
        v[i] = r < c ? v[i] * dr : (r == c ? d : 0.0);
        sA[c * kPL + r] = v[i];
    }
    __syncwarp();
    // inverse, rows from the last up: X[k, :] = w[k, :] / u_kk, w[r, :] -= u_rk X[k, :] (r < k)
    double w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = 8 * h + i == c ? 1.0 : 0.0;
#pragma unroll
    for (int k = 15; k >= 0; --k) {
        const int src = (k >> 3) * 16, kk = k & 7;
        const double dk = __shfl_sync(full, di, k);
        const double xk = __shfl_sync(full, w[kk], src + c) * dk;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (i > k) continue;
            const int r = 8 * h + i;
            const double u = sA[k * kPL + r];  // zero below the diagonal
            w[i] = r < k ? fma(-u, xk, w[i]) : (r == k ? xk : w[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) sX[c * kPL + 8 * h + i] = w[i];
    __syncwarp();
    return 0;
}

// One 8 x 8 tile of A - U_12^T U_12 over the 16 rows k0 .. k0 + 15 at (r0, c0), in place.
__device__ __forceinline__ void panel_update_tile(double* sA, int k0, int r0, int c0) {
    const int lane = threadIdx.x & 31, gr = lane >> 2, gc = lane & 3;
    double acc[2] = {0.0, 0.0};
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
        dmma(acc, sA[(r0 + gr) * kPL + k0 + 4 * ks + gc], sA[(c0 + gr) * kPL + k0 + 4 * ks + gc]);
#pragma unroll
    for (int i = 0; i < 2; ++i) sA[(c0 + 2 * gc + i) * kPL + r0 + gr] -= acc[i];
}

// One 8 x 8 tile (row r0, column c0) of s A B, A(i, k) at a[k la + i], B(k, j) at b[j lb + k], over
// k in [kb, ke).
__device__ __forceinline__ void panel_product_tile(const double* a, int la, const double* b, int lb, int r0, int c0,
                                                   int kb, int ke, double s, double* out, int lo) {
    const int lane = threadIdx.x & 31, gr = lane >> 2, gc = lane & 3;
    double acc[2] = {0.0, 0.0};
    for (int k = kb; k < ke; k += 4) dmma(acc, a[(k + gc) * la + r0 + gr], b[(c0 + gr) * lb + k + gc]);
#pragma unroll
    for (int i = 0; i < 2; ++i) out[(c0 + 2 * gc + i) * lo + r0 + gr] = s * acc[i];
}

__global__ void __launch_bounds__(kThreadsB) bc_panel_kernel(double* __restrict__ U, double* __restrict__ Ub,
                                                             double* __restrict__ Ui, int n, int j0, int* status) {
    extern __shared__ __align__(16) double psm[];
    double* sA = psm;               // the block, then its factor
    double* sX = psm + kNB * kPL;   // the inverse
    double* sT = sX + kNB * kPL;    // scratch of the inverse
    __shared__ int s_bad;
    // the row kernel of this panel may start its own update (it waits for this kernel's results)
    asm volatile("griddepcontrol.launch_dependents;");
    if (failed(status)) return;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, gr = lane >> 2, gc = lane & 3;
    const int jb = min(kNB, n - j0);
    if (t == 0) s_bad = 0;
    {
        // the previous panel's update of this block, A_JJ -= U_IJ^T U_IJ (I the 64 rows above), whose
        // shared tiles overlap sA and sX
        double cur[2][4][2], acc[2][4][2] = {};
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const int r = out_row(i), c = out_col(j, x);
                    cur[i][j][x] = r == c ? 1.0 : 0.0;
                    if (r < jb && c < jb) cur[i][j][x] = r <= c ? U[(j0 + r) + (long long)(j0 + c) * n] : 0.0;
                }
        if (j0 > 0) {
            const Opnd P{U + j0 - kNB, n, n, kNB};
            tile_product<true, true>(P, P, j0, j0, 0, kNB, psm, acc);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const int r = out_row(i), c = out_col(j, x);
                    // padded rows and columns of the product are zero
                    sA[c * kPL + r] = r <= c ? cur[i][j][x] - acc[i][j][x] : 0.0;
                    sX[c * kPL + r] = 0.0;
                }
    }
    __syncthreads();
    for (int kb = 0; kb < kNB; kb += 16) {
        const int tiles = (kNB - kb) / 8;  // 8-wide tiles from kb on
        if (warp == 0) {
            if (kb > 0) {
                panel_update_tile(sA, kb - 16, kb, kb);
                panel_update_tile(sA, kb - 16, kb, kb + 8);
                panel_update_tile(sA, kb - 16, kb + 8, kb + 8);
                __syncwarp();
            }
            const int bad = panel_factor16(sA + kb * kPL + kb, sX + kb * kPL + kb);
            if (bad && lane == 0) s_bad = kb + bad;
        } else if (kb > 0) {
            // the rest of the previous block's update: upper tiles (ti <= tj) but the three above
            int q = 0;
            for (int tj = 2; tj < tiles; ++tj)
                for (int ti = 0; ti <= tj; ++ti, ++q)
                    if (q % (kPW - 1) == warp - 1) panel_update_tile(sA, kb - 16, kb + 8 * ti, kb + 8 * tj);
        }
        __syncthreads();
        if (s_bad) {
            if (t == 0) atomicCAS(status, 0, j0 + s_bad);
            return;
        }
        // U_12 = U_11^-T A_12 in place: a warp per 8 columns, both row tiles
        const int c0 = kb + 16 + 8 * warp;
        if (c0 < kNB) {
            double acc[2][2] = {};
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
                const double bf = sA[(c0 + gr) * kPL + kb + 4 * ks + gc];
#pragma unroll
                for (int i = 0; i < 2; ++i)  // A(i, k) = X(k, i)
                    dmma(acc[i], sX[(kb + 8 * i + gr) * kPL + kb + 4 * ks + gc], bf);
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int x = 0; x < 2; ++x) sA[(c0 + 2 * gc + x) * kPL + kb + 8 * i + gr] = acc[i][x];
        }
        __syncthreads();
    }
    // inverse: pairs of 16, then of 32: X_01 = -X_00 (U_01 X_11)
    {
        const int o = 32 * (warp >> 2), r0 = 8 * ((warp >> 1) & 1), c0 = 8 * (warp & 1);
        panel_product_tile(sA + (o + 16) * kPL + o, kPL, sX + (o + 16) * kPL + o + 16, kPL, r0, c0, 0, 16, 1.0,
                           sT + (warp >> 2) * 16 * kPT, kPT);
        __syncthreads();
        panel_product_tile(sX + o * kPL + o, kPL, sT + (warp >> 2) * 16 * kPT, kPT, r0, c0, 0, 16, -1.0,
                           sX + (o + 16) * kPL + o, kPL);
        __syncthreads();
        for (int q = warp; q < 16; q += kPW)
            panel_product_tile(sA + 32 * kPL, kPL, sX + 32 * kPL + 32, kPL, 8 * (q & 3), 8 * (q >> 2), 0,
                               8 * (q >> 2) + 8, 1.0, sT, kPT);
        __syncthreads();
        for (int q = warp; q < 16; q += kPW)
            panel_product_tile(sX, kPL, sT, kPT, 8 * (q & 3), 8 * (q >> 2), 8 * (q & 3), 32, -1.0, sX + 32 * kPL, kPL);
        __syncthreads();
    }
    for (int e = t; e < kNB * kNB; e += kThreadsB) {
        const int r = e % kNB, c = e / kNB;
        const double x = sX[c * kPL + r];
        Ub[e] = x;
        if (r <= c && c < jb) {
            U[(j0 + r) + (long long)(j0 + c) * n] = sA[c * kPL + r];
            if (Ui) Ui[(j0 + r) + (long long)(j0 + c) * n] = x;
        }
    }
}

// Row block of panel j0, 64 columns per CTA: A_12 -= U_I1^T U_I2 (I the previous panel's 64 rows, its
// update of this row block), then U_12 = U_11^-T A_12 in place.  Doing the update here (and that of
// the diagonal block in the panel kernel) takes the trailing kernel of panel j0 - 64 off the chain of
// panels, which needs the trailing update of panel j0 - 128 only.
__global__ void __launch_bounds__(kThreadsB) bc_panel_row_kernel(double* __restrict__ U, const double* Ub, int n, int j0, const int* status) {
    extern __shared__ double smem[];
    const int jb = min(kNB, n - j0), j1 = j0 + jb;
    const int c0 = j1 + blockIdx.x * kNB;
    double cur[2][4][2], acc[2][4][2] = {};
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = out_row(i), c = c0 + out_col(j, h);
                cur[i][j][h] = (r < jb && c < n) ? U[(j0 + r) + (long long)c * n] : 0.0;
            }
    if (j0 > 0) {
        const Opnd P{U + j0 - kNB, n, n, kNB};
        tile_product<true, true>(P, P, j0, c0, 0, kNB, smem, acc);
    }
    // everything so far is older than the panel kernel, which this kernel was launched beside
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (failed(status)) return;
    // the updated tile as the k-contiguous B operand and U_11^-T as the A operand, two 32-deep halves each
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = out_row(i), c = out_col(j, h);
                smem[(2 + (r >> 5)) * kTileDoubles + c * kStrideKC + (r & 31)] = cur[i][j][h] - acc[i][j][h];
                acc[i][j][h] = 0.0;
            }
    for (int e = threadIdx.x; e < kNB * kNB; e += kThreadsB) {
        const int k = e % kNB, i = e / kNB;
        smem[(k >> 5) * kTileDoubles + i * kStrideKC + (k & 31)] = __ldcg(Ub + e);
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gr = lane >> 2, gc = lane & 3;
    const int wm = (warp & 3) * 16, wn = (warp >> 2) * 32;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const double* a = smem + half * kTileDoubles;
        const double* b = smem + (2 + half) * kTileDoubles;
#pragma unroll
        for (int kk = 0; kk < kKS; kk += 4) {
            double af[2], bf[4];
#pragma unroll
            for (int i = 0; i < 2; ++i) af[i] = frag<true>(a, wm + 8 * i + gr, kk + gc);
#pragma unroll
            for (int j = 0; j < 4; ++j) bf[j] = frag<true>(b, wn + 8 * j + gr, kk + gc);
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) dmma(acc[i][j], af[i], bf[j]);
        }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = out_row(i), c = c0 + out_col(j, h);
                if (r < jb && c < n) U[(j0 + r) + (long long)c * n] = acc[i][j][h];
            }
}

// A_22 -= U_12^T U_12 over the row blocks that the next panel and row kernels do not update
// themselves: the upper 64 x 64 tiles (ti <= tj) of the matrix from row j0 + 128 on, enumerated as
// t = tj (tj + 1) / 2 + ti.  Each tile's current entries are loaded first, so that their latency
// overlaps the product.
__global__ void __launch_bounds__(kThreadsB, 2) bc_trailing_kernel(double* __restrict__ U, int n, int j0,
                                                                   const int* status) {
    extern __shared__ double smem[];
    if (failed(status)) return;
    const int j2 = j0 + 2 * kNB;
    const long long b = blockIdx.x;
    int tj = (int)((sqrt(8.0 * (double)b + 1.0) - 1.0) * 0.5);
    while ((long long)tj * (tj + 1) / 2 > b) --tj;
    while ((long long)(tj + 1) * (tj + 2) / 2 <= b) ++tj;
    const int ti = (int)(b - (long long)tj * (tj + 1) / 2);
    const int r0 = j2 + kNB * ti, c0 = j2 + kNB * tj;
    const Opnd P{U + j0, n, n, kNB};
    double cur[2][4][2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = r0 + out_row(i), c = c0 + out_col(j, h);
                cur[i][j][h] = (r <= c && c < n) ? U[r + (long long)c * n] : 0.0;
            }
    double acc[2][4][2] = {};
    tile_product<true, true>(P, P, r0, c0, 0, kNB, smem, acc);
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = r0 + out_row(i), c = c0 + out_col(j, h);
                if (r <= c && c < n) U[r + (long long)c * n] = cur[i][j][h] - acc[i][j][h];
            }
}

// One level of the pairwise inverse: pair p has A = Ui block at rows/columns [r0, r0 + b), C at
// [c0, c0 + cs) with c0 = r0 + b, and B = U[r0 .., c0 ..].  STAGE 0: T = B C^-1 (k <= column:
// C^-1 is upper triangular); STAGE 1: Ui[r0 .., c0 ..] = -A^-1 T (k >= row).
template <int STAGE>
__global__ void __launch_bounds__(kThreadsB) bc_level_kernel(const double* __restrict__ U, double* __restrict__ Ui,
                                                             double* __restrict__ T, int n, int b, const int* status) {
    extern __shared__ double smem[];
    if (failed(status)) return;
    const int r0 = 2 * b * blockIdx.y, c0 = r0 + b;
    if (c0 >= n) return;
    const int cs = min(b, n - c0);
    const int tr = b / kNB;
    const int ti = blockIdx.x % tr, tj = blockIdx.x / tr;
    if (kNB * tj >= cs) return;
    const long long ln = n;
    double acc[2][4][2] = {};
    if (STAGE == 0) {
        const int ke = min(cs, kNB * tj + kNB);
        tile_product<false, true>(Opnd{U + r0 + c0 * ln, ln, b, cs}, Opnd{Ui + c0 + c0 * ln, ln, cs, cs}, kNB * ti,
                                  kNB * tj, 0, ke, smem, acc);
    } else {
        tile_product<false, true>(Opnd{Ui + r0 + r0 * ln, ln, b, b}, Opnd{T + r0 + c0 * ln, ln, cs, b}, kNB * ti,
                                  kNB * tj, kNB * ti, b, smem, acc);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = kNB * ti + out_row(i), c = kNB * tj + out_col(j, h);
                if (r < b && c < cs) {
                    const long long at = (r0 + r) + (c0 + c) * ln;
                    if (STAGE == 0)
                        T[at] = acc[i][j][h];
                    else
                        Ui[at] = -acc[i][j][h];
                }
            }
}

}  // namespace

size_t blocked_cholesky_workspace(int n, bool inverse) {
    const size_t t = inverse ? sizeof(double) * (size_t)n * n : 0;
    return t + sizeof(double) * kNB * kNB + 256;
}

// U (n x n, device, column-major; the lower triangle is written with zeros) and, when Ui is not
// null, U^-1 (same layout) of the device matrix M; `work` holds blocked_cholesky_workspace(n, Ui)
// bytes.  *info: order of the first failing pivot, 0 on success.  Synchronizes the stream.
namespace {

// High-priority auxiliary streams (with their two events) for the look-ahead panels, pooled per
// device: a call takes one for its duration, so concurrent calls from several host threads never
// share one.
struct AuxStream {
    int device = -1;
    cudaStream_t stream = nullptr;
    cudaEvent_t row_done = nullptr, trailing_done[2] = {nullptr, nullptr};
};
std::mutex g_aux_mutex;
std::vector<AuxStream> g_aux_free;

cudaError_t acquire_aux(AuxStream* out) {
    int device = 0;
    cudaError_t err = cudaGetDevice(&device);
    if (err != cudaSuccess) return err;
    {
        std::lock_guard<std::mutex> lock(g_aux_mutex);
        for (size_t i = 0; i < g_aux_free.size(); ++i)
            if (g_aux_free[i].device == device) {
                *out = g_aux_free[i];
                g_aux_free.erase(g_aux_free.begin() + (long)i);
                return cudaSuccess;
            }
    }
    AuxStream a;
    a.device = device;
    int least = 0, greatest = 0;
    err = cudaDeviceGetStreamPriorityRange(&least, &greatest);
    if (err == cudaSuccess) err = cudaStreamCreateWithPriority(&a.stream, cudaStreamNonBlocking, greatest);
    if (err == cudaSuccess) err = cudaEventCreateWithFlags(&a.row_done, cudaEventDisableTiming);
    for (cudaEvent_t& e : a.trailing_done)
        if (err == cudaSuccess) err = cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
    if (err != cudaSuccess) return err;
    *out = a;
    return cudaSuccess;
}

void release_aux(const AuxStream& a) {
    std::lock_guard<std::mutex> lock(g_aux_mutex);
    g_aux_free.push_back(a);
}

}  // namespace

cudaError_t blocked_cholesky(const double* M, int n, double* U, double* Ui, void* work, int* info,
                             cudaStream_t s) {
    *info = 0;
    unsigned char* w = static_cast<unsigned char*>(work);
    double* T = Ui ? reinterpret_cast<double*>(w) : nullptr;
    double* Ub = reinterpret_cast<double*>(w + (Ui ? sizeof(double) * (size_t)n * n : 0));
    int* status = reinterpret_cast<int*>(Ub + kNB * kNB);
    cudaError_t err = allow_dynamic_smem((const void*)bc_panel_kernel, kPanelSmem);
    if (err == cudaSuccess) err = allow_dynamic_smem((const void*)bc_panel_row_kernel, kProductSmem);
    if (err == cudaSuccess) err = allow_dynamic_smem((const void*)bc_trailing_kernel, kProductSmem);
    if (err == cudaSuccess) err = allow_dynamic_smem((const void*)bc_level_kernel<0>, kProductSmem);
    if (err == cudaSuccess) err = allow_dynamic_smem((const void*)bc_level_kernel<1>, kProductSmem);
    if (err == cudaSuccess) err = cudaMemsetAsync(status, 0, sizeof(int), s);
    if (err == cudaSuccess && Ui) err = cudaMemsetAsync(Ui, 0, sizeof(double) * (size_t)n * n, s);
    if (err != cudaSuccess) return err;
    const long long total = (long long)n * n;
    bc_init_kernel<<<(unsigned)std::min<long long>(4096, (total + 255) / 256), 256, 0, s>>>(M, U, n);
    // Look-ahead: the chain panel J, row J, panel J + 1, row J + 1, ... runs on a high-priority
    // auxiliary stream, each kernel applying the previous panel's update to its own blocks; the
    // trailing update of panel J (row blocks J + 2 on) runs on s and has until panel J + 2.
    AuxStream aux;
    if ((err = acquire_aux(&aux)) != cudaSuccess) return err;
    err = cudaEventRecord(aux.row_done, s);
    if (err == cudaSuccess) err = cudaStreamWaitEvent(aux.stream, aux.row_done, 0);
    for (int j0 = 0; j0 < n && err == cudaSuccess; j0 += kNB) {
        const cudaEvent_t trailing = aux.trailing_done[(j0 / kNB) & 1];
        if (j0 >= 2 * kNB && (err = cudaStreamWaitEvent(aux.stream, trailing, 0)) != cudaSuccess) break;
        bc_panel_kernel<<<1, kThreadsB, kPanelSmem, aux.stream>>>(U, Ub, Ui, n, j0, status);
        const int j1 = j0 + kNB;
        if (j1 >= n) break;
        // programmatic dependent launch: the row kernel's update of its block by the previous panel runs
        // beside the panel kernel.  The first call of a process takes 9 to 15 ms either way (n = 600; 0.35 ms
        // later, 0.59 without it), the first of eight threads at once, each on a new auxiliary stream, 3 ms
        // (10 without), and a new engine's first batch 67 ms (103 to 138).
        cudaLaunchAttribute beside{};
        beside.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        beside.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t row{};
        row.gridDim = dim3((n - j1 + kNB - 1) / kNB);
        row.blockDim = dim3(kThreadsB);
        row.dynamicSmemBytes = kProductSmem;
        row.stream = aux.stream;
        row.attrs = &beside;
        row.numAttrs = 1;
        err = cudaLaunchKernelEx(&row, bc_panel_row_kernel, U, (const double*)Ub, n, j0, (const int*)status);
        if (err != cudaSuccess) break;
        const int m = n - j1 - kNB;
        if (m > 0) {
            if ((err = cudaEventRecord(aux.row_done, aux.stream)) != cudaSuccess) break;
            if ((err = cudaStreamWaitEvent(s, aux.row_done, 0)) != cudaSuccess) break;
            const long long nt = (m + kNB - 1) / kNB;
            bc_trailing_kernel<<<(unsigned)(nt * (nt + 1) / 2), kThreadsB, kProductSmem, s>>>(U, n, j0, status);
            if ((err = cudaEventRecord(trailing, s)) != cudaSuccess) break;
        }
        err = cudaGetLastError();
    }
    // join: the chain precedes the rest of s
    cudaError_t join = cudaEventRecord(aux.row_done, aux.stream);
    if (join == cudaSuccess) join = cudaStreamWaitEvent(s, aux.row_done, 0);
    if (err == cudaSuccess) err = join;
    release_aux(aux);
    if (Ui) {
        for (int b = kNB; b < n && err == cudaSuccess; b *= 2) {
            const int pairs = (n + 2 * b - 1) / (2 * b);
            const int tr = b / kNB;
            const dim3 grid((unsigned)(tr * tr), (unsigned)pairs);
            bc_level_kernel<0><<<grid, kThreadsB, kProductSmem, s>>>(U, Ui, T, n, b, status);
            bc_level_kernel<1><<<grid, kThreadsB, kProductSmem, s>>>(U, Ui, T, n, b, status);
            err = cudaGetLastError();
        }
    }
    int h = 0;
    if (err == cudaSuccess) err = cudaMemcpyAsync(&h, status, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (err == cudaSuccess) err = cudaStreamSynchronize(s);
    if (err == cudaSuccess) *info = h;
    return err;
}

}  // namespace vbcore
