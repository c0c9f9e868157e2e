// Determinant pairs of covalent lists straight from the frame tables (sm_100a).
//
// In a covalent list every orbital is singly occupied: the beta string of a determinant is the
// complement x of its alpha string u, every alpha string carries one determinant, and each spin-pair
// record is used by exactly one determinant pair (two that are equal, with spin-flip symmetry).  Writing
// the records (R + 4 doubles a pair: 2.2 GB for the 5.9 M pairs of 14 orbitals) and gathering them again
// took as long as the products behind them.  covalent_pairs takes both spins of a determinant pair in the
// same warp and keeps the two u-vectors in tensor-core accumulators until they are multiplied.
//
// Holes of (u, v) are the particles of (x, y), y the complement of v, and the other way round: one
// descriptor serves both spins, lanes 0 .. 15 take the alpha side of 16 determinant pairs and lanes 16 ..
// 31 the beta side, and every lane runs the same code at the same excitation level.  The beta table is
// staged transposed (blocks by particle, columns by hole position), so that the blocks of a tile's alpha
// hole set are also the beta side's particle set and both products walk the same k-steps.
//
// With spin-flip symmetry one member of each orbit {(d, e), (flip d, flip e)} is evaluated and written to
// both places.  Pairs of which a side cannot be evaluated here (uncertified in an ill-conditioned frame or at
// a level above five) are listed: that side's record goes to the exact path, and listed_covalent_pairs
// evaluates the other side and combines them.  (Both records in the exact path, 14 orbitals of which two
// are nearly dependent: 520,853 of them in 8.7 ms, against 291,373 and 6.2 ms for the records alone.)
//
// 14 orbitals, 2.9 M orbits: 1361 us (1428 us with a test per row tile in the product), against 1280 us for
// the records and 537 us for the pairs gathered from them; 12-orbital triplet: 160 us, against 235 us.
// Bound by latency: one CTA of up to 16 warps per SM (two blocks and the warps' adj B slots in shared
// memory, 128 registers a thread) waits on fixed latencies and on the tensor pipe, and saturates neither the
// issue slots (42 %) nor the FP64 tensor pipe (37 % active).
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "device_algebra.cuh"
#include "frame.cuh"
#include "frame_pair.cuh"
#include "internal.h"
#include "kernels.h"
#include "pair_value.cuh"

namespace vbcore {
namespace {

constexpr int kSms = 148;
constexpr int kCovalentMaxWarps = 16;
constexpr int kCovalentTiles = 7;  // table row tiles per pass (accumulators of both spins)

// determinant pairs of a chunk: lane p the alpha side, lane 16 + p the beta side
__host__ __device__ constexpr int covalent_chunk(int e) { return e <= kMinorsEMax ? 16 : (e <= 7 ? 8 : 4); }
static_assert(2 * covalent_chunk(5) * compact_slot(5) <= 32 * kCompactSlot &&
                  2 * covalent_chunk(7) * compact_slot(7) <= 32 * kCompactSlot &&
                  2 * covalent_chunk(8) * compact_slot(8) <= 32 * kCompactSlot,
              "a warp's slots hold both spins of a chunk");

// Parity of the row -> column assignment of the pair (L, R) (see pair_descriptor): the common orbitals
// between the i-th hole and the i-th particle, summed over i.
__device__ __forceinline__ unsigned excitation_parity(uint64_t mL, uint64_t mR) {
    uint64_t h = mL & ~mR, p = mR & ~mL;
    const uint64_t common = mL & mR;
    int n = 0;
    while (h) {
        const uint64_t hb = h & (~h + 1), pb = p & (~p + 1);
        h ^= hb;
        p ^= pb;
        const uint64_t lo = hb < pb ? hb : pb, hi = hb < pb ? pb : hb;
        n += __popcll(common & (hi - 1) & ~(lo | (lo - 1)));
    }
    return (unsigned)(n & 1);
}

// One warp per alpha string u: its partners v >= u (with flip, one of each orbit) by hole set, in order
// of excitation level, then hole mask, then v.  Descriptor: hole mask, particle mask << 8, alpha parity
// << 16, beta parity << 17, and << 19 whether the orbit is its own flip (both spins hold the same record).
constexpr int kSortWarps = 4;
__global__ void __launch_bounds__(32 * kSortWarps) sort_covalent_pairs(CovalentArgs a, const uint64_t* __restrict__ occ,
                                                                       int* __restrict__ list, unsigned* __restrict__ desc,
                                                                       int* __restrict__ bounds) {
    __shared__ int cursor[kSortWarps][256];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, K = a.ka, N = a.n_strings;
    const int u = blockIdx.x * kSortWarps + warp;
    if (u >= N) return;
    int* cur = cursor[warp];
    const int bins = 1 << K;
    for (int x = lane; x < bins; x += 32) cur[x] = 0;
    __syncwarp();
    const uint64_t wL = __ldg(occ + 2 * (long long)u), mL = occ_mask(wL, K);
    const uint64_t all = a.n >= 64 ? ~0ull : (1ull << a.n) - 1;
    const int x = __ldg(a.beta + u);
    auto holes = [&](int v) -> int {
        if (v >= N) return -1;
        if (a.fold) {
            const int y = __ldg(a.beta + v), lo = min(x, y), hi = max(x, y);
            if (lo < u || (lo == u && hi < v)) return -1;
        }
        const uint64_t mR = occ_mask(__ldg(occ + 2 * (long long)v), K);
        int hm = 0;
        for (int c = 0; c < K; ++c) hm |= ((mR >> ((wL >> (8 * c)) & 0xFFu)) & 1ull) ? 0 : (1 << c);
        return hm;
    };
    auto own = [&](int v) -> unsigned {
        const int y = __ldg(a.beta + v);
        return a.fold && min(x, y) == u && max(x, y) == v;
    };
    for (int v0 = u; v0 < N; v0 += 32) {
        const int hm = holes(v0 + lane);
        const unsigned same = __match_any_sync(0xffffffffu, hm);
        if (hm >= 0 && lane == __ffs(same) - 1) cur[hm] += __popc(same);
        __syncwarp();
    }
    if (lane == 0) {
        int run = 0;
        int* eb = bounds + (long long)u * (K + 2);
        for (int e = 0; e <= K; ++e) {
            eb[e] = run;
            for (int b = 0; b < bins; ++b)
                if (__popc(b) == e) {
                    const int c = cur[b];
                    cur[b] = run;
                    run += c;
                }
        }
        eb[K + 1] = run;
    }
    __syncwarp();
    const long long base = record_index(u, u, N);
    for (int v0 = u; v0 < N; v0 += 32) {
        const int v = v0 + lane, hm = holes(v);
        const unsigned same = __match_any_sync(0xffffffffu, hm);
        int pos = 0;
        if (hm >= 0) pos = cur[hm] + __popc(same & ((1u << lane) - 1u));
        __syncwarp();
        if (hm >= 0) {
            const uint64_t mR = occ_mask(__ldg(occ + 2 * (long long)v), K);
            unsigned pm = 0;
            for (uint64_t p = mR & ~mL; p; p &= p - 1) pm |= 1u << __popcll(~mL & ((p & (~p + 1)) - 1));
            list[base + pos] = v;
            desc[base + pos] = (unsigned)hm | (pm << 8) | (excitation_parity(mL, mR) << 16) |
                               (excitation_parity(all & ~mL, all & ~mR) << 17) | (own(v) << 19);
            if (lane == __ffs(same) - 1) cur[hm] += __popc(same);
        }
        __syncwarp();
    }
}

// Upper-triangle position of the determinants of strings u and v.
__device__ __forceinline__ long long covalent_position(const CovalentArgs& a, int u, int v) {
    const long long d = __ldg(a.det + u), e = __ldg(a.det + v);
    return d < e ? d * a.ldb + e : e * a.ldb + d;
}

__device__ __forceinline__ void covalent_store(const CovalentArgs& a, int u, int v, double H, double S) {
    const double w = u == v ? 0.5 : 1.0;  // H_d = U' + U'^T
    H *= w;
    S *= w;
    const long long at = covalent_position(a, u, v);
    a.Hb[at] = H;
    a.Sb[at] = S;
    if (a.fold) {
        const long long flipped = covalent_position(a, __ldg(a.beta + u), __ldg(a.beta + v));
        a.Hb[flipped] = H;
        a.Sb[flipped] = S;
    }
}

// Appends the values of the lanes that have one, with one atomic per warp (all lanes call).
__device__ __forceinline__ void append(unsigned long long* list, unsigned long long* count, bool has,
                                       unsigned long long value, int lane) {
    const unsigned mask = __ballot_sync(0xffffffffu, has);
    if (mask == 0) return;
    unsigned long long at = 0;
    if (lane == 0) at = atomicAdd(count, (unsigned long long)__popc(mask));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (has) list[at + __popc(mask & ((1u << lane) - 1u))] = value;
}

// Doubles of a block from Q on.
__host__ __device__ inline int covalent_rest(const FrameLayout& F) { return F.total - F.o_q; }

template <int K>
__global__ void __launch_bounds__(32 * kCovalentMaxWarps, 1) covalent_pairs(CovalentArgs a) {
    extern __shared__ __align__(16) double smem[];
    constexpr int KFS = fr_kfs(K);
    const int R = a.R, KB = a.kb, n = a.n;
    const FrameLayout FA = frame_layout(n, K, R), FB = frame_layout(n, KB, R);
    const int NT = FA.rows / 8;
    double* tabA = smem;                       // [row][hole position of u][particle]
    double* tabB = tabA + FA.rows * KFS;       // [row][particle of x][hole position]: the same blocks
    double* restA = tabB + FA.rows * KFS;
    double* restB = restA + covalent_rest(FA);
    double* sY = restB + covalent_rest(FB);
    __shared__ int s_task, s_chunk;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    const bool beta = lane >= 16;
    const FrameLayout& FS = beta ? FB : FA;
    const FrameViewAny view{beta ? restB : restA, beta ? KB : K,       FS.o_p - FS.o_q,
                            FS.o_rowsq - FS.o_q,  FS.o_prow2 - FS.o_q, FS.o_scal - FS.o_q};
    const long long N = a.n_strings;
    double* yw = sY + (size_t)warp * 32 * kCompactSlot;
    // passes of nearly equal length over the table rows
    const int passes = (NT + kCovalentTiles - 1) / kCovalentTiles, per_pass = (NT + passes - 1) / passes;
    const bool pad = KB <= 7;  // the trace stands in the last column of every block
    for (;;) {
        if (threadIdx.x == 0) {
            s_task = (int)atomicAdd(a.task_counter, 1ull);
            s_chunk = 0;
        }
        __syncthreads();
        const int u = s_task;
        if (u >= N) break;
        int bound[K + 2];
        const int* eb = a.bounds + (long long)u * (K + 2);
#pragma unroll
        for (int e = 0; e < K + 2; ++e) bound[e] = __ldg(eb + e);
        if (bound[K + 1] == 0) {
            __syncthreads();
            continue;
        }
        {
            const double2* src = reinterpret_cast<const double2*>(a.tables_a + (long long)u * FA.total);
            double2* dst = reinterpret_cast<double2*>(tabA);
            for (int i = threadIdx.x; i < FA.rows * KFS / 2; i += blockDim.x) dst[i] = __ldg(src + i);
            for (int i = threadIdx.x; i < covalent_rest(FA) / 2; i += blockDim.x)
                reinterpret_cast<double2*>(restA)[i] = __ldg(src + FA.o_q / 2 + i);
            const double* sb = a.tables_b + (long long)__ldg(a.beta + u) * FB.total;
            for (int i = threadIdx.x; i < covalent_rest(FB) / 2; i += blockDim.x)
                reinterpret_cast<double2*>(restB)[i] = __ldg(reinterpret_cast<const double2*>(sb + FB.o_q) + i);
            for (int i = threadIdx.x; i < FA.rows * KFS; i += blockDim.x) {
                const int r = i / KFS, col = i % KFS, b = col >> 3, c = col & 7;
                const double* row = sb + r * FB.kfs;
                double v = 0.0;
                if (col >= 8 * K)
                    v = __ldg(row + 8 * KB + col - 8 * K);
                else if (c < KB)
                    v = __ldg(row + 8 * c + b);
                else if (c == 7)
                    v = __ldg(row + 8 * KB);
                tabB[i] = v;
            }
        }
        const long long base = record_index(u, u, N);
        __syncthreads();
        // warps take chunks dynamically, highest excitation level first, and load the next chunk's
        // strings and descriptors while they evaluate the current one
        auto claim = [&](int* e_out, int* cnt_out, int* v_out, unsigned* d_out) {
            int left = 0;
            if (lane == 0) left = atomicAdd(&s_chunk, 1);
            left = __shfl_sync(0xffffffffu, left, 0);
            int e = -1, start = 0, cnt = 0;
#pragma unroll
            for (int ee = K; ee >= 0; --ee) {
                const int cs = covalent_chunk(ee), c = (bound[ee + 1] - bound[ee] + cs - 1) / cs;
                if (left >= 0 && left < c) {
                    e = ee;
                    start = bound[ee] + cs * left;
                    cnt = min(cs, bound[ee + 1] - start);
                }
                left -= c;
            }
            const bool valid = (lane & 15) < cnt;
            const long long at = base + start + (lane & 15);
            *v_out = valid ? __ldg(a.list + at) : u;
            *d_out = valid ? __ldg(a.desc + at) : 0u;
            *e_out = e;
            *cnt_out = cnt;
        };
        int e_next, cnt_next, v_next;
        unsigned d_next;
        claim(&e_next, &cnt_next, &v_next, &d_next);
        for (;;) {
            const int e = e_next, cnt = cnt_next, v = v_next;
            unsigned desc = d_next;
            if (e < 0) break;
            claim(&e_next, &cnt_next, &v_next, &d_next);
            const unsigned hm = desc & 0x800FFu;  // holes, and bit 19
            if (beta) desc = ((desc >> 8) & 0xFFu) | ((desc & 0xFFu) << 8) | ((desc >> 1) & 0x10000u);
            const int slot = compact_slot(e);
            FramePair o{};
            o.hmap = o.pmap = 0xFFFFFFFFu;
            const bool valid = (lane & 15) < cnt;
            // slots of the alpha pairs, then of the beta pairs
            if (valid) o = frame_pair_dispatch<K>(e, view, desc, yw + ((lane & 15) + (beta ? covalent_chunk(e) : 0)) * slot);
            const unsigned okbits = __ballot_sync(0xffffffffu, o.ok), both = okbits & (okbits >> 16);
            // pairs evaluated outside the certificate, every record once (an orbit that is its own flip holds
            // one, listed unless both sides are evaluated)
            const unsigned poly = __ballot_sync(
                0xffffffffu, o.ok && !o.certified && (!(hm >> 19) || (!beta && ((both >> lane) & 1u))));
            if (lane == 0 && (poly & 0xFFFFu)) atomicAdd(a.uncertified_a, (unsigned long long)__popc(poly & 0xFFFFu));
            if (lane == 0 && (poly >> 16)) atomicAdd(a.uncertified_b, (unsigned long long)__popc(poly >> 16));
            const unsigned fail = __ballot_sync(0xffffffffu, valid) & ~both & 0xFFFFu;
            if (fail) {
                // bit 0: alpha evaluated in its frame, bit 1: beta
                const unsigned sides = hm >> 19 ? 0u : ((okbits >> (lane & 15)) & 1u) | ((okbits >> (15 + (lane & 15))) & 2u);
                const bool mine = (fail >> lane) & 1u;
                const unsigned long long pair = ((unsigned long long)u << 32) | (unsigned long long)v;
                const int x = __ldg(a.beta + u), y = __ldg(a.beta + v);
                append(a.listed, a.listed_count, mine, pair | ((unsigned long long)sides << 30), lane);
                append(a.list_a, a.count_a, mine && !(sides & 1u), pair, lane);
                append(a.list_b, a.count_b, mine && !(sides & 2u) && !(hm >> 19),
                       ((unsigned long long)min(x, y) << 32) | (unsigned long long)max(x, y), lane);
            }
            __syncwarp();
            const int tiles = (covalent_chunk(e) + 7) / 8;
#pragma unroll 1
            for (int mt = 0; mt < tiles; ++mt) {
                const unsigned uh = __reduce_or_sync(0xffffffffu, (lane >> 3) == mt ? hm & 0xFFu : 0u);
                if (((both >> (8 * mt)) & 0xFFu) == 0) continue;
                const int owner = 8 * mt + g;
                const double deta = __shfl_sync(0xffffffffu, o.detb, owner), detb = __shfl_sync(0xffffffffu, o.detb, owner + 16);
                const unsigned hmap = __shfl_sync(0xffffffffu, o.hmap, owner), pmap = __shfl_sync(0xffffffffu, o.pmap, owner);
                const bool ok = (both >> owner) & 1u;
                const double* ya = yw + owner * slot;
                const double* yb = yw + (owner + covalent_chunk(e)) * slot;
                const unsigned i0 = (pmap >> (4 * tq)) & 0xFu, i1 = (pmap >> (4 * (tq + 4))) & 0xFu;
                const bool pad_trace = e >= 1 && pad;
                double dot = 0.0, ha = 0.0, hb = 0.0;
                // one pass over nt tiles of table rows from nt0 on (nt at compile time: no test per tile)
                auto pass = [&](auto tiles_of_pass, int nt0) {
                    constexpr int T = decltype(tiles_of_pass)::value;
                    const double* rowA = tabA + (8 * nt0 + g) * KFS + tq;
                    const double* rowB = tabB + (8 * nt0 + g) * KFS + tq;
                    double ua[T][2], ub[T][2];
#pragma unroll
                    for (int j = 0; j < T; ++j) ua[j][0] = ua[j][1] = ub[j][0] = ub[j][1] = 0.0;
                    auto step = [&](double fa, double fb, int col) {
#pragma unroll
                        for (int j = 0; j < T; ++j) {
                            mma_f64(ua[j], fa, rowA[8 * j * KFS + col]);
                            mma_f64(ub[j], fb, rowB[8 * j * KFS + col]);
                        }
                    };
                    if (!pad_trace) step(tq == 0 && ok ? deta : 0.0, tq == 0 && ok ? detb : 0.0, 8 * K);
                    unsigned rest = uh;
#pragma unroll 1
                    while (rest) {
                        const int c = __ffs(rest) - 1;
                        rest &= rest - 1;
                        const unsigned jh = (hmap >> (4 * c)) & 0xFu;
#pragma unroll
                        for (int ks = 0; ks < 2; ++ks) {
                            const unsigned ip = ks ? i1 : i0;
                            // alpha: hole slot jh, particle slot ip; beta: the other way round
                            const bool on = ok && jh < (unsigned)e && ip < (unsigned)e;
                            double fa = on ? ya[jh * e + ip] : 0.0, fb = on ? yb[ip * e + jh] : 0.0;
                            if (pad_trace && ks == 1 && tq == 3) {
                                fa = ok && jh == 0 ? deta : 0.0;
                                fb = ok && jh == 0 ? detb : 0.0;
                            }
                            step(fa, fb, 8 * c + 4 * ks);
                        }
                    }
                    // columns 2 tq and 2 tq + 1 of pair g: table rows 0 = h, 1 = two-electron linear, 2 + m
#pragma unroll
                    for (int j = 0; j < T; ++j)
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const int m = 8 * (nt0 + j) + 2 * tq + i - 2;
                            const double prod = ua[j][i] * ub[j][i];
                            if (m >= 0 && m < R) dot += m < a.r_pos ? prod : -prod;
                        }
                    if (nt0 == 0) {
                        ha = ua[0][0] + ua[0][1];
                        hb = ub[0][0] + ub[0][1];
                    }
                };
#pragma unroll 1
                for (int nt0 = 0; nt0 < NT; nt0 += per_pass) {
                    switch (min(per_pass, NT - nt0)) {
                        case 1: pass(std::integral_constant<int, 1>{}, nt0); break;
                        case 2: pass(std::integral_constant<int, 2>{}, nt0); break;
                        case 3: pass(std::integral_constant<int, 3>{}, nt0); break;
                        case 4: pass(std::integral_constant<int, 4>{}, nt0); break;
                        case 5: pass(std::integral_constant<int, 5>{}, nt0); break;
                        case 6: pass(std::integral_constant<int, 6>{}, nt0); break;
                        default: pass(std::integral_constant<int, 7>{}, nt0); break;
                    }
                }
                dot += __shfl_xor_sync(0xffffffffu, dot, 1);
                dot += __shfl_xor_sync(0xffffffffu, dot, 2);
                const double d = __shfl_sync(0xffffffffu, o.d, owner) * __shfl_sync(0xffffffffu, o.d, owner + 16);
                const double qa = __shfl_sync(0xffffffffu, o.quad, owner), qb = __shfl_sync(0xffffffffu, o.quad, owner + 16);
                const int v_g = __shfl_sync(0xffffffffu, v, owner);
                if (ok && tq == 0) covalent_store(a, u, v_g, d * fma(ha + qa, detb, fma(hb + qb, deta, dot)), d * (deta * detb));
            }
            __syncwarp();
        }
        __syncthreads();
    }
}

// Listed pairs: a warp takes up to 32 of them.  A lane per pair runs the algebra of the side that is evaluated
// in its frame (read from the tables in place), then the warp forms that side's u-vector row by row, lanes
// over rows, against the other side's record; without such a side it multiplies the two records.
constexpr int kListedWarps = 4;
// doubles of a pair's adj B (odd stride)
__host__ __device__ inline int listed_slot(int ka) { return (ka * ka) | 1; }

__global__ void __launch_bounds__(32 * kListedWarps, 3) listed_covalent_pairs(CovalentArgs a, FullPairArgs f) {
    extern __shared__ __align__(16) double smem[];
    const long long count = (long long)*a.listed_count, N = a.n_strings;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, R = a.R;
    const long long nwarps = (long long)gridDim.x * kListedWarps;
    long long chunk = (count + nwarps - 1) / nwarps;
    chunk = chunk < 1 ? 1 : (chunk > 32 ? 32 : chunk);
    const FrameLayout FA = frame_layout(a.n, a.ka, R), FB = frame_layout(a.n, a.kb, R);
    const uint64_t all = a.n >= 64 ? ~0ull : (1ull << a.n) - 1;
    const int slot = listed_slot(a.ka);
    double* slots = smem + (size_t)warp * 32 * slot;
    for (long long base = ((long long)blockIdx.x * kListedWarps + warp) * chunk; base < count; base += nwarps * chunk) {
        const int cnt = (int)(count - base < chunk ? count - base : chunk);
        const unsigned long long w = lane < cnt ? a.listed[base + lane] : 0ull;
        const int u = (int)(w >> 32), v = (int)(w & 0x3fffffffull);
        const unsigned sides = (unsigned)(w >> 30) & 3u;
        const bool beta = sides & 2u;
        unsigned desc = 0;
        FramePair o{};
        if (sides) {
            const uint64_t wL = __ldg(a.occ + 2 * (long long)u), mL = occ_mask(wL, a.ka);
            const uint64_t mR = occ_mask(__ldg(a.occ + 2 * (long long)v), a.ka);
            unsigned hm = 0, pm = 0;
            for (uint64_t h = mL & ~mR; h; h &= h - 1) hm |= 1u << __popcll(mL & ((h & (~h + 1)) - 1));
            for (uint64_t p = mR & ~mL; p; p &= p - 1) pm |= 1u << __popcll(~mL & ((p & (~p + 1)) - 1));
            desc = beta ? pm | (hm << 8) | (excitation_parity(all & ~mL, all & ~mR) << 16)
                        : hm | (pm << 8) | (excitation_parity(mL, mR) << 16);
            const FrameLayout& F = beta ? FB : FA;
            const double* blk = beta ? a.tables_b + (long long)__ldg(a.beta + u) * F.total : a.tables_a + (long long)u * F.total;
            const FrameViewAny view{blk + F.o_q, beta ? a.kb : a.ka, F.o_p - F.o_q, F.o_rowsq - F.o_q, F.o_prow2 - F.o_q,
                                    F.o_scal - F.o_q};
            o = frame_pair_dispatch<8>(__popc(desc & 0xFFu), view, desc, slots + lane * slot);
        }
        __syncwarp();
        for (int j = 0; j < cnt; ++j) {
            const int uj = __shfl_sync(0xffffffffu, u, j), vj = __shfl_sync(0xffffffffu, v, j);
            const unsigned sj = __shfl_sync(0xffffffffu, sides, j), dj = __shfl_sync(0xffffffffu, desc, j);
            const double d = __shfl_sync(0xffffffffu, o.d, j), detb = __shfl_sync(0xffffffffu, o.detb, j);
            const double quad = __shfl_sync(0xffffffffu, o.quad, j);
            const int x = __ldg(a.beta + uj), y = __ldg(a.beta + vj);
            const double* ra = f.rec_a + record_index(uj, vj, N) * f.stride_a;
            const double* rb = f.rec_b + record_index(min(x, y), max(x, y), N) * f.stride_b;
            const FrameLayout& F = sj & 2u ? FB : FA;
            const double* blk = sj & 2u ? a.tables_b + (long long)x * F.total : a.tables_a + (long long)uj * F.total;
            const int k = sj & 2u ? a.kb : a.ka;
            const double* rec = sj & 1u ? rb : ra;  // a side of the exact path
            double dot = 0.0, energy = 0.0;         // energy: h and two-electron linear rows
            if (sj) {
                // rows r0 + lane and r0 + lane + 32 of the frame side's table, a hole's block of eight columns
                // at a time (the adj B of columns without a particle is zero)
                const unsigned pm = (dj >> 8) & 0xFFu;
                const int e = __popc(pm);
                for (int r0 = 0; r0 < R + 2; r0 += 64) {
                    const int ra0 = min(r0 + lane, R + 1), ra1 = min(r0 + lane + 32, R + 1);
                    const double *t0 = blk + (long long)ra0 * F.kfs, *t1 = blk + (long long)ra1 * F.kfs;
                    double v0 = detb * __ldg(t0 + 8 * k), v1 = detb * __ldg(t1 + 8 * k);
                    const double* yj = slots + j * slot;
#pragma unroll 1
                    for (unsigned h = dj & 0xFFu; h; h &= h - 1, yj += e) {
                        const int c = 8 * (__ffs(h) - 1);
                        const double2 *b0 = reinterpret_cast<const double2*>(t0 + c), *b1 = reinterpret_cast<const double2*>(t1 + c);
                        double2 x0[4], x1[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            x0[q] = __ldg(b0 + q);
                            x1[q] = __ldg(b1 + q);
                        }
#pragma unroll
                        for (int b = 0; b < 8; ++b) {
                            const double y = (pm >> b) & 1u ? yj[__popc(pm & ((1u << b) - 1u))] : 0.0;
                            v0 = fma(y, b & 1 ? x0[b / 2].y : x0[b / 2].x, v0);
                            v1 = fma(y, b & 1 ? x1[b / 2].y : x1[b / 2].x, v1);
                        }
                    }
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const int r = r0 + lane + 32 * q, m = r - 2;
                        const double v = d * (q ? v1 : v0);
                        if (r < 2) energy = v;
                        if (m >= 0 && m < R) dot = fma(m < a.r_pos ? v : -v, rec[m], dot);
                    }
                }
            } else {
                for (int m = lane; m < R; m += 32) dot = fma(m < a.r_pos ? ra[m] : -ra[m], rb[m], dot);
            }
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, s);
            energy += __shfl_xor_sync(0xffffffffu, energy, 1);
            if (lane == 0) {
                const double s1 = rec[R], h1 = rec[R + 1];
                const double s2 = sj ? d * detb : rb[R], h2 = sj ? fma(d, quad, energy) : rb[R + 1];
                covalent_store(a, uj, vj, fma(h1, s2, fma(h2, s1, dot)), s1 * s2);
            }
        }
        __syncwarp();
    }
}

template <int K>
size_t covalent_smem(int n, int kb, int R, int warps) {
    const FrameLayout FA = frame_layout(n, K, R), FB = frame_layout(n, kb, R);
    return sizeof(double) * (2 * (size_t)FA.rows * fr_kfs(K) + covalent_rest(FA) + covalent_rest(FB) +
                             (size_t)warps * 32 * kCompactSlot);
}

constexpr size_t kCovalentSmemMax = 226 * 1024;

// Warps per CTA: enough for a left string's chunks (16 pairs each) in four rounds, at least four to load the
// blocks, within shared memory (6 orbitals: 18 us with two warps, 12.5 us with four).
template <int K>
int covalent_warps(const CovalentArgs& a) {
    int warps = 4;
    while (warps < kCovalentMaxWarps && warps * 64 < a.n_strings) warps *= 2;
    while (warps > 2 && covalent_smem<K>(a.n, a.kb, a.R, warps) > kCovalentSmemMax) warps /= 2;
    return warps;
}

template <int K>
cudaError_t launch_covalent(const CovalentArgs& a, cudaStream_t stream) {
    const int warps = covalent_warps<K>(a);
    const size_t smem = covalent_smem<K>(a.n, a.kb, a.R, warps);
    cudaError_t err = allow_dynamic_smem((const void*)covalent_pairs<K>, smem);
    if (err != cudaSuccess) return err;
    int per_sm = 1;
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, covalent_pairs<K>, 32 * warps, smem);
    if (err != cudaSuccess) return err;
    const long long grid = (long long)kSms * (per_sm > 0 ? per_sm : 1);
    covalent_pairs<K><<<(unsigned)(a.n_strings < grid ? a.n_strings : grid), 32 * warps, smem, stream>>>(a);
    return cudaGetLastError();
}

}  // namespace

bool covalent_pairs_supported(int n, int ka, int kb, int R) {
    if (ka < 2 || ka > 8 || kb < 1 || kb > ka || ka + kb != n || !frame_spin_supported(n, ka, R) || !frame_spin_supported(n, kb, R))
        return false;
    size_t smem = 0;
    switch (ka) {
        case 2: smem = covalent_smem<2>(n, kb, R, 2); break;
        case 3: smem = covalent_smem<3>(n, kb, R, 2); break;
        case 4: smem = covalent_smem<4>(n, kb, R, 2); break;
        case 5: smem = covalent_smem<5>(n, kb, R, 2); break;
        case 6: smem = covalent_smem<6>(n, kb, R, 2); break;
        case 7: smem = covalent_smem<7>(n, kb, R, 2); break;
        default: smem = covalent_smem<8>(n, kb, R, 2); break;
    }
    return smem <= kCovalentSmemMax;
}

cudaError_t launch_sort_covalent_pairs(const CovalentArgs& a, const uint64_t* occ, int* list, unsigned* desc, int* bounds,
                                       cudaStream_t stream) {
    sort_covalent_pairs<<<(a.n_strings + kSortWarps - 1) / kSortWarps, 32 * kSortWarps, 0, stream>>>(a, occ, list, desc, bounds);
    return cudaGetLastError();
}

cudaError_t launch_covalent_pairs(const CovalentArgs& a, cudaStream_t stream, int* launches) {
    ++*launches;
    switch (a.ka) {
        case 2: return launch_covalent<2>(a, stream);
        case 3: return launch_covalent<3>(a, stream);
        case 4: return launch_covalent<4>(a, stream);
        case 5: return launch_covalent<5>(a, stream);
        case 6: return launch_covalent<6>(a, stream);
        case 7: return launch_covalent<7>(a, stream);
        case 8: return launch_covalent<8>(a, stream);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_listed_covalent_pairs(const CovalentArgs& a, const FullPairArgs& f, cudaStream_t stream, int* launches) {
    const size_t smem = sizeof(double) * kListedWarps * 32 * listed_slot(a.ka);
    const cudaError_t err = allow_dynamic_smem((const void*)listed_covalent_pairs, smem);
    if (err != cudaSuccess) return err;
    // at most a warp per four pairs of the table: the list is usually empty
    const long long pairs = (long long)a.n_strings * (a.n_strings + 1) / 2, grid = (pairs + 4 * kListedWarps - 1) / (4 * kListedWarps);
    listed_covalent_pairs<<<(unsigned)(grid < 3 * kSms ? grid : 3 * kSms), 32 * kListedWarps, smem, stream>>>(a, f);
    ++*launches;
    return cudaGetLastError();
}

}  // namespace vbcore
