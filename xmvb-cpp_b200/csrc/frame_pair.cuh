// Per-pair algebra of the left-string frame: adj B, det B, the quadratic two-electron term and the
// certificate of one pair, in the thread that calls (spin_frame.cu, covalent_pairs.cu).
#pragma once

#include "frame.cuh"

namespace vbcore {

// What phase A leaves of one pair: d = sign det S_LL, detb = det B, quad = the quadratic two-electron
// term times det B, the hole mask and the slot maps (hmap: nibble c = hole slot of position c, pmap:
// nibble b = particle slot of complement index b, 0xF elsewhere).  adj B = det B B^-1 goes to
// yrow[j E + i] (hole slot j, particle slot i).
struct FramePair {
    double d, detb, quad;
    unsigned hm, hmap, pmap;
    bool ok;         // evaluated here (else listed for the exact path)
    bool certified;  // well conditioned under the certificate
};

// Phase A at excitation level E <= 5, by minors: every quantity is a polynomial in the E x E entries
// of B = P[p, h], so nothing is divided by det B and blocks of any rank come out right (in the
// reference's terms: singular values below its 1e-12 are not truncated, a difference of that order).
// For each particle pair I (ascending) the minors m(J^c) of the other E - 2 rows over the columns
// outside the hole pair J give the quadratic term, as the 2 x 2 minors of B^-1 are
// (-1)^(I + J) m / det B (Jacobi); one more row of the Laplace expansion gives adj B, the last one
// det B.  700 multiply-adds at E = 5 and 160 at E = 4 (36 % of the pairs at K = 7), no division and
// no pivoting: the Gauss-Jordan inverse with row selects before it needed both (n = 14, 5.9 M
// certified pairs: 1378 -> 1280 us for the kernel).  Uncertified pairs no longer go to the
// one-thread-per-block exact path: 14 stretched hydrogen atoms, 268 ms -> 1.3 ms here and 3.0 ms for
// the levels E >= 6.
template <int E, class View>
__device__ __forceinline__ FramePair frame_pair_minors(const View& f, unsigned desc, double* __restrict__ yrow) {
    const int CP = f.cp();
    constexpr int EE = E > 0 ? E : 1;
    constexpr int NP = E > 1 ? E * (E - 1) / 2 : 1;
    FramePair o;
    o.hm = desc & 0xFFu;
    int hc[EE], pb[EE];  // holes (positions in L) and particles (Lbar indices), ascending
    {
        unsigned h = o.hm, pm = (desc >> 8) & 0xFFu;
#pragma unroll
        for (int j = 0; j < E; ++j) {
            hc[j] = __ffs(h) - 1;
            h &= h - 1;
            pb[j] = __ffs(pm) - 1;
            pm &= pm - 1;
        }
    }
    const double* P = f.p();
    double b[EE][EE];
#pragma unroll
    for (int i = 0; i < E; ++i)
#pragma unroll
        for (int j = 0; j < E; ++j) b[i][j] = P[pb[i] * f.k() + hc[j]];
    double detb = 1.0, quad = 0.0, na2 = 0.0;
    if constexpr (E == 1) {
        detb = b[0][0];
        na2 = 1.0;
        yrow[0] = 1.0;
    }
    if constexpr (E >= 2) {
        const double* Q = f.q();
        int cp[NP];
#pragma unroll
        for (int j2 = 1; j2 < E; ++j2)
#pragma unroll
            for (int j1 = 0; j1 < j2; ++j1) cp[pair_slot(j1, j2)] = hc[j2] * (hc[j2] - 1) / 2 + hc[j1];
        // row i of the cofactors from the minors m of rows (all but i and r) by expansion along row r
        auto cofactor_row = [&](const double (&m)[NP], int i, int r, bool last) {
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
                yrow[j * E + i] = acc;
                na2 = fma(acc, acc, na2);
                if (last) detb = j == 0 ? b[i][j] * acc : fma(b[i][j], acc, detb);
            }
        };
#pragma unroll
        for (int i2 = 1; i2 < E; ++i2)
#pragma unroll
            for (int i1 = 0; i1 < i2; ++i1) {
                double m[NP];
                if constexpr (E == 2) {
                    m[0] = 1.0;
                } else if constexpr (E == 3) {
                    const int ra = nth_other(i1, i2, 0);
#pragma unroll
                    for (int j2 = 1; j2 < E; ++j2)
#pragma unroll
                        for (int j1 = 0; j1 < j2; ++j1) m[pair_slot(j1, j2)] = b[ra][nth_other(j1, j2, 0)];
                } else if constexpr (E == 4) {
                    const int ra = nth_other(i1, i2, 0), rb = nth_other(i1, i2, 1);
#pragma unroll
                    for (int j2 = 1; j2 < E; ++j2)
#pragma unroll
                        for (int j1 = 0; j1 < j2; ++j1) {
                            const int x = nth_other(j1, j2, 0), y = nth_other(j1, j2, 1);
                            m[pair_slot(j1, j2)] = fma(b[ra][x], b[rb][y], -b[ra][y] * b[rb][x]);
                        }
                } else {
                    const int ra = nth_other(i1, i2, 0), rb = nth_other(i1, i2, 1), rc = nth_other(i1, i2, 2);
                    double m2[NP];
#pragma unroll
                    for (int y = 1; y < E; ++y)
#pragma unroll
                        for (int x = 0; x < y; ++x) m2[pair_slot(x, y)] = fma(b[ra][x], b[rb][y], -b[ra][y] * b[rb][x]);
#pragma unroll
                    for (int j2 = 1; j2 < E; ++j2)
#pragma unroll
                        for (int j1 = 0; j1 < j2; ++j1) {
                            const int x = nth_other(j1, j2, 0), y = nth_other(j1, j2, 1), z = nth_other(j1, j2, 2);
                            m[pair_slot(j1, j2)] =
                                fma(b[rc][x], m2[pair_slot(y, z)],
                                    fma(-b[rc][y], m2[pair_slot(x, z)], b[rc][z] * m2[pair_slot(x, y)]));
                        }
                }
                const double* q = Q + (pb[i2] * (pb[i2] - 1) / 2 + pb[i1]) * CP;
                double part = 0.0;
#pragma unroll
                for (int j2 = 1; j2 < E; ++j2)
#pragma unroll
                    for (int j1 = 0; j1 < j2; ++j1) {
                        const double v = m[pair_slot(j1, j2)];
                        part = fma(((i1 + i2 + j1 + j2) & 1) ? -v : v, q[cp[pair_slot(j1, j2)]], part);
                    }
                quad += part;
                if (i2 == E - 1) {
                    cofactor_row(m, i1, E - 1, false);
                    if (i1 == E - 2) cofactor_row(m, E - 1, E - 2, true);
                }
            }
    }
    const double* scal = f.scal();
    o.d = ((desc >> 16) & 1u ? -1.0 : 1.0) * scal[0];
    o.detb = detb;
    o.quad = quad;
    o.certified = frame_certificate<E>(f, hc, pb, na2, detb);
    o.ok = o.certified || (scal[1] * scal[2] < kFrameCondition2 && isfinite(detb) && isfinite(na2) && isfinite(quad));
    o.hmap = o.pmap = 0xFFFFFFFFu;
#pragma unroll
    for (int j = 0; j < E; ++j) {
        o.hmap &= ~((0xFu ^ (unsigned)j) << (4 * hc[j]));
        o.pmap &= ~((0xFu ^ (unsigned)j) << (4 * pb[j]));
    }
    return o;
}

// Phase A at the levels E >= 6 (about 1.5 % of the pairs at K = 7): Gauss-Jordan inverse of B with
// partial pivoting; uncertified blocks are listed.
template <int E, class View>
__device__ __forceinline__ FramePair frame_pair_inverse(const View& f, unsigned desc, double* __restrict__ yrow) {
    const int CP = f.cp();
    FramePair o;
    o.hm = desc & 0xFFu;
    int hc[E], pb[E];
    {
        unsigned h = o.hm, pm = (desc >> 8) & 0xFFu;
#pragma unroll
        for (int j = 0; j < E; ++j) {
            hc[j] = __ffs(h) - 1;
            h &= h - 1;
            pb[j] = __ffs(pm) - 1;
            pm &= pm - 1;
        }
    }
    const double* P = f.p();
    double x[E][E];
#pragma unroll
    for (int i = 0; i < E; ++i)
#pragma unroll
        for (int j = 0; j < E; ++j) x[i][j] = P[pb[i] * f.k() + hc[j]];
    int lab[E];
#pragma unroll
    for (int i = 0; i < E; ++i) lab[i] = i;
    double detb = 1.0;
#pragma unroll
    for (int s = 0; s < E; ++s) {
        int p = s;
        double best = fabs(x[s][s]);
#pragma unroll
        for (int i = s + 1; i < E; ++i) {
            const double av = fabs(x[i][s]);
            if (av > best) {
                best = av;
                p = i;
            }
        }
#pragma unroll
        for (int i = s + 1; i < E; ++i) {
            const bool sw = (p == i);
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const double a0 = x[s][j], a1 = x[i][j];
                x[s][j] = sw ? a1 : a0;
                x[i][j] = sw ? a0 : a1;
            }
            const int l0 = lab[s], l1 = lab[i];
            lab[s] = sw ? l1 : l0;
            lab[i] = sw ? l0 : l1;
        }
        if (p != s) detb = -detb;
        const double piv = x[s][s];
        detb *= piv;
        const double ip = 1.0 / piv;
        x[s][s] = 1.0;
#pragma unroll
        for (int j = 0; j < E; ++j) x[s][j] *= ip;
#pragma unroll
        for (int i = 0; i < E; ++i) {
            if (i == s) continue;
            const double f = x[i][s];
            x[i][s] = 0.0;
#pragma unroll
            for (int j = 0; j < E; ++j) x[i][j] = fma(-f, x[s][j], x[i][j]);
        }
    }
    // x[j][jj] = B^-1(j, lab[jj]): hole slot j, particle slot lab[jj]
    double na2 = 0.0;
#pragma unroll
    for (int i = 0; i < E; ++i)
#pragma unroll
        for (int j = 0; j < E; ++j) {
            const double v = detb * x[i][j];
            na2 = fma(v, v, na2);
        }
    // packed particle Lbar indices by slot, to read the particle of a permuted column
    uint64_t bword = 0;
#pragma unroll
    for (int i = 0; i < E; ++i) bword |= (uint64_t)pb[i] << (8 * i);
    int bj[E];
#pragma unroll
    for (int jj = 0; jj < E; ++jj) bj[jj] = (int)((bword >> (8 * lab[jj])) & 0xFFu);
    double quad = 0.0;
    const double* Q = f.q();
#pragma unroll
    for (int j1 = 0; j1 < E; ++j1)
#pragma unroll
        for (int j2 = j1 + 1; j2 < E; ++j2) {
            const int cp = hc[j2] * (hc[j2] - 1) / 2 + hc[j1];
            double part = 0.0;
#pragma unroll
            for (int jj1 = 0; jj1 < E; ++jj1)
#pragma unroll
                for (int jj2 = jj1 + 1; jj2 < E; ++jj2) {
                    const int ba = bj[jj1], bb = bj[jj2];
                    const bool ordered = ba < bb;
                    const int lo = ordered ? ba : bb, hi = ordered ? bb : ba;
                    const double m2 = fma(x[j1][jj1], x[j2][jj2], -x[j1][jj2] * x[j2][jj1]);
                    const double qv = Q[(hi * (hi - 1) / 2 + lo) * CP + cp];
                    part = fma(ordered ? qv : -qv, m2, part);
                }
            quad += part;
        }
    o.d = ((desc >> 16) & 1u ? -1.0 : 1.0) * f.scal()[0];
    o.detb = detb;
    o.quad = detb * quad;
    o.certified = frame_certificate<E>(f, hc, pb, na2, detb);
    o.ok = o.certified;
    o.hmap = o.pmap = 0xFFFFFFFFu;
    if (o.ok) {
#pragma unroll
        for (int j = 0; j < E; ++j) {
            o.hmap &= ~((0xFu ^ (unsigned)j) << (4 * hc[j]));
            o.pmap &= ~((0xFu ^ (unsigned)j) << (4 * pb[j]));
#pragma unroll
            for (int jj = 0; jj < E; ++jj) yrow[j * E + lab[jj]] = detb * x[j][jj];
        }
    }
    return o;
}

// The high excitation levels out of line: their E x E registers do not count against the register
// budget of the common levels.
template <int E, class View>
__device__ __noinline__ FramePair frame_pair_out_of_line(const View* f, unsigned desc, double* __restrict__ yrow) {
    return frame_pair_inverse<E>(*f, desc, yrow);
}

// K: largest level
template <int K, class View>
__device__ __forceinline__ FramePair frame_pair_dispatch(int e, const View& f, unsigned desc, double* yrow) {
    FramePair o{};
#define VB_FRAME_CASE(E_)                                             \
    case E_:                                                          \
        if constexpr (E_ <= K) {                                      \
            if constexpr (E_ > kMinorsEMax)                           \
                o = frame_pair_out_of_line<E_>(&f, desc, yrow);       \
            else                                                      \
                o = frame_pair_minors<E_>(f, desc, yrow);             \
        }                                                             \
        break;
    switch (e) {
        VB_FRAME_CASE(0)
        VB_FRAME_CASE(1)
        VB_FRAME_CASE(2)
        VB_FRAME_CASE(3)
        VB_FRAME_CASE(4)
        VB_FRAME_CASE(5)
        VB_FRAME_CASE(6)
        VB_FRAME_CASE(7)
        VB_FRAME_CASE(8)
        default: break;
    }
#undef VB_FRAME_CASE
    return o;
}

}  // namespace vbcore
