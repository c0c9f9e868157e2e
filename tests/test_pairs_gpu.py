"""GPU parity of the determinant-pair path through the C ABI against the oracle.

Tolerances are the north-star bar for structure matrices: 1e-10 relative on every H/S element
(relative to max(1, max |H|)), and the reference's own per-pair closeness for the determinant
level."""

import numpy as np
import pytest

import oracle as O
import vbcore
from vbcore import workloads
from conftest import golden_cases, load_golden

pytestmark = pytest.mark.gpu
REL = 1e-10


@pytest.fixture(scope="module")
def ctx():
    c = vbcore.Context(0)
    yield c
    c.close()


def _rel(a, b):
    return np.abs(a - b).max() / max(1.0, np.abs(b).max())


def _plan(ctx, kw, n, nel, mult=1):
    rows = vbcore.generate_structures(kw, n, nel, mult)
    ex = vbcore.expand_structures(rows, nel, mult)
    return vbcore.HsPlan(ctx, ex, n), O.expand(O.generate_structures(kw, n, nel, mult), nel, mult)


@pytest.mark.parametrize("name", golden_cases())
def test_structure_matrices_match_golden(ctx, name):
    z = load_golden(name)
    n, nel, mult, kw = int(z["n"]), int(z["n_el"]), int(z["mult"]), str(z["keyword"])
    plan, _ = _plan(ctx, kw, n, nel, mult)
    H, S = plan.execute(z["S"], z["h"], z["eri"])
    assert _rel(H, z["Hs"]) < REL
    assert _rel(S, z["Ss"]) < REL


@pytest.mark.parametrize("kw,n,seed", [("COV", 8, 1), ("COV", 10, 2), ("COV", 12, 3), ("COV ION(1)", 8, 4),
                                       ("COV ION(1)", 6, 5), ("FULL", 6, 6), ("COV ION(1)", 10, 7)])
def test_structure_matrices_match_oracle(ctx, kw, n, seed):
    S, h, eri = workloads.active_space(n, 3 * n, seed)
    plan, ex = _plan(ctx, kw, n, n)
    H, So = plan.execute(S, h, eri)
    Hr, Sr, _ = O.structure_matrices(n, ex, S, h, eri)
    assert _rel(H, Hr) < REL
    assert _rel(So, Sr) < REL
    assert np.array_equal(H, H.T) and np.array_equal(So, So.T)
    st = plan.stats()
    assert st["spin_pairs"] > 0 and st["kernel_launches"] >= 5
    # (ij|kl) = sum_P B_ij^P B_kl^P with 3n auxiliary functions: the factorization stops at that rank
    assert st["factor_columns"] == min(3 * n, n * (n + 1) // 2)
    if n <= 8:
        # one evaluation per orbit {(d, e), (flip d, flip e)} of unordered pairs (brute force)
        n_det = ex.n_determinants
        index = {(int(a), int(b)): d for d, (a, b) in enumerate(zip(ex.det_alpha, ex.det_beta))}
        flip = [index.get((int(b), int(a))) for a, b in zip(ex.det_alpha, ex.det_beta)]
        orbits = set()
        for d in range(n_det):
            for e in range(d, n_det):
                if None in (flip[d], flip[e]):
                    orbits.add((d, e))
                    continue
                f = tuple(sorted((flip[d], flip[e])))
                orbits.add(min((d, e), f))
        if None in flip:
            assert st["determinant_pairs"] == n_det * (n_det + 1) // 2
        else:
            assert st["determinant_pairs"] == len(orbits)


def test_open_shell_tables(ctx):
    # doublet and triplet: alpha and beta string tables differ
    for n, nel, mult in ((5, 5, 2), (6, 4, 3), (7, 6, 3)):
        S, h, eri = workloads.active_space(n, 2 * n, 11 + n)
        plan, ex = _plan(ctx, "COV", n, nel, mult)
        H, So = plan.execute(S, h, eri)
        Hr, Sr, _ = O.structure_matrices(n, ex, S, h, eri)
        assert _rel(H, Hr) < REL and _rel(So, Sr) < REL


def test_orthogonal_orbitals_take_the_exact_path(ctx):
    z = load_golden("orthogonal_n6")
    plan, _ = _plan(ctx, str(z["keyword"]), int(z["n"]), int(z["n_el"]))
    H, S = plan.execute(z["S"], z["h"], z["eri"])
    assert _rel(H, z["Hs"]) < REL and _rel(S, z["Ss"]) < REL
    st = plan.stats()
    assert st["careful_spin_pairs"] > 0  # singular blocks (nullity 1, 2, ...) present


def test_determinant_pairs_match_oracle(ctx):
    n = 8
    S, h, eri = workloads.active_space(n, 24, 7)
    plan, ex = _plan(ctx, "COV ION(1)", n, n)
    Hd, Sd = O.determinant_matrices(n, ex.det_alpha_occ, ex.det_beta_occ, S, h, eri)
    rng = np.random.default_rng(0)
    pairs = rng.integers(0, ex.n_determinants, size=(4000, 2))
    ho, so = plan.determinant_pairs(S, h, eri, pairs)
    assert np.abs(ho - Hd[pairs[:, 0], pairs[:, 1]]).max() < REL * max(1.0, np.abs(Hd).max())
    assert np.abs(so - Sd[pairs[:, 0], pairs[:, 1]]).max() < REL * max(1.0, np.abs(Sd).max())


def test_determinant_pairs_in_device_memory_use_the_callers_order(ctx):
    # this covalent + ionic list is reordered inside the plan (determinants grouped by the first
    # structure group using them); pair indices in device memory are mapped like host ones
    import ctypes
    import torch
    n = 8
    S, h, eri = workloads.active_space(n, 24, 7)
    plan, ex = _plan(ctx, "COV ION(1)", n, n)
    rng = np.random.default_rng(1)
    pairs = rng.integers(0, ex.n_determinants, size=(3000, 2)).astype(np.int64)
    ho, so = plan.determinant_pairs(S, h, eri, pairs)
    dev = torch.device("cuda", 0)
    dS = torch.tensor(np.ascontiguousarray(S.T), device=dev)
    dh = torch.tensor(np.ascontiguousarray(h.T), device=dev)
    de = torch.tensor(np.ascontiguousarray(eri, dtype=np.float64), device=dev)
    dp = torch.tensor(pairs, device=dev)
    dho = torch.zeros(len(pairs), dtype=torch.float64, device=dev)
    dso = torch.zeros(len(pairs), dtype=torch.float64, device=dev)
    torch.cuda.synchronize()
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    st = vbcore.load_library().vb_hs_plan_determinant_pairs(plan._h, p(dS), p(dh), p(de), len(pairs), p(dp),
                                                            vbcore.VB_MEM_DEVICE, p(dho), p(dso))
    assert st == 0
    assert np.array_equal(dho.cpu().numpy(), ho) and np.array_equal(dso.cpu().numpy(), so)


@pytest.mark.parametrize("k", [1, 2, 3, 4, 6, 7, 9])
def test_resolve_overlaps_reference_semantics(ctx, k):
    rng = np.random.default_rng(k)
    blocks = []
    for drop in range(0, min(k, 3) + 1):
        for _ in range(6):
            x = rng.standard_normal((k, k))
            if drop:
                u, s, vt = np.linalg.svd(x)
                s[k - drop:] = 0.0
                x = (u * s) @ vt
            blocks.append(x)
    blocks.append(np.zeros((k, k)))
    blocks = np.array(blocks)
    det, nul, cof = ctx.resolve_overlaps(blocks)
    for i, x in enumerate(blocks):
        d_ref, n_ref, _, c_ref = O.resolve(x)
        assert nul[i] == n_ref
        assert abs(det[i] - d_ref) <= 1e-12 * max(1.0, abs(d_ref))
        assert np.abs(cof[i] - c_ref).max() <= 1e-11 * max(1.0, np.abs(c_ref).max())


def test_same_spin_pairs_match_oracle(ctx):
    n, k = 10, 5
    S, h, eri = workloads.active_space(n, 30, 3)
    rng = np.random.default_rng(5)
    L = np.array([np.sort(rng.choice(n, k, replace=False)) for _ in range(300)])
    R = np.array([np.sort(rng.choice(n, k, replace=False)) for _ in range(300)])
    R[:20] = L[:20]  # diagonal pairs
    sc, cof = ctx.same_spin_pairs(n, L, R, S, h, eri)
    for i in range(len(L)):
        ref = O.spin_pair(n, L[i], R[i], S, h, eri)
        assert int(sc[i, 3]) == ref["nullity"]
        for j, key in enumerate(("det", "h1", "htot")):
            assert abs(sc[i, j] - ref[key]) <= 1e-11 * max(1.0, abs(ref[key]))


def test_reproducible_and_device_path(ctx):
    import torch
    n = 10
    S, h, eri = workloads.active_space(n, 30, 9)
    plan, _ = _plan(ctx, "COV", n, n)
    H1, S1 = plan.execute(S, h, eri)
    H2, S2 = plan.execute(S, h, eri)
    assert np.array_equal(H1, H2) and np.array_equal(S1, S2)
    dev = torch.device("cuda:0")
    tS = torch.tensor(S.T.copy(), device=dev)
    th = torch.tensor(h.T.copy(), device=dev)
    te = torch.tensor(eri, device=dev)
    ns = plan.n_structures
    tH = torch.empty((ns, ns), dtype=torch.float64, device=dev)
    tSo = torch.empty((ns, ns), dtype=torch.float64, device=dev)
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    plan.execute_device(tS.data_ptr(), th.data_ptr(), te.data_ptr(), tH.data_ptr(), tSo.data_ptr())
    torch.cuda.synchronize()
    ctx.set_stream(None)
    assert np.array_equal(tH.cpu().numpy().T, H1) and np.array_equal(tSo.cpu().numpy().T, S1)


def test_full_size_microbenchmark_properties(ctx):
    """n_active = 14, 3432 determinants, 429 structures (the microbenchmark shape): every one of
    the 429 x 429 H and S elements against the oracle (all 5,891,028 unordered determinant pairs,
    all host threads), plus size-independent properties (symmetry, positive metric, linearity of H
    in (h, (ij|kl)))."""
    import os

    n = 14
    S, h, eri = workloads.active_space(n, 42, 2026)
    plan, ex = _plan(ctx, "COV", n, n)
    H, So = plan.execute(S, h, eri)
    assert H.shape == (429, 429)
    ex_o = O.expand(O.generate_structures("COV", n, n), n)
    Hr, Sr, done = O.structure_matrices(n, ex_o, S, h, eri, threads=os.cpu_count() or 1)
    assert done == 3432 * 3433 // 2
    scale_h = max(1.0, np.abs(Hr).max())
    scale_s = max(1.0, np.abs(Sr).max())
    assert np.abs(H - Hr).max() <= REL * scale_h
    assert np.abs(So - Sr).max() <= REL * scale_s
    assert np.array_equal(H, H.T)
    assert np.linalg.eigvalsh(So).min() > 0
    H1, S1 = plan.execute(S, h, np.zeros_like(eri))
    H2, S2 = plan.execute(S, np.zeros_like(h), eri)
    assert np.array_equal(S1, So) and np.array_equal(S2, So)
    assert np.abs(H1 + H2 - H).max() <= 1e-12 * scale_h


@pytest.mark.parametrize("kw,n,nel", [("COV", 8, 6), ("COV", 10, 8), ("COV ION(1)", 6, 2), ("COV", 5, 2),
                                      ("FULL", 5, 4), ("COV ION(1)", 7, 6)])
def test_more_orbitals_than_electrons(ctx, kw, n, nel):
    """Active spaces with n > 2k (complements larger than the strings): every excitation level
    from 0 to min(k, n - k) occurs in the frame kernel."""
    S, h, eri = workloads.active_space(n, 3 * n, 40 + n + nel)
    plan, ex = _plan(ctx, kw, n, nel)
    H, So = plan.execute(S, h, eri)
    Hr, Sr, _ = O.structure_matrices(n, ex, S, h, eri)
    assert _rel(H, Hr) < REL and _rel(So, Sr) < REL


@pytest.mark.parametrize("n,k", [(3, 1), (6, 2), (7, 3), (8, 4), (9, 5), (10, 6), (10, 7), (11, 8), (9, 8)])
def test_spin_pair_records_every_electron_count(n, k):
    """Every spin pair of a complete string table (det, one-electron and total same-spin energy,
    nullity) against the oracle for k = 1 .. 8, through the allocation-free entry point (which
    returns the record scalars of the same kernels); one random and one stretched overlap."""
    import itertools

    import torch

    masks = sorted(sum(1 << o for o in occ) for occ in itertools.combinations(range(n), k))
    N = len(masks)
    n_pairs = N * (N + 1) // 2
    occ = [[o for o in range(n) if (m >> o) & 1] for m in masks]
    S0, h, eri = workloads.active_space(n, 2 * n, 90 + 10 * n + k)
    idx = np.arange(n)
    S1 = np.exp(-0.8 * np.abs(idx[:, None] - idx[None, :]))  # overlaps decaying along a chain
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(n * 100 + k)
    sample = rng.choice(n_pairs, size=min(n_pairs, 3000), replace=False)
    for S in (S0, S1):
        d_masks = torch.tensor(np.array(masks, dtype=np.uint64).view(np.int64), device=dev)
        dS = torch.tensor(np.ascontiguousarray(S.T), device=dev)
        dh = torch.tensor(np.ascontiguousarray(h.T), device=dev)
        de = torch.tensor(eri, device=dev)
        out = torch.full((4 * n_pairs,), float("nan"), dtype=torch.float64, device=dev)
        torch.cuda.synchronize()
        vbcore.spin_pairs_noalloc(torch.cuda.current_stream(dev).cuda_stream, n, k, N, d_masks.data_ptr(),
                                  dS.data_ptr(), dh.data_ptr(), de.data_ptr(), out.data_ptr())
        torch.cuda.synchronize()
        got = out.cpu().numpy().reshape(n_pairs, 4)
        uu = np.repeat(np.arange(N), np.arange(N, 0, -1))
        vv = np.concatenate([np.arange(u, N) for u in range(N)])
        for t in sample:
            ref = O.spin_pair(n, occ[uu[t]], occ[vv[t]], S, h, eri)
            assert int(got[t, 3]) == ref["nullity"]
            for col, key in ((0, "det"), (1, "h1"), (2, "htot")):
                assert abs(got[t, col] - ref[key]) <= REL * max(1.0, abs(ref[key])), (n, k, t, key)


def test_band_reduction_wait_timeout_is_reported_and_the_plan_recovers():
    """The band reduction's tile waits are bounded: with a one-poll limit the first wait gives up,
    the CTAs flag it and leave after their copies in flight land, and the execute returns
    VB_ERR_TIMEOUT (no trap, no hang); with the default limit restored the same plan evaluates
    the structure matrices."""
    n = 8
    S, h, eri = workloads.active_space(n, 3 * n, 21)
    c = vbcore.Context(0)
    try:
        plan, ex = _plan(c, "COV", n, n)
        c.set_barrier_spin_limit(1)
        with pytest.raises(vbcore.VbError) as e:
            plan.execute(S, h, eri)
        assert e.value.status == 6 and "band_reduce" in str(e.value)
        c.set_barrier_spin_limit(0)
        H, So = plan.execute(S, h, eri)
        Hr, Sr, _ = O.structure_matrices(n, ex, S, h, eri)
        assert _rel(H, Hr) < REL and _rel(So, Sr) < REL
        plan.close()
    finally:
        c.close()


@pytest.mark.parametrize("kw,n,nel,mult", [("COV", 8, 8, 3), ("COV", 9, 2, 1), ("COV", 10, 4, 1), ("COV", 11, 11, 4),
                                           ("COV", 12, 12, 3), ("COV", 13, 13, 4)])
def test_wide_complements_take_the_frame_kernel(ctx, kw, n, nel, mult):
    """Strings of k electrons with up to eight empty orbitals, more than a closed shell has (open
    shells: 5 + 3, 7 + 4, 7 + 5, 8 + 5 electrons; one and two electrons over nine and ten
    orbitals): well-conditioned overlaps leave (almost) nothing to the exact path, and the
    structure matrices match the oracle."""
    S, h, eri = workloads.active_space(n, 2 * n, 60 + n)
    plan, ex = _plan(ctx, kw, n, nel, mult)
    H, So = plan.execute(S, h, eri)
    Hr, Sr, _ = O.structure_matrices(n, ex, S, h, eri)
    assert _rel(H, Hr) < REL and _rel(So, Sr) < REL
    st = plan.stats()
    assert st["careful_spin_pairs"] <= st["spin_pairs"] // 100


@pytest.mark.parametrize("kw,n,nel,mult", [("COV ION(1)", 8, 8, 1), ("COV ION(1)", 9, 9, 2), ("COV ION(1)", 8, 8, 3),
                                           ("COV ION(1)", 10, 10, 1), ("COV ION(1-2)", 8, 8, 1), ("FULL", 6, 6, 1),
                                           ("COV ION(1)", 9, 8, 1)])
def test_block_ordered_determinants_match_oracle(ctx, kw, n, nel, mult):
    """Determinant lists that fill blocks of alpha x beta strings (5 x 5 to 8 x 8, with and without
    empty cells, equal and unequal string tables, sets cut into several blocks): structure matrices
    against the oracle, through host and device pointers, and determinant pairs in the caller's order."""
    S, h, eri = workloads.active_space(n, 2 * n, 80 + n)
    plan, ex = _plan(ctx, kw, n, nel, mult)
    H, So = plan.execute(S, h, eri)
    Hr, Sr, _ = O.structure_matrices(n, ex, S, h, eri, threads=8)
    assert _rel(H, Hr) < REL and _rel(So, Sr) < REL
    H2, S2 = plan.execute(S, h, eri)
    assert np.array_equal(H, H2) and np.array_equal(So, S2)
    rng = np.random.default_rng(n)
    pairs = rng.integers(0, plan.expansion.n_determinants, size=(500, 2))
    ho, so = plan.determinant_pairs(S, h, eri, pairs)
    a, b = plan.expansion.occupations(), plan.expansion.occupations(beta=True)
    for q, (d, e) in enumerate(pairs[:100]):
        x = S[np.ix_(a[e], a[d])]
        y = S[np.ix_(b[e], b[d])]
        ref = np.linalg.det(x) * np.linalg.det(y)
        assert abs(so[q] - ref) < 1e-11 * max(1.0, abs(ref))


def _full_blocks(n, holders):
    """An expansion over n orbitals whose determinants fill 8 x 8 blocks but for the diagonal: for each of
    the last `holders` orbitals x, the alpha strings {x, c} and the beta strings (orbitals 0 .. 7 without e),
    c != e; structures of one to three random determinants."""
    rng = np.random.default_rng(n)
    alpha = sorted((1 << (n - 1 - x)) | (1 << c) for x in range(holders) for c in range(8))
    beta = sorted(0xFF ^ (1 << e) for e in range(8))
    dets = sorted((i, k) for i, a in enumerate(alpha) for k, b in enumerate(beta) if bin(a & b).count("1") == 1)
    per_det = [[] for _ in dets]
    n_str = len(dets)
    for I in range(n_str):
        for d in {I, *rng.integers(0, len(dets), size=2).tolist()}:
            per_det[d].append((I, float(rng.choice([-1.0, 1.0]))))
    offsets = np.cumsum([0] + [len(t) for t in per_det]).astype(np.int64)
    ts = np.array([t[0] for d in per_det for t in sorted(d)], dtype=np.int32)
    tc = np.array([t[1] for d in per_det for t in sorted(d)])
    da, db = (np.array([d[q] for d in dets], dtype=np.int32) for q in (0, 1))
    ex = vbcore.Expansion(n_str, 2, 7, np.array(alpha, dtype=np.uint64), np.array(beta, dtype=np.uint64), da, db,
                          offsets, ts, tc)
    ref = O.Expansion(n_str, 2, 7, alpha, beta, da, db, offsets, ts, tc)
    ref.det_alpha_occ, ref.det_beta_occ = ex.occupations(), ex.occupations(beta=True)
    return ex, ref


@pytest.mark.parametrize("n", [18, 19, 20])
def test_block_ordered_lists_of_any_factor_rank(ctx, n):
    """Full-rank pair kernels of 171, 190 and 210 columns: the records of a pair of 8 x 8 blocks fit shared
    memory up to 186 columns (190 with 7 of 8 cells taken)."""
    ex, ref = _full_blocks(n, 10)
    S, h, _ = workloads.active_space(n, n, 40 + n)
    P = n * (n + 1) // 2
    B = 0.2 * np.random.default_rng(n).standard_normal((P, P))
    eri = workloads.pack_pair_kernel(B @ B.T / P + 0.01 * np.eye(P))
    plan = vbcore.HsPlan(ctx, ex, n)
    H, So = plan.execute(S, h, eri)
    assert plan.stats()["factor_columns"] == P
    Hr, Sr, _ = O.structure_matrices(n, ref, S, h, eri, threads=8)
    assert _rel(H, Hr) < REL and _rel(So, Sr) < REL
    plan.close()


@pytest.mark.parametrize("n,mult,budget_mb", [(8, 1, 0), (9, 2, 128), (10, 1, 0)])
def test_block_ordered_lists_with_the_tiled_reduction(ctx, n, mult, budget_mb):
    """Every term given twice with half its coefficient: the dense groups do not take repeated terms, so block
    pairs feed the tiled reduction, over one band and several."""
    S, h, eri = workloads.active_space(n, 2 * n, 50 + n)
    ref = O.expand(O.generate_structures("COV ION(1)", n, n, mult), n, mult)
    ex = vbcore.expand_structures(vbcore.generate_structures("COV ION(1)", n, n, mult), n, mult)
    ex.term_offsets = 2 * ex.term_offsets
    ex.term_structure = np.repeat(ex.term_structure, 2)
    ex.term_coefficient = 0.5 * np.repeat(ex.term_coefficient, 2)
    own = vbcore.Context(0, budget_mb << 20) if budget_mb else ctx
    plan = vbcore.HsPlan(own, ex, n)
    H, So = plan.execute(S, h, eri)
    Hr, Sr, _ = O.structure_matrices(n, ref, S, h, eri, threads=8)
    assert _rel(H, Hr) < REL and _rel(So, Sr) < REL
    plan.close()
    if budget_mb:
        own.close()


@pytest.mark.parametrize("n,mult,budget_mb", [(8, 1, 16), (8, 1, 24), (9, 2, 128), (10, 1, 400)])
def test_block_ordered_determinants_in_bands(ctx, n, mult, budget_mb):
    """Block-ordered lists over several bands of determinant columns (a small budget): bands end at block
    boundaries, 65 to 512 columns and not multiples of 16 apart.  A column of the determinant matrix and its
    sums do not depend on the band it is in: the bits of one band, and the oracle's matrices."""
    S, h, eri = workloads.active_space(n, 2 * n, 30 + n)
    plan, ex = _plan(ctx, "COV ION(1)", n, n, mult)
    H, So = plan.execute(S, h, eri)
    one = plan.stats()["kernel_launches"]
    small = vbcore.Context(0, budget_mb << 20)
    try:
        banded, _ = _plan(small, "COV ION(1)", n, n, mult)
        H2, S2 = banded.execute(S, h, eri)
        assert banded.stats()["kernel_launches"] >= one + 4  # two kernels a band
        assert np.array_equal(H, H2) and np.array_equal(So, S2)
        banded.close()
    finally:
        small.close()
    Hr, Sr, _ = O.structure_matrices(n, ex, S, h, eri, threads=8)
    assert _rel(H2, Hr) < REL and _rel(S2, Sr) < REL
    plan.close()


@pytest.mark.parametrize("n,mult", [(4, 1), (5, 2), (6, 1), (6, 3), (7, 4), (8, 1), (9, 2), (10, 3), (11, 2), (12, 1), (13, 2)])
@pytest.mark.parametrize("overlap", ["random", "orthogonal", "dependent"])
def test_covalent_pairs_match_records(ctx, n, mult, overlap):
    """Covalent lists take both spins of a determinant pair in one kernel; the same matrices from the
    spin-pair records (the listed determinant pairs of the same plan, all of them, contracted with the
    expansion here).  Closed and open shells, one pair per spin-flip orbit and all of them, levels 0 ..
    6, regular overlaps, overlaps of 0 (every excited block singular, the highest levels listed) and two
    nearly dependent orbitals (strings that hold both have kappa(S_LL) near 1e8 and are listed with all
    their pairs, or certified just below it).  Both forms add the same terms in another order, 1e-11 of
    the largest element; dependent orbitals: a certified block carries eps kappa_F < 2.2e-16 1e8 = 2.2e-8,
    and the two forms take a pair from either of its strings."""
    rng = np.random.default_rng(10 * n + mult)
    S, h, eri = workloads.active_space(n, 3 * n, 90 + n)
    if overlap == "orthogonal":
        S = np.eye(n)
    elif overlap == "dependent":
        C = np.eye(n) + 0.05 * rng.standard_normal((n, n))
        C[:, 1] = C[:, 0] + 1e-4 * C[:, 1]
        S = C.T @ C
        d = 1.0 / np.sqrt(np.diag(S))
        S = d[:, None] * S * d[None, :]
    tol = 2.2e-8 if overlap == "dependent" else 1e-11
    rows = vbcore.generate_structures("COV", n, n, mult)
    ex = vbcore.expand_structures(rows, n, mult)
    plan = vbcore.HsPlan(ctx, ex, n)
    H, So = plan.execute(S, h, eri)
    assert np.array_equal(H, H.T) and np.array_equal(So, So.T)
    oex = O.expand(O.generate_structures("COV", n, n, mult), n, mult)
    if n <= 8:
        Hr, Sr, _ = O.structure_matrices(n, oex, S, h, eri)
        assert _rel(H, Hr) < max(REL, tol) and _rel(So, Sr) < max(REL, tol)
    nd = ex.n_determinants
    pairs = np.array([(d, e) for d in range(nd) for e in range(d, nd)], dtype=np.int64)
    hd, sd = plan.determinant_pairs(S, h, eri, pairs)
    Hd = np.zeros((nd, nd))
    Sd = np.zeros((nd, nd))
    Hd[pairs[:, 0], pairs[:, 1]] = Hd[pairs[:, 1], pairs[:, 0]] = hd
    Sd[pairs[:, 0], pairs[:, 1]] = Sd[pairs[:, 1], pairs[:, 0]] = sd
    T = np.zeros((nd, plan.n_structures))
    off = ex.term_offsets
    for d in range(nd):
        T[d, ex.term_structure[off[d]:off[d + 1]]] = ex.term_coefficient[off[d]:off[d + 1]]
    assert _rel(H, T.T @ Hd @ T) < tol and _rel(So, T.T @ Sd @ T) < tol
    plan.close()


@pytest.mark.parametrize("n,mult", [(4, 1), (6, 1), (7, 2), (8, 1), (8, 3), (10, 1), (12, 1)])
def test_covalent_diagnostics_count_every_record_once(ctx, n, mult):
    """careful_spin_pairs: with orthogonal orbitals every pair of different strings has a singular block.  With
    two of them nearly dependent (kappa = 2e6) the strings that hold both list all their pairs, and with each
    the record of the other spin, which alone would be evaluated; no record is counted for both."""
    _, h, eri = workloads.active_space(n, 3 * n, 10 + n)
    rows = vbcore.generate_structures("COV", n, n, mult)
    ex = vbcore.expand_structures(rows, n, mult)
    plan = vbcore.HsPlan(ctx, ex, n)
    S = np.eye(n)
    plan.execute(S, h, eri)
    st = plan.stats()
    tables = [ex.alpha_strings] if mult == 1 else [ex.alpha_strings, ex.beta_strings]
    assert st["spin_pairs"] == sum(len(t) * (len(t) + 1) // 2 for t in tables)
    assert st["careful_spin_pairs"] == sum(len(t) * (len(t) - 1) // 2 for t in tables)
    S[0, 1] = S[1, 0] = 1.0 - 1e-6
    plan.execute(S, h, eri)
    singular = 0
    for t in tables:
        occ = [[i for i in range(n) if (int(s) >> i) & 1] for s in t]
        singular += sum(np.linalg.det(S[np.ix_(occ[u], occ[v])]) == 0.0 for u in range(len(t)) for v in range(u, len(t))) \
            if len(t) < 300 else 0
    assert singular <= plan.stats()["careful_spin_pairs"] <= st["spin_pairs"]
    plan.close()


@pytest.mark.parametrize("n,mult", [(8, 1), (10, 1), (10, 3), (11, 2), (12, 1)])
def test_covalent_pairs_list_only_the_side_that_fails(ctx, n, mult):
    """Two nearly dependent orbitals: a string that holds both leaves its uncertified pairs to the exact path,
    the complement's record is evaluated in its own frame.  No more records outside the certificate than the
    records path has (its frames are those of the lower string of every pair: 10 %), where listing both sides
    gave nearly twice as many."""
    rng = np.random.default_rng(n)
    C = np.eye(n) + 0.05 * rng.standard_normal((n, n))
    C[:, 1] = C[:, 0] + 2e-3 * C[:, 1]
    S = C.T @ C
    d = 1.0 / np.sqrt(np.diag(S))
    S = d[:, None] * S * d[None, :]
    _, h, eri = workloads.active_space(n, 3 * n, 90 + n)
    plan, _ = _plan(ctx, "COV", n, n, mult)
    plan.execute(S, h, eri)
    covalent = plan.stats()["careful_spin_pairs"]
    plan.determinant_pairs(S, h, eri, np.array([[0, 0]]))
    records = plan.stats()["careful_spin_pairs"]
    assert records > 0 and covalent <= 1.1 * records + 10
    plan.close()


@pytest.mark.parametrize("n", [2, 3, 7, 8, 10, 11, 13, 14, 15, 16, 17])
@pytest.mark.parametrize("kernel", ["definite", "indefinite", "low_rank", "tied"])
def test_pair_kernel_factorization_sizes(ctx, n, kernel):
    """Two electrons: H_de holds (ij|kl) itself through the factored pair kernel, sum_m sigma_m l_m l_m^T.
    Row counts 3 .. 153 at the edges of the factorization's launch classes (32, 64, 96, 128, 152 rows and
    the general form), pivots of both signs, early stop and equal diagonals."""
    P = n * (n + 1) // 2
    rng = np.random.default_rng(n)
    S, h, _ = workloads.active_space(n, 3 * n, 60 + n)
    B = rng.standard_normal((P, P))
    K = {"definite": lambda: B @ B.T / P, "indefinite": lambda: 0.5 * (B + B.T),
         "low_rank": lambda: B[:, :n] @ B[:, :n].T / n,
         "tied": lambda: np.eye(P) + 0.01 * np.sign(np.triu(B, 1) + np.triu(B, 1).T)}[kernel]()
    eri = workloads.pack_pair_kernel(K)
    plan, ex = _plan(ctx, "COV", n, 2)
    H, So = plan.execute(S, h, eri)
    Hr, Sr, _ = O.structure_matrices(n, ex, S, h, eri)
    assert _rel(H, Hr) < REL and _rel(So, Sr) < REL
    assert plan.stats()["factor_columns"] == (n if kernel == "low_rank" else P)
    plan.close()


@pytest.mark.parametrize("n,mult", [(8, 1), (10, 3)])
def test_small_budget_takes_records_and_exact_path(ctx, n, mult):
    """A budget without room for the covalent pair lists (and an open shell's frame tables) beside what
    later calls may take: the plan works from records; same matrices (same bound as above)."""
    S, h, eri = workloads.active_space(n, 3 * n, n)
    plan, _ = _plan(ctx, "COV", n, n, mult)
    H, So = plan.execute(S, h, eri)
    small = vbcore.Context(0, 200 << 20)
    try:
        tight, _ = _plan(small, "COV", n, n, mult)
        H2, S2 = tight.execute(S, h, eri)
        assert _rel(H2, H) < 1e-11 and _rel(S2, So) < 1e-11
        tight.close()
    finally:
        small.close()
