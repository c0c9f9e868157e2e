"""Metric Cholesky and the dense generalized eigenproblem on the device against LAPACK
(dpotrf / dsygvd through SciPy, the routines the reference's Eigen LLT and
GeneralizedEigensolver::solve_dense stand on)."""

import numpy as np
import pytest

import oracle as O
import vbcore
from vbcore import workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = vbcore.Context(0)
    yield c
    c.close()


def _random_symmetric(n, seed):
    rng = np.random.default_rng(seed)
    a = rng.standard_normal((n, n))
    return 0.5 * (a + a.T)


@pytest.mark.parametrize("n", [1, 2, 5, 31, 32, 33, 64, 97, 200, 429, 1000])
@pytest.mark.parametrize("cond", [1e2, 1e6, 1e10])
def test_cholesky_matches_lapack(ctx, n, cond):
    S = O.conditioned_metric(n, cond, seed=n)
    U = vbcore.metric_cholesky(ctx, S)
    assert np.array_equal(U, np.triu(U))
    backward = np.linalg.norm(U.T @ U - S) / np.linalg.norm(S)
    assert backward < 1e-15 * max(1, n) ** 0.5 * 4
    Ur = O.metric_cholesky(S)
    # forward error of a Cholesky factor is bounded by cond(S) eps
    assert np.abs(U - Ur).max() <= 1e-15 * cond * np.abs(Ur).max() * 10


def test_cholesky_reads_upper_triangle_only(ctx):
    S = O.conditioned_metric(40, 1e3, seed=3)
    Sl = np.triu(S) + np.tril(np.full_like(S, 7.0), -1)  # garbage below the diagonal
    assert np.abs(vbcore.metric_cholesky(ctx, Sl) - O.metric_cholesky(S)).max() < 1e-12


@pytest.mark.parametrize("n,bad", [(10, 4), (70, 40), (150, 1), (300, 200)])
def test_cholesky_reports_the_failing_minor(ctx, n, bad):
    S = O.conditioned_metric(n, 1e2, seed=n)
    S[bad - 1, bad - 1] = -1.0  # leading minor of order `bad` is the first that is not positive
    with pytest.raises(vbcore.VbError) as e:
        vbcore.metric_cholesky(ctx, S)
    assert e.value.status == 4 and e.value.info == bad


@pytest.mark.parametrize("n", [1, 2, 3, 5, 14, 42, 97, 132, 429])
def test_generalized_eigh_matches_dsygvd(ctx, n):
    H = _random_symmetric(n, 100 + n)
    S = O.conditioned_metric(n, 1e4, seed=200 + n)
    w, C = vbcore.generalized_eigh(ctx, H, S)
    wr, Cr = O.generalized_eigh(H, S)
    scale = np.abs(wr).max()
    assert np.abs(w - wr).max() < 1e-11 * scale
    assert np.all(np.diff(w) >= 0)
    # C^T S C = I and H C = S C diag(w)
    assert np.abs(C.T @ S @ C - np.eye(n)).max() < 1e-10
    assert np.abs(H @ C - S @ C * w).max() < 1e-10 * scale * max(1.0, np.abs(C).max())
    # lowest root's vector up to sign
    c0, r0 = C[:, 0], Cr[:, 0]
    assert min(np.abs(c0 - r0).max(), np.abs(c0 + r0).max()) < 1e-8 * np.abs(r0).max()


def test_generalized_eigh_uses_upper_triangles(ctx):
    n = 50
    H = _random_symmetric(n, 1)
    S = O.conditioned_metric(n, 1e3, seed=2)
    junk = np.tril(np.full((n, n), 3.0), -1)
    w, _ = vbcore.generalized_eigh(ctx, np.triu(H) + junk, np.triu(S) + junk)
    assert np.abs(w - O.generalized_eigh(H, S)[0]).max() < 1e-11 * np.abs(w).max()


def test_generalized_eigh_rejects_indefinite_overlap(ctx):
    n = 20
    H = _random_symmetric(n, 5)
    S = O.conditioned_metric(n, 1e2, seed=6)
    S[7, 7] = -2.0
    with pytest.raises(vbcore.VbError) as e:
        vbcore.generalized_eigh(ctx, H, S)
    assert e.value.status == 4 and e.value.info == n + 8
    assert "not positive definite" in str(e.value)


def test_degenerate_spectrum(ctx):
    # repeated eigenvalues: the eigenvalues must still match and C must stay S-orthonormal
    n = 60
    rng = np.random.default_rng(9)
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    d = np.repeat(np.arange(12, dtype=np.float64), 5)
    A = (q * d) @ q.T
    S = O.conditioned_metric(n, 1e2, seed=10)
    Ls = np.linalg.cholesky(S)
    H = Ls @ A @ Ls.T
    H = 0.5 * (H + H.T)
    w, C = vbcore.generalized_eigh(ctx, H, S)
    assert np.abs(w - np.sort(d)).max() < 1e-11 * 12
    assert np.abs(C.T @ S @ C - np.eye(n)).max() < 1e-10


def test_structure_energy_matches_oracle(ctx):
    # lowest root of the structure problem (the VBSCF energy without core and nuclear terms)
    n = 10
    S, h, eri = workloads.active_space(n, 3 * n, 77)
    rows = vbcore.generate_structures("COV", n, n)
    ex = vbcore.expand_structures(rows, n)
    plan = vbcore.HsPlan(ctx, ex, n)
    Hs, Ss = plan.execute(S, h, eri)
    w, C = vbcore.generalized_eigh(ctx, Hs, Ss)
    ex_o = O.expand(O.generate_structures("COV", n, n), n)
    Hr, Sr, _ = O.structure_matrices(n, ex_o, S, h, eri)
    wr, _ = O.generalized_eigh(Hr, Sr)
    assert abs(w[0] - wr[0]) < 1e-9
    plan.close()


def test_batched_matches_single(ctx):
    problems = []
    for i, n in enumerate([1, 2, 5, 14, 42, 60, 33]):
        problems.append((_random_symmetric(n, 300 + i), O.conditioned_metric(n, 1e3, seed=400 + i)))
    out = vbcore.generalized_eigh_batched(ctx, problems)
    for (H, S), (w, C) in zip(problems, out):
        wr, _ = O.generalized_eigh(H, S)
        assert np.abs(w - wr).max() < 1e-11 * np.abs(wr).max()
        assert np.abs(C.T @ S @ C - np.eye(len(w))).max() < 1e-10


@pytest.mark.parametrize("kw,n", [("COV", 8), ("COV ION(1)", 8), ("COV ION(1)", 10)])
def test_lowest_root_matches_dsygvd_on_structure_problems(ctx, kw, n):
    S, h, eri = workloads.active_space(n, 3 * n, 300 + n)
    rows = vbcore.generate_structures(kw, n, n)
    ex = vbcore.expand_structures(rows, n)
    plan = vbcore.HsPlan(ctx, ex, n)
    Hs, Ss = plan.execute(S, h, eri)
    E, c, its = vbcore.lowest_root(ctx, Hs, Ss, tolerance=1e-11)
    wr, Cr = O.generalized_eigh(Hs, Ss)
    assert abs(E - wr[0]) < 1e-9 * max(1.0, abs(wr[0]))
    assert abs(c @ Ss @ c - 1.0) < 1e-10
    r0 = Cr[:, 0]
    assert min(np.abs(c - r0).max(), np.abs(c + r0).max()) < 1e-6 * np.abs(r0).max()
    plan.close()


def test_lowest_root_random(ctx):
    n = 700
    H = _random_symmetric(n, 12)
    S = O.conditioned_metric(n, 1e3, seed=13)
    E, c, its = vbcore.lowest_root(ctx, H, S, tolerance=1e-11, max_iterations=3000)
    assert abs(E - O.generalized_eigh(H, S)[0][0]) < 1e-9 * max(1.0, abs(E))


def test_grid_barrier_timeout_is_reported_and_the_context_stays_usable():
    """The cooperative solver's grid barrier gives up after a bounded number of polls: with a
    one-poll limit the waits run out, the kernel ends and the call returns VB_ERR_TIMEOUT (no
    trap, no hang); after the default limit is restored the same context solves the problem.
    The blocked Cholesky above the one-CTA size has no grid barrier: the limit does not touch it."""
    c = vbcore.Context(0)
    try:
        n = 200  # above the one-CTA size: a grid-wide cooperative launch with a grid barrier
        H = _random_symmetric(n, 7)
        S = O.conditioned_metric(n, 1e3, seed=8)
        c.set_barrier_spin_limit(1)
        with pytest.raises(vbcore.VbError) as e:
            vbcore.generalized_eigh(c, H, S)
        assert e.value.status == 6 and "grid barrier timed out" in str(e.value)
        U = vbcore.metric_cholesky(c, S)
        assert np.abs(U - O.metric_cholesky(S)).max() < 1e-12
        c.set_barrier_spin_limit(0)
        w, _ = vbcore.generalized_eigh(c, H, S)
        wr, _ = O.generalized_eigh(H, S)
        assert np.abs(w - wr).max() < 1e-11 * np.abs(wr).max()
        with pytest.raises(vbcore.VbError):
            c.set_barrier_spin_limit(-1)
    finally:
        c.close()


@pytest.mark.parametrize("n", [98, 112, 127, 128, 129, 144, 191, 192, 193, 257, 320, 705])
def test_blocked_cholesky_panel_edges(ctx, n):
    """Sizes at and around the 64-column panels and the 16-column blocks inside them (one, two,
    three and more panels: the look-ahead chain's first links)."""
    S = O.conditioned_metric(n, 1e4, seed=n)
    U = vbcore.metric_cholesky(ctx, S)
    assert np.array_equal(U, np.triu(U))
    assert np.linalg.norm(U.T @ U - S) / np.linalg.norm(S) < 4e-15 * n ** 0.5


@pytest.mark.parametrize("bad", [1, 16, 17, 33, 64, 65, 80, 128, 129, 200])
def test_blocked_cholesky_failing_minor_at_block_edges(ctx, bad):
    n = 200
    S = O.conditioned_metric(n, 1e2, seed=bad)
    S[bad - 1, bad - 1] = -1.0
    with pytest.raises(vbcore.VbError) as e:
        vbcore.metric_cholesky(ctx, S)
    assert e.value.status == 4 and e.value.info == bad


@pytest.mark.parametrize("n", [1, 2, 3, 7, 47, 48, 49, 63, 64, 65, 130, 300, 700])
def test_lowest_root_sizes(ctx, n):
    """Davidson at the edges of its 64-row tiles and of the 48-vector subspace: full subspaces
    (n <= 48), the thick restart and the shift-invert phase.  The eigenvalue of a vector with
    relative residual 1e-11 is off by less than 1e-11 cond(S) of the spectrum's scale."""
    H = _random_symmetric(n, 300 + n) + np.diag(np.linspace(-3.0, 8.0, n))
    S = O.conditioned_metric(n, 1e3, seed=400 + n)
    e, c, its = vbcore.lowest_root(ctx, H, S, tolerance=1e-11)
    wr, _ = O.generalized_eigh(H, S)
    assert abs(e - wr[0]) < 1e-8 * np.abs(wr).max()
    assert abs(c @ S @ c - 1.0) < 1e-9
    r = H @ c - e * (S @ c)
    assert np.linalg.norm(r) < 1e-10 * (np.linalg.norm(H @ c) + abs(e) * np.linalg.norm(S @ c))


@pytest.mark.parametrize("n", [33, 34, 47, 64, 95, 96, 127, 128, 129, 159, 160])
@pytest.mark.parametrize("spectrum", ["random", "close", "degenerate", "diagonal", "zero"])
def test_tridiagonal_eigh_sizes_and_clusters(ctx, n, spectrum):
    """The tridiagonal path (33 <= n <= 160) at the edges of its tiles, for spread, nearly equal
    (1e-9 apart) and equal roots, a matrix that is already diagonal, and H = 0.  Backward-stable
    bounds: residual and S-orthonormality of order n eps cond(S)^(1/2), below 1e-10 here."""
    rng = np.random.default_rng(n)
    S = O.conditioned_metric(n, 1e3, seed=n)
    if spectrum == "random":
        H = _random_symmetric(n, n + 1)
    elif spectrum == "diagonal":
        S, H = np.eye(n), np.diag(rng.permutation(np.arange(n, dtype=np.float64)))
    elif spectrum == "zero":
        H = np.zeros((n, n))
    else:
        q, _ = np.linalg.qr(rng.standard_normal((n, n)))
        d = np.repeat(np.arange((n + 4) // 5, dtype=np.float64), 5)[:n]
        if spectrum == "close":
            d = d + 1e-9 * np.arange(n)
        L = np.linalg.cholesky(S)
        H = L @ ((q * d) @ q.T) @ L.T
        H = 0.5 * (H + H.T)
    w, C = vbcore.generalized_eigh(ctx, H, S)
    wr, _ = O.generalized_eigh(H, S)
    scale = max(np.abs(wr).max(), 1e-3)
    assert np.abs(w - wr).max() < 1e-11 * scale
    assert np.all(np.diff(w) >= 0)
    assert np.abs(C.T @ S @ C - np.eye(n)).max() < 1e-10
    assert np.abs(H @ C - S @ C * w).max() < 1e-10 * scale * max(1.0, np.abs(C).max())


def test_tridiagonal_eigh_beside_other_solves(ctx):
    """The reduction's four CTAs exchange sums through each other's shared memory: solves of several threads
    with contexts of their own, all at once, give the bits of a solve alone."""
    import threading

    n, workers = 150, 6
    problems = [(_random_symmetric(n, 900 + i), O.conditioned_metric(n, 1e3, seed=950 + i)) for i in range(workers)]
    alone = [vbcore.generalized_eigh(ctx, H, S) for H, S in problems]
    wrong = []

    def work(i):
        own = vbcore.Context(0)
        try:
            for _ in range(10):
                w, C = vbcore.generalized_eigh(own, *problems[i])
                if not (np.array_equal(w, alone[i][0]) and np.array_equal(C, alone[i][1])):
                    wrong.append(i)
        except Exception as e:  # reported below: an exception in a thread does not fail the test
            wrong.append((i, e))
        finally:
            own.close()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(workers)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


@pytest.mark.parametrize("n", [33, 100, 160])
@pytest.mark.parametrize("power", [-1000, -700, -520, 500, 600])
def test_tridiagonal_eigh_at_any_scale(ctx, n, power):
    """H scaled by a power of two: the same vectors and scaled roots, to the bit (squares of the elements leave
    the range of the exponent from 2^-511 and 2^511 on)."""
    H = _random_symmetric(n, n)
    S = O.conditioned_metric(n, 1e3, seed=n)
    w, C = vbcore.generalized_eigh(ctx, H, S)
    w2, C2 = vbcore.generalized_eigh(ctx, np.ldexp(H, power), S)
    assert np.array_equal(w2, np.ldexp(w, power)) and np.array_equal(C, C2)


def test_problems_the_tridiagonal_path_does_not_settle(ctx):
    """33 <= n <= 160 take a path without a grid barrier; what it does not settle (here a NaN in H) goes on to the
    block Jacobi, whose barrier gives up under a limit of one poll.  Vectors may lie over H: they are not
    written before everything is settled, so that Jacobi finds H as it was."""
    import ctypes

    import torch

    n = 120
    c = vbcore.Context(0)
    lib = vbcore.load_library()
    try:
        c.set_barrier_spin_limit(1)
        H = _random_symmetric(n, 3)
        S = O.conditioned_metric(n, 1e3, seed=4)
        wr, Cr = vbcore.generalized_eigh(c, H, S)
        for spoilt in (False, True):
            Hd = torch.tensor(H, device="cuda")
            if spoilt:
                Hd[5, 3] = Hd[3, 5] = float("nan")
            before = Hd.cpu().numpy().copy()
            Sd, w = torch.tensor(S, device="cuda"), torch.empty(n, dtype=torch.float64, device="cuda")
            info = ctypes.c_int(0)
            torch.cuda.synchronize()
            st = lib.vb_generalized_eigh(c.handle, *(ctypes.c_void_p(t.data_ptr()) for t in (Hd, Sd)), n,
                                         vbcore.VB_MEM_DEVICE, ctypes.c_void_p(w.data_ptr()),
                                         ctypes.c_void_p(Hd.data_ptr()), ctypes.byref(info))
            if spoilt:
                assert st == 6 and np.array_equal(Hd.cpu().numpy(), before, equal_nan=True)
            else:
                assert st == 0 and np.array_equal(w.cpu().numpy(), wr)
                assert np.array_equal(Hd.cpu().numpy().T, Cr)
    finally:
        c.close()
