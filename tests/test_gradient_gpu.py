"""Analytic structure-root gradient on the device against central differences of the oracle's
energy (the reference verifies its gradients the same way: tests/cuda/test_structure_action.cpp
:267-294).  E(S, h, eri) = lowest root of the oracle structure H/S (dsygvd)."""

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


def _energy(n, ex_o, S, h, eri):
    Hs, Ss, _ = O.structure_matrices(n, ex_o, S, h, eri)
    w, _ = O.generalized_eigh(Hs, Ss)
    return w[0]


def _richardson(f, step):
    d1 = (f(step) - f(-step)) / (2 * step)
    d2 = (f(step / 2) - f(-step / 2)) / step
    return (4 * d2 - d1) / 3


def _sym(rng, n):
    a = rng.standard_normal((n, n))
    return 0.5 * (a + a.T)


def _full_rank_eri(n, seed):
    rng = np.random.default_rng(seed)
    P = n * (n + 1) // 2
    M = rng.standard_normal((P, P)) * 0.05
    K = M @ M.T + 0.01 * np.eye(P)
    return workloads.pack_pair_kernel(K)


def _setup(ctx, kw, n, nel, mult, S, h, eri):
    rows = vbcore.generate_structures(kw, n, nel, mult)
    ex = vbcore.expand_structures(rows, nel, mult)
    plan = vbcore.HsPlan(ctx, ex, n)
    ex_o = O.expand(O.generate_structures(kw, n, nel, mult), nel, mult)
    Hs, Ss = plan.execute(S, h, eri)
    w, C = vbcore.generalized_eigh(ctx, Hs, Ss)
    return plan, ex_o, w[0], C[:, 0]


@pytest.mark.parametrize("kw,n,nel,mult", [("COV", 4, 4, 1), ("COV", 6, 6, 1), ("COV ION(1)", 5, 6, 1),
                                           ("COV", 5, 5, 2), ("COV", 6, 4, 3), ("COV ION(1)", 6, 6, 1)])
def test_gradient_matches_differences(ctx, kw, n, nel, mult):
    S, h, _ = workloads.active_space(n, 3 * n, 50 + n + nel)
    eri = _full_rank_eri(n, 60 + n)
    plan, ex_o, lam, c = _setup(ctx, kw, n, nel, mult, S, h, eri)
    g = plan.gradient(S, h, eri, c, lam)
    assert np.allclose(g["S"], g["S"].T) and np.allclose(g["h"], g["h"].T)
    rng = np.random.default_rng(7)
    dS, dh = _sym(rng, n), _sym(rng, n)
    de = rng.standard_normal(eri.size)
    for name, direction, analytic in (
            ("S", lambda t: _energy(n, ex_o, S + t * dS, h, eri), np.sum(g["S"] * dS)),
            ("h", lambda t: _energy(n, ex_o, S, h + t * dh, eri), np.sum(g["h"] * dh)),
            ("eri", lambda t: _energy(n, ex_o, S, h, eri + t * de), np.dot(g["eri"], de))):
        fd = _richardson(direction, 1e-3)
        assert abs(fd - analytic) < 1e-7 * max(1.0, abs(fd)), (name, fd, analytic)
    # single entries, both triangles at once
    for (i, j) in ((0, 0), (0, n - 1), (1, 2)):
        E = np.zeros((n, n))
        E[i, j] = E[j, i] = 1.0
        fd = _richardson(lambda t: _energy(n, ex_o, S + t * E, h, eri), 1e-3)
        assert abs(fd - np.sum(g["S"] * E)) < 1e-7 * max(1.0, abs(fd))
    plan.close()


def test_gradient_with_ri_factors(ctx):
    n, n_aux = 6, 8
    rng = np.random.default_rng(3)
    S, h, _ = workloads.active_space(n, 3 * n, 4)
    P = n * (n + 1) // 2
    F = 0.2 * rng.standard_normal((P, n_aux))
    eri = workloads.pack_pair_kernel(F @ F.T)
    plan, ex_o, lam, c = _setup(ctx, "COV", n, n, 1, S, h, eri)
    with pytest.raises(vbcore.VbError) as e:
        plan.gradient(S, h, eri, c, lam)
    assert e.value.status == 5
    g = plan.gradient(S, h, eri, c, lam, packed_eri=False, ri_factors=F)
    dF = rng.standard_normal(F.shape)
    fd = _richardson(lambda t: _energy(n, ex_o, S, h, workloads.pack_pair_kernel((F + t * dF) @ (F + t * dF).T)),
                     1e-3)
    assert abs(fd - np.sum(g["ri"] * dF)) < 1e-7 * max(1.0, abs(fd))
    plan.close()


def test_gradient_exact_path_orthogonal_orbitals(ctx):
    # S = I: every spin-pair block is a permutation-like 0/1 matrix (nullities 1, 2, ...):
    # the exact-path backward handles all of them
    n = 6
    _, h, _ = workloads.active_space(n, 3 * n, 9)
    S = np.eye(n)
    eri = _full_rank_eri(n, 10)
    plan, ex_o, lam, c = _setup(ctx, "COV", n, n, 1, S, h, eri)
    g = plan.gradient(S, h, eri, c, lam)
    # the energy curves sharply away from S = I: small steps, entry by entry
    for (i, j) in ((0, 0), (1, 1), (0, 1), (0, 2), (2, 5), (4, 5)):
        E = np.zeros((n, n))
        E[i, j] = E[j, i] = 1.0
        fd = _richardson(lambda t: _energy(n, ex_o, S + t * E, h, eri), 1e-4)
        assert abs(fd - np.sum(g["S"] * E)) < 1e-7 * max(1.0, abs(fd)), (i, j)
    assert plan.stats()["careful_spin_pairs"] > 0
    plan.close()


def test_gradient_exact_path_graded_overlaps(ctx):
    # stretched-chain overlaps S_ij = +-exp(-3 |i - j|^2) (0.05, 6e-6, 1e-12, ...): most blocks
    # fail the conditioning certificate and many are rank deficient under the reference
    # semantics (nullity 1..3), which the singular-value-frame adjoint handles
    n = 8
    _, h, _ = workloads.active_space(n, 3 * n, 11)
    dist = np.abs(np.subtract.outer(np.arange(n), np.arange(n)))
    sign = np.sign(_sym(np.random.default_rng(12), n))
    sign = np.triu(sign, 1) + np.triu(sign, 1).T + np.eye(n)
    S = np.exp(-3.0 * dist ** 2) * sign
    eri = _full_rank_eri(n, 13)
    plan, ex_o, lam, c = _setup(ctx, "COV", n, n, 1, S, h, eri)
    g = plan.gradient(S, h, eri, c, lam)
    for (i, j) in ((0, 1), (2, 2), (1, 4), (0, 7)):
        E = np.zeros((n, n))
        E[i, j] = E[j, i] = 1.0
        fd = _richardson(lambda t: _energy(n, ex_o, S + t * E, h, eri), 1e-4)
        assert abs(fd - np.sum(g["S"] * E)) < 1e-7 * max(1.0, abs(fd)), (i, j, fd, np.sum(g["S"] * E))
    assert plan.stats()["careful_spin_pairs"] > plan.stats()["spin_pairs"] // 4
    plan.close()


@pytest.mark.parametrize("kw,n,seed", [("COV", 6, 21), ("COV ION(1)", 8, 22)])
def test_root_gradient_matches_separate_steps(ctx, kw, n, seed):
    # one call with H and S device-resident (dense solver for 5 structures, Davidson for 294)
    # against execute -> eigensolver -> gradient through host buffers
    _, h, _ = workloads.active_space(n, 3 * n, seed)
    S, _, _ = workloads.active_space(n, 3 * n, seed + 1)
    rng = np.random.default_rng(seed)
    F = 0.1 * rng.standard_normal((n * (n + 1) // 2, 3 * n))
    eri = workloads.pack_pair_kernel(F @ F.T)
    ex = vbcore.expand_structures(vbcore.generate_structures(kw, n, n), n)
    plan = vbcore.HsPlan(ctx, ex, n)
    E, c, g = plan.root_gradient(S, h, eri, ri_factors=F)
    Hs, Ss = plan.execute(S, h, eri)
    if Hs.shape[0] <= 200:
        w, C = vbcore.generalized_eigh(ctx, Hs, Ss)
        lam, cr = w[0], C[:, 0]
    else:
        lam, cr, _ = vbcore.lowest_root(ctx, Hs, Ss, tolerance=1e-11, max_iterations=2000)
    gr = plan.gradient(S, h, eri, cr, lam, packed_eri=False, ri_factors=F)
    assert abs(E - lam) < 1e-10 * max(1.0, abs(lam))
    assert abs(abs(c @ Ss @ cr) - 1.0) < 1e-8
    for key in ("S", "h", "ri"):
        assert np.abs(g[key] - gr[key]).max() < 1e-8 * max(1.0, np.abs(gr[key]).max()), key
    plan.close()


def _graded_overlap(n, rate, power, seed):
    dist = np.abs(np.subtract.outer(np.arange(n), np.arange(n))).astype(float)
    sign = np.sign(_sym(np.random.default_rng(seed), n))
    return np.exp(-rate * dist ** power) * (np.triu(sign, 1) + np.triu(sign, 1).T + np.eye(n))


@pytest.mark.parametrize("kw,n,nel,mult", [("COV", 4, 2, 1), ("COV ION(1)", 5, 4, 1), ("COV", 7, 7, 2), ("COV", 8, 8, 3),
                                           ("COV ION(1)", 8, 8, 1), ("COV", 10, 10, 1), ("COV", 11, 11, 4),
                                           ("COV", 12, 12, 1), ("COV", 13, 13, 2)])
@pytest.mark.parametrize("overlap", ["random", "chain", "orthogonal"])
def test_frame_gradient_matches_pair_by_pair(ctx, kw, n, nel, mult, overlap):
    """The gradient in the left strings' frames (the path without packed integrals) against the
    pair-by-pair kernels (the path with them) for 1 .. 7 electrons per string, equal and unequal
    string tables, all excitation levels, well conditioned and exactly singular blocks.  Both are
    exact derivatives; the pair-by-pair form subtracts terms of size G / |X| (inverse of a block of
    norm |X|), which leaves eps G / |X|: below 1e-11 for these overlaps (|X| > 1e-4 or X = 0), but
    up to 1e-4 for graded ones, which the next test takes against differences."""
    rng = np.random.default_rng(100 * n + nel)
    S = {"random": lambda: workloads.active_space(n, 3 * n, 70 + n)[0],
         "chain": lambda: np.exp(-0.8 * np.abs(np.subtract.outer(np.arange(n), np.arange(n)))),
         "orthogonal": lambda: np.eye(n)}[overlap]()
    h = _sym(rng, n)
    P = n * (n + 1) // 2
    F = 0.05 * rng.standard_normal((P, P)) + 0.1 * np.eye(P)
    eri = workloads.pack_pair_kernel(F @ F.T)
    rows = vbcore.generate_structures(kw, n, nel, mult)
    plan = vbcore.HsPlan(ctx, vbcore.expand_structures(rows, nel, mult), n)
    c = rng.standard_normal(plan.n_structures)
    c /= np.linalg.norm(c)
    a = plan.gradient(S, h, eri, c, -1.3, packed_eri=False, ri_factors=F)
    b = plan.gradient(S, h, eri, c, -1.3, packed_eri=True, ri_factors=F)
    for key in ("S", "h", "ri"):
        assert np.abs(a[key] - b[key]).max() < 1e-8 * max(1e-3, np.abs(b[key]).max()), key
    plan.close()


@pytest.mark.parametrize("kw,n,nel,mult", [("COV", 4, 2, 1), ("COV", 8, 8, 1), ("COV", 7, 7, 2), ("COV ION(1)", 6, 6, 1)])
def test_frame_gradient_graded_overlaps(ctx, kw, n, nel, mult):
    """Overlaps S_ij = +-exp(-3 |i - j|^2) (0.05, 6e-6, 2e-12, ...): most blocks are outside the
    conditioning certificate or rank deficient under the reference semantics.  Against Richardson
    differences of the oracle's energy (step 1e-4, error of order 1e-9)."""
    S = _graded_overlap(n, 3.0, 2, n)
    rng = np.random.default_rng(31 * n)
    h = _sym(rng, n)
    P = n * (n + 1) // 2
    F = 0.05 * rng.standard_normal((P, P)) + 0.1 * np.eye(P)
    eri = workloads.pack_pair_kernel(F @ F.T)
    plan, ex_o, lam, c = _setup(ctx, kw, n, nel, mult, S, h, eri)
    g = plan.gradient(S, h, eri, c, lam, packed_eri=False, ri_factors=F)
    for (i, j) in ((0, 1), (2, 2), (1, 3), (0, n - 1)):
        E = np.zeros((n, n))
        E[i, j] = E[j, i] = 1.0
        fd = _richardson(lambda t: _energy(n, ex_o, S + t * E, h, eri), 1e-4)
        assert abs(fd - np.sum(g["S"] * E)) < 1e-7 * max(1.0, abs(fd)), (i, j, fd, np.sum(g["S"] * E))
    dF = rng.standard_normal(F.shape)
    fd = _richardson(lambda t: _energy(n, ex_o, S, h, workloads.pack_pair_kernel((F + t * dF) @ (F + t * dF).T)), 1e-4)
    assert abs(fd - np.sum(g["ri"] * dF)) < 1e-7 * max(1.0, abs(fd))
    plan.close()


@pytest.mark.parametrize("kw,n,mult", [("COV", 12, 1), ("COV ION(1)", 7, 2), ("COV", 14, 1)])
def test_frame_gradient_from_records_and_high_levels(ctx, kw, n, mult):
    """Covalent singlets (one determinant per alpha string: adjoints read from the partners' records)
    and lists without that property, with strings of 6 and 7 electrons whose pairs reach levels 6 and 7
    through the inverse, or through the listed kernel where the overlaps are zero for one orbital.
    Same comparison and bound as above."""
    rng = np.random.default_rng(n)
    S = workloads.active_space(n, 3 * n, 7 + n)[0]
    S[0, 1:] = S[1:, 0] = 0.0
    h = _sym(rng, n)
    P = n * (n + 1) // 2
    F = 0.05 * rng.standard_normal((P, P)) + 0.1 * np.eye(P)
    eri = workloads.pack_pair_kernel(F @ F.T)
    plan = vbcore.HsPlan(ctx, vbcore.expand_structures(vbcore.generate_structures(kw, n, n, mult), n, mult), n)
    c = rng.standard_normal(plan.n_structures)
    c /= np.linalg.norm(c)
    a = plan.gradient(S, h, eri, c, -0.7, packed_eri=False, ri_factors=F)
    b = plan.gradient(S, h, eri, c, -0.7, packed_eri=True, ri_factors=F)
    for key in ("S", "h", "ri"):
        assert np.abs(a[key] - b[key]).max() < 1e-8 * max(1e-3, np.abs(b[key]).max()), key
    plan.close()


def _nearly_dependent(n, separation, seed):
    """Overlaps of orbitals close to orthogonal, but for the second one: the first one plus `separation` times
    another."""
    rng = np.random.default_rng(seed)
    C = np.eye(n) + 0.05 * rng.standard_normal((n, n))
    C[:, 1] = C[:, 0] + separation * C[:, 1]
    S = C.T @ C
    d = 1.0 / np.sqrt(np.diag(S))
    return d[:, None] * S * d[None, :]


@pytest.mark.parametrize("kw,n,nel,mult", [("COV", 6, 6, 1), ("COV ION(1)", 6, 6, 1), ("COV", 7, 7, 2), ("COV", 8, 8, 1)])
@pytest.mark.parametrize("separation", [0.3, 0.1, 0.03, 0.01, 3e-3, 1e-3])
def test_gradient_of_nearly_dependent_orbitals(ctx, kw, n, nel, mult, separation):
    """Two nearly dependent orbitals: strings that hold both have an ill-conditioned S_LL (kappa up to 4e6).
    Against every block inverted by itself in extended precision.  Bound: the inputs themselves are known to
    kappa eps of the gradient, four times that; 5e-14 for pairs that take their own inverse
    (kappa(X)^2 < 1e6, kappa^2 eps / 500 of it).  The frame of such a string would leave kappa^2 eps / 50 and more."""
    S = _nearly_dependent(n, separation, n)
    rng = np.random.default_rng(n)
    h = _sym(rng, n)
    P = n * (n + 1) // 2
    F = 0.05 * rng.standard_normal((P, P)) + 0.1 * np.eye(P)
    eri = workloads.pack_pair_kernel(F @ F.T)
    plan = vbcore.HsPlan(ctx, vbcore.expand_structures(vbcore.generate_structures(kw, n, nel, mult), nel, mult), n)
    ex = O.expand(O.generate_structures(kw, n, nel, mult), nel, mult)
    c = rng.standard_normal(plan.n_structures)
    c /= np.linalg.norm(c)
    ref = O.functional_gradient(n, ex, S, h, F, c, -1.3)
    kappa2 = 1.0
    for strings in (ex.alpha_strings, ex.beta_strings):
        occ = np.array([[i for i in range(n) if (s >> i) & 1] for s in strings])
        X = S[occ[:, :, None], occ[:, None, :]]
        kappa2 = max(kappa2, (np.linalg.norm(X, axis=(1, 2)) * np.linalg.norm(np.linalg.inv(X), axis=(1, 2))).max() ** 2)
    got = plan.gradient(S, h, eri, c, -1.3, packed_eri=False, ri_factors=F)
    for key in ("S", "h", "ri"):
        err = float(np.abs(got[key] - ref[key]).max() / np.abs(ref[key]).max())
        assert err < 5e-14 + 4 * 2.2e-16 * kappa2 ** 0.5, (key, kappa2, err)
    plan.close()


@pytest.mark.parametrize("kw,n,nel,mult", [("COV", 4, 4, 1), ("COV", 5, 5, 2), ("COV ION(1)", 5, 4, 1)])
@pytest.mark.parametrize("rate", [1.0, 3.0])
@pytest.mark.parametrize("separation", [1.0, 0.1, 0.01])
def test_gradient_of_graded_and_nearly_dependent_orbitals(ctx, kw, n, nel, mult, rate, separation):
    """Overlaps exp(-rate |i - j|^2) (down to 1e-33), the second orbital close to the first one: blocks that are
    tiny, ill conditioned or both, of strings in and outside the frame form.  Against blocks inverted one by one
    with 100 digits; same bound (a block's own inverse up to the forward value's certificate would leave
    2e-8)."""
    dist = np.abs(np.subtract.outer(np.arange(n), np.arange(n))).astype(float)
    C = np.eye(n)
    C[:, 1] = (C[:, 0] if separation < 1.0 else 0.0) + separation * C[:, 1]
    S = C.T @ np.exp(-rate * dist ** 2) @ C
    d = 1.0 / np.sqrt(np.diag(S))
    S = d[:, None] * S * d[None, :]
    S = 0.5 * (S + S.T)
    rng = np.random.default_rng(n)
    h = _sym(rng, n)
    P = n * (n + 1) // 2
    F = 0.05 * rng.standard_normal((P, P)) + 0.1 * np.eye(P)
    eri = workloads.pack_pair_kernel(F @ F.T)
    plan = vbcore.HsPlan(ctx, vbcore.expand_structures(vbcore.generate_structures(kw, n, nel, mult), nel, mult), n)
    ex = O.expand(O.generate_structures(kw, n, nel, mult), nel, mult)
    c = rng.standard_normal(plan.n_structures)
    c /= np.linalg.norm(c)
    ref = O.functional_gradient(n, ex, S, h, F, c, -1.3, digits=100)
    got = plan.gradient(S, h, eri, c, -1.3, packed_eri=False, ri_factors=F)
    kappa = np.linalg.cond(S)
    for key in ("S", "h", "ri"):
        err = np.abs(got[key] - ref[key]).max() / np.abs(ref[key]).max()
        assert err < 5e-14 + 4 * 2.2e-16 * kappa, (key, kappa, err)
    plan.close()


@pytest.mark.parametrize("n,mult,budget_mb", [(10, 1, 50), (10, 3, 70)])
def test_gradient_of_nearly_dependent_orbitals_in_a_small_budget(n, mult, budget_mb):
    """The pair-by-pair form of the ill-conditioned strings in as many chunks as the budget leaves room for
    (70 and 100 MB hold one)."""
    kw, nel = "COV", n
    S = _nearly_dependent(n, 0.03, n)
    rng = np.random.default_rng(n)
    h = _sym(rng, n)
    P = n * (n + 1) // 2
    F = 0.05 * rng.standard_normal((P, P)) + 0.1 * np.eye(P)
    eri = workloads.pack_pair_kernel(F @ F.T)
    ex = vbcore.expand_structures(vbcore.generate_structures(kw, n, nel, mult), nel, mult)
    c = rng.standard_normal(ex.n_structures)
    c /= np.linalg.norm(c)
    got = []
    for budget in (0, budget_mb << 20):
        own = vbcore.Context(0, budget) if budget else vbcore.Context(0)
        try:
            plan = vbcore.HsPlan(own, ex, n)
            got.append(plan.gradient(S, h, eri, c, -1.3, packed_eri=False, ri_factors=F))
            plan.close()
        finally:
            own.close()
    # the sums over pairs are atomic: their order differs
    for key in ("S", "h", "ri"):
        assert np.abs(got[0][key] - got[1][key]).max() < 1e-10 * np.abs(got[0][key]).max(), key
