"""The calls whose speed is measured, and what they compute.

Each case is one kind of call that a valence-bond program makes of vbcore, with sizes from the
benchmark's workloads and the tests:

* ``hs``: structure Hamiltonian and overlap of one orbital point (``HsPlan.execute_device``), the
  inner call of every VBSCF step.  Covalent classes from the 5 structures of six electrons to the
  429 of fourteen, and open shells (triplets, doublets), where alpha and beta strings differ.
* ``root``: lowest root and its gradient with respect to S, h and the pair factors
  (``HsPlan.root_gradient``), host arrays in and out: one optimizer step of an active-space
  program, with covalent and singly ionic structures.
* ``scf``: one VBSCF energy and orbital gradient of a hydrogen chain (``ScfProblem.energy_gradient``),
  near equilibrium (latency of a small problem) and stretched (most overlap blocks singular).
* ``ri``: the RI transform of AO pair factors to the active space on device pointers, FP64 with
  the adjoint (an optimizer step's forward and backward) or split precision (early iterations).
* ``cholesky``: factor of a structure or orbital metric; ``eigh``: all roots of a structure problem.
* ``engine``: a batch of small instances of mixed sizes, energies and gradients in one call.
"""

from __future__ import annotations

import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "xmvb-cpp_b200"))
import vbcore  # noqa: E402
from vbcore import molecules, workloads  # noqa: E402

F64 = torch.float64


def listed():
    return [
        # the plain six-orbital solve's inner call: every kernel at its smallest, launches count
        {"name": "hs_cov_6", "kind": "hs", "n": 6, "electrons": 6, "multiplicity": 1, "structures": "COV"},
        # an open shell: two string tables of different electron counts
        {"name": "hs_cov_12_triplet", "kind": "hs", "n": 12, "electrons": 12, "multiplicity": 3, "structures": "COV"},
        # the headline size: 429 structures over 3432 determinants
        {"name": "hs_cov_14", "kind": "hs", "n": 14, "electrons": 14, "multiplicity": 1, "structures": "COV"},
        # an ordinary covalent + ionic instance (294 structures) through host arrays
        {"name": "root_ion_8", "kind": "root", "n": 8, "electrons": 8, "multiplicity": 1, "structures": "COV ION(1)"},
        # the largest batched instance: 5676 structures over 34,188 determinants
        {"name": "root_ion_12", "kind": "root", "n": 12, "electrons": 12, "multiplicity": 1, "structures": "COV ION(1)"},
        # one evaluation of the plain solve: 5 structures, all latency
        {"name": "scf_h6", "kind": "scf", "atoms": 6, "spacing": 1.0},
        # a dissociating chain: singular overlap blocks, the exact path
        {"name": "scf_h14_stretched", "kind": "scf", "atoms": 14, "spacing": 3.0},
        # optimizer step of a large basis: forward with one-index factors, then the adjoint
        {"name": "ri_400_step", "kind": "ri", "n_bf": 400, "n_aux": 1600, "n_act": 16, "precision": "fp64", "adjoint": True},
        # early iterations in split precision
        {"name": "ri_400_bf16x3", "kind": "ri", "n_bf": 400, "n_aux": 1600, "n_act": 16, "precision": "bf16x3", "adjoint": False},
        # factor of a large structure metric
        {"name": "cholesky_2048", "kind": "cholesky", "n": 2048},
        # all roots of the 132 covalent structures of twelve electrons
        {"name": "eigh_132", "kind": "eigh", "n": 132},
        # an optimizer iteration over a mixed batch
        {"name": "engine_24", "kind": "engine", "count": 24, "sizes": "4,6,8,10"},
    ]


def draw(rng):
    kind = rng.choice(["hs", "hs", "root", "scf", "ri", "ri", "cholesky", "eigh", "engine"])
    if kind == "hs":
        n = rng.randint(4, 14)
        if n % 2:
            return {"kind": "hs", "n": n, "electrons": n, "multiplicity": 2, "structures": "COV"}
        return {"kind": "hs", "n": n, "electrons": n, "multiplicity": rng.choice([1, 3]), "structures": "COV"}
    if kind == "root":
        n = rng.randint(4, 12)
        return {"kind": "root", "n": n, "electrons": n, "multiplicity": 2 if n % 2 else 1,
                "structures": rng.choice(["COV", "COV ION(1)"])}
    if kind == "scf":
        return {"kind": "scf", "atoms": 2 * rng.randint(2, 7), "spacing": round(rng.uniform(0.7, 3.0), 3)}
    if kind == "ri":
        n_bf = int(round(math.exp(rng.uniform(math.log(24), math.log(440)))))
        return {"kind": "ri", "n_bf": n_bf, "n_aux": n_bf * rng.randint(3, 4) - rng.randint(0, 9),
                "n_act": rng.randint(4, 16), "precision": rng.choice(["fp64", "bf16x3"]), "adjoint": rng.random() < 0.5}
    if kind == "cholesky":
        return {"kind": "cholesky", "n": int(round(math.exp(rng.uniform(math.log(42), math.log(2500)))))}
    if kind == "eigh":
        return {"kind": "eigh", "n": int(round(math.exp(rng.uniform(math.log(5), math.log(200)))))}
    return {"kind": "engine", "count": rng.randint(4, 32), "sizes": rng.choice(["4,6,8", "6,8,10", "4,6,8,10", "8,10"])}


# ---- what a program has in hand -------------------------------------------------------------

_kept = {}


def _context():
    """One context for the process, on torch's default stream."""
    if "ctx" not in _kept:
        _kept["ctx"] = vbcore.Context(0)
        _kept["ctx"].set_stream(0)
    return _kept["ctx"]


def _expansion(case):
    """Structures and their determinant expansion: integer tables that depend on the class only."""
    key = (case["structures"], case["n"], case["electrons"], case["multiplicity"])
    if key not in _kept:
        rows = vbcore.generate_structures(*key)
        _kept[key] = vbcore.expand_structures(rows, case["electrons"], case["multiplicity"])
    return _kept[key]


def _active_space(n, seed):
    """S, h, packed (ij|kl) and the pair factors F [n(n+1)/2, 3n] behind it, of one instance."""
    S, h, _ = workloads.active_space(n, 3 * n, seed)
    rng = np.random.default_rng(seed + 7919)
    B = 0.1 * rng.standard_normal((3 * n, n, n))
    B = 0.5 * (B + B.transpose(0, 2, 1))
    rows, cols = np.tril_indices(n)
    F = np.ascontiguousarray(B[:, rows, cols].T)
    return S, h, workloads.pack_pair_kernel(F @ F.T), F


def _engine_instances(case, seed):
    rng = np.random.default_rng(seed)
    sizes = [int(s) for s in rng.permutation(np.resize([int(x) for x in case["sizes"].split(",")], case["count"]))]
    return sizes, [_active_space(n, seed + 1 + i) for i, n in enumerate(sizes)]


def _engine_class(n):
    return {"structures": "COV ION(1)", "n": n, "electrons": n, "multiplicity": 1}


def _chain(case, seed):
    mol = molecules.h_chain(case["atoms"], case["spacing"], 0.05, seed=seed % (1 << 31))
    pattern = molecules.hao_pattern(mol, case["atoms"])
    C = molecules.hao_guess(mol, pattern)
    rng = np.random.default_rng(seed)
    return mol, pattern, C * (1.0 + 0.05 * rng.standard_normal(C.shape))


def _ri_inputs(case, seed):
    """B (columns = AO pairs, auxiliary functions contiguous), C (row = active orbital), dL."""
    n_bf, n_aux, n_act = case["n_bf"], case["n_aux"], case["n_act"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    r, c = torch.tril_indices(n_bf, n_bf, device="cuda")
    B = torch.randn(r.numel(), n_aux, dtype=F64, device="cuda", generator=g)
    B *= torch.exp(-(r - c).double() / 20.0)[:, None]
    C = torch.randn(n_act, n_bf, dtype=F64, device="cuda", generator=g) / math.sqrt(n_bf)
    P = n_act * (n_act + 1) // 2
    dL = torch.randn(P, n_aux, dtype=F64, device="cuda", generator=g) if case["adjoint"] else None
    return B, C, dL


def _metric(n, decades, g):
    """Symmetric positive definite n x n with eigenvalues spread over `decades` below 1."""
    q, _ = torch.linalg.qr(torch.randn(n, n, dtype=F64, device="cuda", generator=g))
    S = (q * torch.logspace(0, -decades, n, dtype=F64, device="cuda")) @ q.T
    return 0.5 * (S + S.T)


def _metric_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = case["n"]
    if case["kind"] == "cholesky":
        return None, _metric(n, 4, g)
    H = torch.randn(n, n, dtype=F64, device="cuda", generator=g)
    return 0.5 * (H + H.T), _metric(n, 2, g)


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind in ("hs", "root"):
        st["plan"] = vbcore.HsPlan(_context(), _expansion(case), case["n"])
        S, h, eri, F = _active_space(case["n"], seed)
        if kind == "root":
            st["inputs"] = (S, h, eri, F)
        else:
            ns = st["plan"].n_structures
            st["inputs"] = [torch.tensor(x, device="cuda") for x in (S, h, eri)]  # S and h symmetric
            st["out"] = [torch.empty(ns, ns, dtype=F64, device="cuda") for _ in range(2)]
    elif kind == "scf":
        mol, pattern, st["C"] = _chain(case, seed)
        st["problem"] = vbcore.ScfProblem(_context(), mol, pattern, case["atoms"])
    elif kind == "ri":
        st["inputs"] = _ri_inputs(case, seed)
        n_bf, n_aux, n_act = case["n_bf"], case["n_aux"], case["n_act"]
        P = n_act * (n_act + 1) // 2
        shapes = [(n_bf, n_act, n_aux), (P, n_aux), (P * (P + 1) // 2,)] + ([(n_act, n_bf)] if case["adjoint"] else [])
        st["out"] = [torch.empty(s, dtype=F64, device="cuda") for s in shapes]
        _context()
    elif kind in ("cholesky", "eigh"):
        st["H"], st["S"] = _metric_inputs(case, seed)
        n = case["n"]
        st["w"] = torch.empty(n, dtype=F64, device="cuda")
        st["V"] = torch.empty(n, n, dtype=F64, device="cuda")
        st["phase"] = torch.randn(n, dtype=F64, generator=torch.Generator().manual_seed(1)).cuda()
        _context()
    else:
        sizes, data = _engine_instances(case, seed)
        st["engine"] = vbcore.Engine(0, 16 << 30, workers=8)
        st["ids"] = [st["engine"].add_instance(_expansion(_engine_class(n)), n) for n in sizes]
        st["inputs"] = [list(x) for x in zip(*data)]
    return st


# ---- one call ---------------------------------------------------------------------------------


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _ok(status):
    if status != 0:
        raise vbcore.VbError(status, vbcore.load_library().vb_last_error(_context().handle).decode())


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "hs":
        st["plan"].execute_device(*[t.data_ptr() for t in st["inputs"]], *[t.data_ptr() for t in st["out"]])
        return st["out"]
    if kind == "root":
        S, h, eri, F = st["inputs"]
        E, c, g = st["plan"].root_gradient(S, h, eri, ri_factors=F)
        return [np.array([E]), c * np.sign(c[np.argmax(np.abs(c))]), g["S"], g["h"], g["ri"]]
    if kind == "scf":
        E, g = st["problem"].energy_gradient(st["C"])
        return [np.array([E]), g]
    if kind == "engine":
        E, grads = st["engine"].evaluate(st["ids"], *st["inputs"])
        return [E] + [np.concatenate([g[k].ravel() for g in grads]) for k in ("S", "h", "ri")]
    lib, ctx = vbcore.load_library(), _context()
    if kind == "ri":
        B, C, dL = st["inputs"]
        T, L, K = st["out"][:3]
        n_aux, n_bf, n_act = case["n_aux"], case["n_bf"], case["n_act"]
        _ok(lib.vb_active_transform_ri_precision(ctx.handle, _p(B), n_aux, n_bf, _p(C), n_act,
                                                 vbcore.PRECISIONS[case["precision"]], vbcore.VB_MEM_DEVICE, _p(T),
                                                 _p(L), _p(K)))
        if case["adjoint"]:
            _ok(lib.vb_active_transform_ri_adjoint(ctx.handle, _p(T), _p(dL), n_aux, n_bf, n_act, vbcore.VB_MEM_DEVICE,
                                                   _p(st["out"][3])))
        return st["out"]
    info = ctypes.c_int(0)
    if kind == "cholesky":
        _ok(lib.vb_metric_cholesky(ctx.handle, _p(st["S"]), case["n"], vbcore.VB_MEM_DEVICE, _p(st["V"]),
                                   ctypes.byref(info)))
        return st["V"]  # row j = column j of U
    _ok(lib.vb_generalized_eigh(ctx.handle, _p(st["H"]), _p(st["S"]), case["n"], vbcore.VB_MEM_DEVICE, _p(st["w"]),
                                _p(st["V"]), ctypes.byref(info)))
    # row i = eigenvector i, with the phase convention of a program that compares two points
    return [st["w"], st["V"] * torch.sign(st["V"] @ st["phase"])[:, None]]


# ---- what a pass cannot do without --------------------------------------------------------------


def _class_sizes(case):
    ex = _expansion(case)
    n, nd = case["n"], ex.n_determinants
    ka, kb = ex.n_alpha_electrons, ex.n_beta_electrons
    return ex, n, nd, ka, kb


def _hs_work(case):
    """Per unordered spin pair of excitation level E, an E x E inverse, the E^2 entries of every
    factor column and C(E,2)^2 two-electron terms; per unordered determinant pair one dot product
    over the factor columns and two more products; per structure term a row of sums."""
    ex, n, nd, ka, kb = _class_sizes(case)
    R = min(3 * n, n * (n + 1) // 2)
    tables = {(ka, len(ex.alpha_strings))} if ka == kb else {(ka, len(ex.alpha_strings)), (kb, len(ex.beta_strings))}
    flops = 0.0
    for k, N in tables:
        for e in range(1, k + 1):
            pairs = N * math.comb(k, e) * math.comb(n - k, e) / 2
            flops += pairs * (2 * e ** 3 + 2 * e * e * (R + 2) + 5 * math.comb(e, 2) ** 2)
    pairs = nd * (nd + 1) / 2 / (2 if ka == kb else 1)
    flops += pairs * (2 * R + 6) + 2 * len(ex.term_structure) * nd
    return flops, 8.0 * (2 * n * n + (n * (n + 1) // 2) ** 2 / 2), 16.0 * ex.n_structures ** 2


def work(case):
    kind = case["kind"]
    if kind == "hs":
        f, i, o = _hs_work(case)
        return {"bytes": i + o, "flops": f}
    if kind == "root":
        f, i, _ = _hs_work(case)
        n, ns = case["n"], _expansion(case).n_structures
        F = 8.0 * 3 * n * (n * (n + 1) // 2)
        # forward, backward of the same size, and one factorization's worth for the root
        return {"bytes": i + 2 * F + 8.0 * (ns + 2 * n * n), "flops": 2 * f + ns ** 3 / 3.0}
    if kind == "scf":
        n = case["atoms"]
        f, _, _ = _hs_work({"structures": "COV", "n": n, "electrons": n, "multiplicity": 1})
        nb = 2 * n
        return {"bytes": 8.0 * (nb * (nb + 1) // 2) ** 2 / 2 + 16.0 * nb * n, "flops": 2 * f}
    if kind == "ri":
        n_bf, n_aux, a = case["n_bf"], case["n_aux"], case["n_act"]
        P = a * (a + 1) // 2
        b = 8.0 * (n_aux * (n_bf * (n_bf + 1) // 2) + n_bf * a + a * n_aux * n_bf + P * n_aux + P * (P + 1) // 2)
        f = 2.0 * n_aux * n_bf * n_bf * a + 2.0 * n_aux * n_bf * P + n_aux * P * (P + 1)
        if case["adjoint"]:
            b += 8.0 * (P * n_aux + a * n_bf + a * n_aux * n_bf)
            f += 4.0 * n_aux * n_bf * a * a
        return {"bytes": b, "flops": f}
    if kind == "cholesky":
        return {"bytes": 12.0 * case["n"] ** 2, "flops": case["n"] ** 3 / 3.0}
    if kind == "eigh":
        return {"bytes": 24.0 * case["n"] ** 2, "flops": 9.0 * case["n"] ** 3}
    sizes = np.resize([int(x) for x in case["sizes"].split(",")], case["count"])
    parts = [work(dict(_engine_class(int(n)), kind="root")) for n in sizes]
    return {k: float(sum(p[k] for p in parts)) for k in ("bytes", "flops")}


def tolerance(case):
    """FP64 everywhere but the split-precision transform (24-bit operands).  Measured against
    ``exact``: hs 3e-16, ri 3e-15, cholesky 2e-14, eigh 7e-12 (close roots), split precision 1.2e-7.
    Roots are converged to a relative residual of 1e-11, which leaves 3e-10 in vectors and
    gradients; stretched chains hold blocks whose condition number approaches 1e12."""
    kind = case["kind"]
    if kind == "hs":
        return {"rel": 1e-12, "max": 1e-10}
    if kind == "ri":
        return {"rel": 1e-13, "max": 1e-11} if case["precision"] == "fp64" else {"rel": 5e-7, "max": 2e-5}
    if kind == "cholesky":
        return {"rel": 1e-12, "max": 1e-10}
    if kind == "eigh":
        return {"rel": 1e-9, "max": 1e-6}
    if kind == "scf" and case["spacing"] > 1.5:
        return {"rel": 1e-7, "max": 1e-5}
    return {"rel": 5e-9, "max": 5e-7}


# ---- the same results from dense 64-bit algebra ------------------------------------------------


def _full_kernel(Kp, n):
    """Pair kernel over packed pairs [P, P] -> (ij|kl) as [n n, n n]."""
    i = torch.arange(n, device="cuda")
    hi, lo = torch.maximum(i[:, None], i[None]), torch.minimum(i[:, None], i[None])
    p = (hi * (hi + 1) // 2 + lo).reshape(-1)
    return Kp[p][:, p]


def _unpack(packed, P):
    K = torch.zeros(P, P, dtype=F64, device="cuda")
    r, c = torch.tril_indices(P, P, device="cuda")
    K[r, c] = packed
    K[c, r] = packed
    return K


def _spin_table(S, h, K, strings, n):
    """For all (left u, right v) strings: overlap, same-spin energy, and det * density [N, N, n n]."""
    occ = torch.tensor([[i for i in range(n) if (int(s) >> i) & 1] for s in strings], device="cuda")
    onehot = torch.nn.functional.one_hot(occ, n).to(F64)  # [N, k, n]
    Kx = K.reshape(n, n, n, n).permute(0, 3, 2, 1).reshape(n * n, n * n)
    parts = []
    for u in range(0, len(occ), 256):
        left, one = occ[u:u + 256], onehot[u:u + 256]
        X = S[occ[None, :, :, None], left[:, None, None, :]]  # [u, v, row of v, column of u]
        det = torch.linalg.det(X)
        B = torch.linalg.inv(X).transpose(-1, -2)             # cofactor / det, [u, v, r, c]
        G = torch.einsum("uvrc,vri,ucj->uvij", B, onehot, one).reshape(len(left), len(occ), n * n)
        energy = G @ h.reshape(-1) + 0.5 * ((G @ (K - Kx)) * G).sum(-1)
        parts.append((det, det * energy, det[..., None] * G))
    return [torch.cat(p) for p in zip(*parts)]


def _tables(S, h, K, ex, n):
    a = _spin_table(S, h, K, ex.alpha_strings, n)
    same = np.array_equal(ex.alpha_strings, ex.beta_strings)
    return a, a if same else _spin_table(S, h, K, ex.beta_strings, n)


def _terms(ex):
    T = torch.zeros(ex.n_determinants, ex.n_structures, dtype=F64, device="cuda")
    d = np.repeat(np.arange(ex.n_determinants), np.diff(ex.term_offsets))
    T.index_put_((torch.tensor(d, device="cuda"), torch.tensor(ex.term_structure, device="cuda").long()),
                 torch.tensor(ex.term_coefficient, device="cuda"), accumulate=True)
    return T


def _structure_matrices(S, h, K, ex, n):
    (Sa, Ha, Ga), (Sb, Hb, Gb) = _tables(S, h, K, ex, n)
    KGb = Gb @ K
    a, b = (torch.tensor(x, device="cuda").long() for x in (ex.det_alpha, ex.det_beta))
    nd = ex.n_determinants
    T = _terms(ex)
    HT, ST = (torch.empty(nd, ex.n_structures, dtype=F64, device="cuda") for _ in range(2))
    step = max(1, min(nd, (1 << 28) // (nd * n * n)))
    block = max(step, 256)
    for d0 in range(0, nd, block):
        rows = []
        for d in range(d0, min(nd, d0 + block), step):
            q = slice(d, min(nd, d0 + block, d + step))
            ia, ib = (a[q][:, None], a[None]), (b[q][:, None], b[None])
            rows.append(torch.stack([Ha[ia] * Sb[ib] + Hb[ib] * Sa[ia] + (Ga[ia] * KGb[ib]).sum(-1), Sa[ia] * Sb[ib]]))
        m = torch.cat(rows, 1)
        HT[d0:d0 + block], ST[d0:d0 + block] = m[0] @ T, m[1] @ T
    H, O = T.T @ HT, T.T @ ST
    return 0.5 * (H + H.T), 0.5 * (O + O.T)


def _lowest(H, O):
    L = torch.linalg.cholesky(O)
    A = torch.linalg.solve_triangular(L, torch.linalg.solve_triangular(L, H, upper=False).T, upper=False)
    w, V = torch.linalg.eigh(0.5 * (A + A.T))
    return w[0], torch.linalg.solve_triangular(L.T, V[:, :1], upper=True)[:, 0]


def _functional(S, h, K, ex, n, c, root):
    """c^T (H - root O) c as a differentiable function of S, h and K, at a fixed root and vector."""
    (Sa, Ha, Ga), (Sb, Hb, Gb) = _tables(S, h, K, ex, n)
    W = torch.zeros(len(ex.alpha_strings), len(ex.beta_strings), dtype=F64, device="cuda")
    W[torch.tensor(ex.det_alpha, device="cuda").long(), torch.tensor(ex.det_beta, device="cuda").long()] = _terms(ex) @ c
    M = torch.stack([Sa, Ha])
    M = W.T @ M @ W
    E = (M[1] * Sb).sum() + (M[0] * Hb).sum() - root * (M[0] * Sb).sum()
    return E + ((W.T @ Ga.permute(2, 0, 1) @ W) * (Gb @ K).permute(2, 0, 1)).sum()


def _root_exact(S, h, F, ex, n):
    S, h, F = (torch.tensor(x, device="cuda").requires_grad_() for x in (S, h, F))
    with torch.no_grad():
        root, c = _lowest(*_structure_matrices(S, h, _full_kernel(F @ F.T, n), ex, n))
    gS, gh, gF = torch.autograd.grad(_functional(S, h, _full_kernel(F @ F.T, n), ex, n, c, root), (S, h, F))
    c = c * torch.sign(c[torch.argmax(c.abs())])
    return [root.reshape(1), c, 0.5 * (gS + gS.T), 0.5 * (gh + gh.T), gF]


def _boys0(t):
    s = torch.sqrt(t.clamp_min(1e-8))
    return torch.where(t < 1e-8, 1.0 - t / 3.0, 0.5 * math.sqrt(math.pi) * torch.erf(s) / s)


def _ao_integrals(mol):
    """S, core Hamiltonian and (mu nu|la si) of contracted s functions, over the primitives."""
    xyz = torch.tensor(mol.coords, device="cuda")[torch.tensor(mol.shell_atom).long().cuda()]
    prim = torch.repeat_interleave(torch.arange(mol.n_basis), torch.tensor(mol.shell_nprim).long()).cuda()
    e = torch.tensor(mol.shell_exponents, device="cuda")
    co = torch.tensor(mol.shell_coefficients, device="cuda") * (2 * e / math.pi) ** 0.75
    D = torch.zeros(mol.n_basis, e.numel(), dtype=F64, device="cuda")
    D[prim, torch.arange(e.numel(), device="cuda")] = co
    X = xyz[prim]
    p = e[:, None] + e[None]
    mu = e[:, None] * e[None] / p
    r2 = ((X[:, None] - X[None]) ** 2).sum(-1)
    s = (math.pi / p) ** 1.5 * torch.exp(-mu * r2)
    D = D / torch.sqrt(torch.einsum("mi,ij,mj->m", D, (math.pi / p) ** 1.5, D))[:, None]
    P = (e[:, None, None] * X[:, None] + e[None, :, None] * X[None]) / p[..., None]
    nuc = torch.tensor(mol.coords, device="cuda")
    V = -(2 * math.pi / p)[..., None] * torch.exp(-mu * r2)[..., None] * _boys0(p[..., None] * ((P[:, :, None] - nuc) ** 2).sum(-1))
    core = mu * (3 - 2 * mu * r2) * s + (V * torch.tensor(mol.charges, device="cuda")).sum(-1)
    m = e.numel()
    pf, Pf, pre = p.reshape(-1), P.reshape(-1, 3), torch.exp(-mu * r2).reshape(-1) / p.reshape(-1)
    psum = pf[:, None] + pf[None]
    eri = 2 * math.pi ** 2.5 * pre[:, None] * pre[None] / torch.sqrt(psum)
    eri = eri * _boys0(pf[:, None] * pf[None] / psum * ((Pf[:, None] - Pf[None]) ** 2).sum(-1))
    eri = torch.einsum("mi,nj,ijq->mnq", D, D, eri.reshape(m, m, -1))
    eri = torch.einsum("lk,st,qkt->qls", D, D, eri.reshape(-1, m, m)).reshape([mol.n_basis] * 4)
    d = (nuc[:, None] - nuc[None]).norm(dim=-1)
    enuc = sum(mol.charges[i] * mol.charges[j] / float(d[i, j]) for i in range(len(nuc)) for j in range(i))
    return D @ s @ D.T, D @ core @ D.T, eri, enuc


def _scf_exact(case, seed):
    mol, pattern, C = _chain(case, seed)
    n = case["atoms"]
    ex = _expansion({"structures": "COV", "n": n, "electrons": n, "multiplicity": 1})
    Sao, hao, eri, enuc = _ao_integrals(mol)
    C = torch.tensor(C, device="cuda").requires_grad_()

    def active():
        K = torch.einsum("abcd,ai,bj->ijcd", eri, C, C)
        return C.T @ Sao @ C, C.T @ hao @ C, torch.einsum("ijcd,ck,dl->ijkl", K, C, C).reshape(n * n, n * n)

    with torch.no_grad():
        root, c = _lowest(*_structure_matrices(*active(), ex, n))
    g, = torch.autograd.grad(_functional(*active(), ex, n, c, root), C)
    mask = torch.zeros_like(g)
    for a, functions in enumerate(pattern):
        mask[functions, a] = 1.0
    return [root.reshape(1) + enuc, g * mask]


def _ri_exact(case, seed):
    B, C, dL = _ri_inputs(case, seed)
    n_bf, n_act = case["n_bf"], case["n_act"]
    C = C.requires_grad_()
    i = torch.arange(n_bf, device="cuda")
    hi, lo = torch.maximum(i[:, None], i[None]), torch.minimum(i[:, None], i[None])
    full = B[(hi * (hi + 1) // 2 + lo).reshape(-1)].reshape(n_bf, n_bf, -1)
    T = torch.einsum("mvP,am->vaP", full, C)
    r, c = torch.tril_indices(n_act, n_act, device="cuda")
    L = torch.einsum("vaP,bv->abP", T, C)[r, c]
    K = L @ L.T
    pr, pc = torch.tril_indices(L.shape[0], L.shape[0], device="cuda")
    out = [T.detach(), L.detach(), K[pr, pc].detach()]
    return out + ([torch.autograd.grad((L * dL).sum(), C)[0]] if case["adjoint"] else [])


def exact(case, seed):
    kind = case["kind"]
    if kind == "hs":
        S, h, eri, _ = _active_space(case["n"], seed)
        n = case["n"]
        K = _full_kernel(_unpack(torch.tensor(eri, device="cuda"), n * (n + 1) // 2), n)
        S, h = (torch.tensor(x, device="cuda") for x in (S, h))
        return list(_structure_matrices(S, h, K, _expansion(case), n))
    if kind == "root":
        S, h, _, F = _active_space(case["n"], seed)
        return _root_exact(S, h, F, _expansion(case), case["n"])
    if kind == "scf":
        # singular overlap blocks have no inverse, and the tables of 14 orbitals with their
        # gradients are too large
        return _scf_exact(case, seed) if case["spacing"] <= 1.5 and case["atoms"] <= 12 else None
    if kind == "ri":
        return _ri_exact(case, seed)
    if kind in ("cholesky", "eigh"):
        H, S = _metric_inputs(case, seed)
        if kind == "cholesky":
            return torch.linalg.cholesky(S)  # row j = column j of U
        L = torch.linalg.cholesky(S)
        A = torch.linalg.solve_triangular(L, torch.linalg.solve_triangular(L, H, upper=False).T, upper=False)
        w, V = torch.linalg.eigh(0.5 * (A + A.T))
        V = torch.linalg.solve_triangular(L.T, V, upper=True).T
        phase = torch.randn(case["n"], dtype=F64, generator=torch.Generator().manual_seed(1)).cuda()
        return [w, V * torch.sign(V @ phase)[:, None]]
    sizes, data = _engine_instances(case, seed)
    parts = [_root_exact(S, h, F, _expansion(_engine_class(n)), n) for n, (S, h, _, F) in zip(sizes, data)]
    return [torch.cat([p[0] for p in parts])] + [torch.cat([p[k].reshape(-1) for p in parts]) for k in (2, 3, 4)]
