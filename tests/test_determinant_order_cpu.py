"""Determinant order and reduction form of a plan (csrc/determinant_order.cpp), built into a shared object of
its own: host code, no GPU."""

import ctypes
import os
import subprocess

import numpy as np
import pytest

import vbcore

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TILE_ROWS = 64


@pytest.fixture(scope="module")
def order_of(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("order") / "libdeterminant_order.so")
    proc = subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-I", os.path.join(ROOT, "include"), "-I",
                           os.path.join(ROOT, "xmvb-cpp_b200", "csrc"), "-I", "/usr/local/cuda/include",
                           os.path.join(ROOT, "xmvb-cpp_b200", "csrc", "determinant_order.cpp"),
                           os.path.join(ROOT, "tests", "shim", "determinant_order_shim.cpp"), "-o", so],
                          capture_output=True, text=True)
    assert proc.returncode == 0, proc.stderr
    lib = ctypes.CDLL(so)

    def call(ex, n, coefficients=False):
        arrays = [np.ascontiguousarray(x, dtype=t) for x, t in (
            (ex.alpha_strings, np.uint64), (ex.beta_strings, np.uint64), (ex.det_alpha, np.int32),
            (ex.det_beta, np.int32), (ex.term_offsets, np.int64), (ex.term_structure, np.int32),
            (ex.term_coefficient, np.float64))]
        p = [a.ctypes.data for a in arrays]
        nd = ex.n_determinants
        c = vbcore._Expansion(n, ex.n_alpha_electrons, ex.n_beta_electrons, len(ex.alpha_strings),
                              len(ex.beta_strings), p[0], p[1], nd, p[2], p[3], ex.n_structures, p[4], p[5], p[6])
        out, position = np.zeros(5, dtype=np.int64), np.zeros(nd, dtype=np.int64)
        T = np.zeros((ex.n_structures, nd)) if coefficients else None
        lib.order_of(ctypes.byref(c), out.ctypes.data_as(ctypes.c_void_p), position.ctypes.data_as(ctypes.c_void_p),
                     T.ctypes.data_as(ctypes.c_void_p) if coefficients else None)
        return dict(zip(("blocks", "groups", "rows", "segments", "caller"), out.tolist())), position, T

    return call


def _expansion(kw, n, mult):
    return vbcore.expand_structures(vbcore.generate_structures(kw, n, n, mult), n, mult)


def _first_structure_segments(ex):
    """Segments with every determinant at the structure group that uses it first (alpha-major inside)."""
    d_of = np.repeat(np.arange(ex.n_determinants), np.diff(ex.term_offsets))
    first = np.full(ex.n_determinants, ex.n_structures)
    np.minimum.at(first, d_of, ex.term_structure)
    order = np.lexsort((ex.det_beta, ex.det_alpha, first // 64))
    position = np.empty(ex.n_determinants, dtype=np.int64)
    position[order] = np.arange(ex.n_determinants)
    return len(np.unique(ex.term_structure.astype(np.int64) // 64 * (1 << 32) + position[d_of] // TILE_ROWS))


@pytest.mark.parametrize("kw,n,mult", [("COV", 8, 1), ("COV", 12, 1), ("COV", 11, 2), ("COV ION(1)", 6, 1), ("COV ION(1)", 8, 1),
                                       ("COV ION(1)", 9, 2), ("COV ION(1)", 8, 3), ("COV ION(1-2)", 8, 1), ("FULL", 6, 1),
                                       ("COV ION(1)", 12, 1), ("COV ION(1)", 13, 2), ("COV ION(1)", 14, 1)])
def test_reduction_reads_no_more_than_the_other_orders(order_of, kw, n, mult):
    """Rows of the determinant matrix that the reduction streams for every column: those of the dense groups, or
    64 per segment.  Neither the caller's order nor the first-structure order would stream fewer than half, and
    lists ordered by blocks (whose pair products that order serves) at most four times their rows more."""
    ex = _expansion(kw, n, mult)
    got, position, _ = order_of(ex, n)
    assert np.array_equal(np.sort(position), np.arange(ex.n_determinants))
    rows = got["rows"] if got["groups"] else TILE_ROWS * got["segments"]
    other = TILE_ROWS * min(got["caller"], _first_structure_segments(ex))
    assert rows <= (max(2 * other, 4 * ex.n_determinants) if got["blocks"] else 2 * other)


@pytest.mark.parametrize("kw,n,mult", [("COV ION(1)", 8, 1), ("COV ION(1)", 9, 2), ("COV ION(1)", 10, 1), ("COV ION(1-2)", 8, 1)])
def test_groups_hold_every_term_once(order_of, kw, n, mult):
    ex = _expansion(kw, n, mult)
    got, position, T = order_of(ex, n, coefficients=True)
    assert got["blocks"] and got["groups"]
    ref = np.zeros_like(T)
    d_of = np.repeat(np.arange(ex.n_determinants), np.diff(ex.term_offsets))
    np.add.at(ref, (ex.term_structure, position[d_of]), ex.term_coefficient)
    assert np.array_equal(T, ref)


def test_repeated_terms_take_the_tiled_reduction(order_of):
    """Two terms of one structure and determinant do not fit the dense groups; the block order is kept only
    where the tiled reduction reads few rows more in it."""
    for n in (8, 10, 12, 14):
        ex = _expansion("COV ION(1)", n, 1)
        ex.term_offsets = 2 * ex.term_offsets
        ex.term_structure = np.repeat(ex.term_structure, 2)
        ex.term_coefficient = 0.5 * np.repeat(ex.term_coefficient, 2)
        got, _, _ = order_of(ex, n)
        assert got["groups"] == 0
        extra = got["segments"] - _first_structure_segments(ex)
        assert extra < ex.n_determinants if got["blocks"] else extra <= 0 or got["segments"] == got["caller"]
