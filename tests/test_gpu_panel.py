"""The panel kernel at the edges of its tiles: pivot blocks of 1 to 64 pivots (parts of 16-column
groups, of four-column loads), 1 row to several chunks of 64 rows below a block. A chain of blocks
with `w` DOFs per node, dissected into leaves of one node, has fronts of w pivots with w or 2w later
rows. Pivots D and the solution against the oracle at the FP64 parity bar."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import refcpu
from rustyfem_b200 import ffi, workloads as W

pytestmark = pytest.mark.gpu


def block_chain(nodes, w, seed=0, shift=None):
    """SPD: a chain of dense w × w blocks, diagonally dominant (or with the given shift)."""
    rng = np.random.default_rng(seed)
    n = nodes * w
    A = sp.lil_matrix((n, n))
    for b in range(nodes):
        D = rng.uniform(-1, 1, (w, w))
        A[b * w:(b + 1) * w, b * w:(b + 1) * w] = D + D.T + (8 * w if shift is None else shift) * np.eye(w)
        if b + 1 < nodes:
            O = rng.uniform(-1, 1, (w, w))
            A[(b + 1) * w:(b + 2) * w, b * w:(b + 1) * w] = O
            A[b * w:(b + 1) * w, (b + 1) * w:(b + 2) * w] = O.T
    A = sp.csc_matrix(A)
    A.sort_indices()
    xyz = np.zeros((nodes, 3))
    xyz[:, 0] = np.arange(nodes)
    return W.Model(f"block chain {w}", n, nodes, np.repeat(np.arange(nodes), w), xyz.ravel(),
                   A.indptr.astype(np.int64), A.indices.astype(np.int64), A.data, np.ones(n), symmetric_storage="full")


@pytest.mark.parametrize("w", [1, 2, 3, 4, 5, 8, 15, 16, 17, 31, 33, 47, 49, 63, 64, 65, 80, 130])
def test_block_widths(gpu, w):
    m = block_chain(7, w, seed=w)
    ho, _, do = refcpu.factor(m, want_d=True)
    h, _, d = ffi.factor(m, want_d=True, leaf=1)
    assert h is not None, ffi.last_error()
    hm, _, dm = ffi.factor(m, want_d=True, precision=ffi.MIXED, leaf=1)
    assert hm is not None, ffi.last_error()
    try:
        xo = ho.solve(m.rhs)
        assert np.linalg.norm(h.solve(m.rhs) - xo) <= 1e-10 * np.linalg.norm(xo)
        assert np.linalg.norm(hm.solve(m.rhs) - xo) <= 1e-8 * np.linalg.norm(xo)
        # the same permutation gives the same pivots (the product of all of them in any order)
        assert abs(np.log(d).sum() - np.log(do).sum()) <= 1e-10 * m.n
        assert abs(np.log(dm).sum() - np.log(do).sum()) <= 1e-5 * m.n
    finally:
        h.free()
        hm.free()


@pytest.mark.parametrize("w", [1, 2, 3, 4, 5, 8, 15, 16, 17, 31, 33, 47, 49, 63, 64, 65, 80, 130])
def test_block_widths_unrefined(gpu, w):
    """The FP32 panels without refinement to hide an error, on a matrix whose coupling counts: a block's
    D + Dᵀ has a spectral radius near 1.63·√w and each of its two neighbours adds 1.15·√w, so the shift
    5·√w + 2 leaves a condition below (5 + 3.93) / (5 − 3.93) = 8.4, and a coupling term of w/3 / (5·√w) is
    1.3 % of the pivots it changes: a column left out moves them and the solution by 1e-4 at w = 130 and by
    more below. FP32 rounding over fronts of at most 260 pivots stays under 8.4·√260·2⁻²⁴ = 8e-6; the bar
    is 1e-5. Pivots one by one against the FP64 handle of the same order."""
    m = block_chain(7, w, seed=w, shift=5 * np.sqrt(w) + 2)
    h, _, d = ffi.factor(m, want_d=True, leaf=1)
    assert h is not None, ffi.last_error()
    hm, _, dm = ffi.factor(m, want_d=True, precision=ffi.MIXED, leaf=1, refine_max_iter=0)
    assert hm is not None, ffi.last_error()
    try:
        assert np.max(np.abs(dm - d) / d) <= 1e-5
        b = np.random.default_rng(w).standard_normal(m.n)
        x = h.solve(b)
        assert np.linalg.norm(hm.solve(b) - x) <= 1e-5 * np.linalg.norm(x)
        assert np.linalg.norm(m.matvec(x) - b) <= 1e-13 * np.linalg.norm(b)
    finally:
        h.free()
        hm.free()
