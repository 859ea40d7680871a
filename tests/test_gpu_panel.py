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


def block_chain(nodes, w, seed=0):
    """SPD: a chain of dense w × w blocks, diagonally dominant."""
    rng = np.random.default_rng(seed)
    n = nodes * w
    A = sp.lil_matrix((n, n))
    for b in range(nodes):
        D = rng.uniform(-1, 1, (w, w))
        A[b * w:(b + 1) * w, b * w:(b + 1) * w] = D + D.T + 8 * w * np.eye(w)
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
