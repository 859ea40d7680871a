"""Sweeps of five and more right-hand sides (groups of eight on the FP64 tensor-core path), stepped
and on chains, with the FP64 and the FP32 factor; and a front without pivots.

The widths are the edges of the groups (5, 8, 9, 16, 17, 24, 25, 32) and one beyond a sweep (33).
Bars: FP64 the parity bar against the oracle; FP32 factor, one sweep without refinement against
the same factor's single right-hand-side sweeps (same factor, another order of sums in FP64)."""
import dataclasses

import numpy as np
import pytest

from oracle import refcpu
from rustyfem_b200 import ffi, workloads as W

pytestmark = pytest.mark.gpu

WIDTHS = (5, 8, 9, 16, 17, 24, 25, 32, 33)
MODELS = {
    "plate 30x3": lambda: W.plate(30, 3),
    "cube 2": lambda: W.hex8_cube(2),
    "cube 7": lambda: W.hex8_cube(7),
    "cube 15": lambda: W.hex8_cube(15),
    "hex20 4": lambda: W.hex20_cube(4),
}


def set_chain(monkeypatch, chain):
    if chain is None:
        monkeypatch.delenv("RFG_SOLVE_CHAIN", raising=False)
    else:
        monkeypatch.setenv("RFG_SOLVE_CHAIN", chain)


@pytest.mark.parametrize("chain", [None, "0", "100000"])
@pytest.mark.parametrize("name", list(MODELS))
def test_widths(gpu, monkeypatch, name, chain):
    set_chain(monkeypatch, chain)
    m = MODELS[name]().full()
    rng = np.random.default_rng(17)
    b = rng.standard_normal((max(WIDTHS), m.n)) * 1e3
    ho, _, _ = refcpu.factor(m)
    xo = np.stack([ho.solve(bb) for bb in b])
    h, _, _ = ffi.factor(m)
    assert h is not None, ffi.last_error()
    hm, _, _ = ffi.factor(m, precision=ffi.MIXED, refine_max_iter=0)
    assert hm is not None, ffi.last_error()
    try:
        x1 = np.stack([hm.solve(bb) for bb in b])
        for nrhs in WIDTHS:
            for _ in range(3):  # launched, captured, replayed
                x = h.solve(b[:nrhs])
                assert np.linalg.norm(x - xo[:nrhs]) <= 1e-10 * np.linalg.norm(xo[:nrhs]), nrhs
            xm = hm.solve(b[:nrhs])
            assert np.linalg.norm(xm - x1[:nrhs]) <= 1e-10 * np.linalg.norm(x1[:nrhs]), nrhs
    finally:
        h.free()
        hm.free()


def two_chains(n):
    """Two uncoupled chains of n nodes, the second moved aside: separators without nodes."""
    a = W.chain(n, lambda c: 2.5 + 0.01 * c, lambda r, c: -1.0)
    xyz = a.coords.reshape(-1, 3).copy()
    far = xyz + np.array([4.0 * n, 0.0, 0.0])
    nnz = a.indptr[-1]
    return dataclasses.replace(
        a, name="two chains", n=2 * n, nn=2 * n, loc=np.arange(2 * n, dtype=np.int64),
        coords=np.concatenate([xyz, far]).ravel(), indptr=np.concatenate([a.indptr, a.indptr[1:] + nnz]),
        indices=np.concatenate([a.indices, a.indices + n]), data=np.concatenate([a.data, a.data]),
        rhs=np.zeros(2 * n))


def comb(arms, n, dy):
    """Parallel chains joined at one end: parts of the dissection that are not connected, so that a
    separator without nodes has later rows to pass on."""
    import scipy.sparse as sp

    e = [(a * n + i, a * n + i + 1) for a in range(arms) for i in range(n - 1)]
    e += [(a * n - 1, (a + 1) * n - 1) for a in range(1, arms)]
    i, j = np.array(e).T
    N = arms * n
    A = sp.coo_matrix((-np.ones(len(i)), (i, j)), shape=(N, N))
    A = (A + A.T + sp.diags(np.linspace(3.5, 4.0, N))).tocsc()
    A.sort_indices()
    xyz = np.zeros((N, 3))
    xyz[:, 0] = np.tile(np.arange(n), arms)
    xyz[:, 1] = np.repeat(np.arange(arms), n) * dy
    return W.Model("comb", N, N, np.arange(N, dtype=np.int64), xyz.ravel(), A.indptr.astype(np.int64),
                   A.indices.astype(np.int64), A.data, np.zeros(N), symmetric_storage="full")


@pytest.mark.parametrize("chain", [None, "100000"])
@pytest.mark.parametrize("name", ["two chains", "comb"])
def test_front_without_pivots(gpu, monkeypatch, name, chain):
    set_chain(monkeypatch, chain)
    m = two_chains(90) if name == "two chains" else comb(8, 64, 3.0)
    ho, _, _ = refcpu.factor(m)
    h, _, _ = ffi.factor(m)
    assert h is not None, ffi.last_error()
    empty = h.fronts()[h.fronts()[:, 1] == 0]
    assert len(empty) and (name == "two chains" or (empty[:, 2] > 0).any())
    b = np.random.default_rng(23).standard_normal((12, m.n))
    try:
        for nrhs in (1, 3, 12):
            x = h.solve(b[:nrhs])
            xo = np.stack([ho.solve(bb) for bb in b[:nrhs]])
            assert np.linalg.norm(x - xo) <= 1e-10 * np.linalg.norm(xo), nrhs
    finally:
        h.free()
