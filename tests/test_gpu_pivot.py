"""The pivot block at the edges of its sub-panels (8 pivots) and 16 × 16 inverses: fronts of 1 to 64
pivots. Pivots D one by one against the oracle (relative 1e-10, the FP64 parity bar), and a pivot
that breaks the rule at each place of a sub-panel gives the oracle's DOF."""
import dataclasses

import numpy as np
import pytest

from oracle import refcpu
from rustyfem_b200 import ffi
from test_gpu_panel import block_chain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [1, 7, 8, 9, 15, 16, 17, 24, 25, 40, 48, 56, 57, 63, 64])
def test_pivots(gpu, w):
    m = block_chain(3, w, seed=100 + w)
    _, _, do = refcpu.factor(m, want_d=True)
    h, _, d = ffi.factor(m, want_d=True)  # leaf 16: one front of all the nodes' DOFs
    assert h is not None, ffi.last_error()
    h.free()
    assert np.max(np.abs(d - do) / np.abs(do)) <= 1e-10


@pytest.mark.parametrize("bad", [0, 1, 7, 8, 13, 15, 16, 31, 38])
@pytest.mark.parametrize("value", [0.0, -5.0, float("nan")])
def test_refused_pivot(gpu, bad, value):
    m = block_chain(1, 39, seed=7)
    data = m.data.copy()
    data[m.indptr[bad] + np.searchsorted(m.indices[m.indptr[bad]:m.indptr[bad + 1]], bad)] = value
    m = dataclasses.replace(m, data=data)
    ho, eo, _ = refcpu.factor(m)
    h, e, _ = ffi.factor(m)
    assert ho is None and h is None and e == eo == bad
