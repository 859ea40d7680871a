"""FP64 factorizations whose outer updates run partly beside the next outer block's steps (fronts of
several 256-pivot blocks with a rest of at least one CTA per SM): pivots against the oracle, and the
same bits from the directly launched, the captured and the replayed numeric phase, and with
profiling on (every launch on one stream)."""
import numpy as np
import pytest

from oracle import refcpu
from rustyfem_b200 import ffi, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [17, 21])
def test_side_stream(gpu, n):
    m = W.hex8_cube(n, emod=W.log_uniform_moduli(n, 1e9, 1e11, seed=n)).full()
    _, _, do = refcpu.factor(m, want_d=True)
    h, _, d = ffi.factor(m, want_d=True)
    assert h is not None, ffi.last_error()
    try:
        assert np.max(np.abs(d - do) / np.abs(do)) <= 1e-10
        x = h.solve(m.rhs)
        for level in (0, 0, 1, 2, 0):
            h.set_profiling(level)
            assert h.refactor(m.data) == -1
            assert np.array_equal(h.solve(m.rhs), x), level
    finally:
        h.free()
