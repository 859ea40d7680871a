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


@pytest.mark.parametrize("n", [17, 27])
def test_forks_and_other_values(gpu, n):
    """The look-ahead runs (a step that forks with a next block's columns launches its outer update in two
    parts): four of the five forked steps of the 17³ cube have their rest on 64-tiles alone, fourteen of the
    27³ cube's eighteen on 128-tiles alone. With other values in between every factorization gives the bits of a fresh
    handle's."""
    ms = [W.hex8_cube(n, emod=W.log_uniform_moduli(n, 1e9, 1e11, seed=s)).full() for s in range(3)]
    want = []
    for m in ms:
        h, _, _ = ffi.factor(m)
        assert h is not None, ffi.last_error()
        want.append(h.solve(m.rhs))
        h.free()
    h, _, _ = ffi.factor(ms[0])
    try:
        launches = h.stats()["launches"]
        h.set_profiling(1)
        assert h.refactor(ms[1].data) == -1
        assert launches > h.stats()["launches"]
        h.set_profiling(0)
        for i in (1, 2, 0, 2, 1, 0):
            assert h.refactor(ms[i].data) == -1
            assert np.array_equal(h.solve(ms[i].rhs), want[i]), i
    finally:
        h.free()
