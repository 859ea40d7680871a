"""Outer updates of an FP32 factor without tensor cores: the trailing matrices from the 128-tile line on
run on 128-tiles whatever their number in a step (the rule that sends few of them to 64-tiles was
measured for, and holds for, an FP64 factor)."""
import numpy as np
import pytest

from oracle import refcpu
from rustyfem_b200 import ffi, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [13, 20])
def test_128_tiles(gpu, n):
    m = W.hex8_cube(n).full()
    h, _, _ = ffi.factor(m, precision=ffi.MIXED, tensor_cores=False)
    assert h is not None, ffi.last_error()
    ho, _, _ = refcpu.factor(m)
    try:
        # the root of the 13³ cube: 588 pivots, 332 of them behind the first outer block
        assert h.stats()["schur_flops"] > 0
        x, xo = h.solve(m.rhs), ho.solve(m.rhs)
        assert np.linalg.norm(x - xo) <= 1e-8 * np.linalg.norm(xo)
    finally:
        h.free()
