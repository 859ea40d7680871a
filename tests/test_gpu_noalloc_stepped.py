"""rfg_solve_device_noalloc where the solve chains do not fit beside its need in the fixed scratch: every
level runs stepped. With chains asked for on every level (RFG_SOLVE_CHAIN) the column pieces' partial sums
of an FP64 factor, and in the mixed path the flags alone, take the need over 16 MiB. The values are those of
a handle without chains bit for bit, and not those of the chained one."""
import ctypes

import numpy as np
import pytest

from rustyfem_b200 import ffi, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,model,nrhs", [
    # need with chains / without (bytes): 18,096,384 / 15,929,344; 19,211,008 / 8,997,120
    (ffi.FP64, lambda: W.hex8_cube(20), 8), (ffi.FP64, lambda: W.plate(200, 20), 24),
    # 16,796,928 / 16,772,096; 16,782,336 / 16,765,952
    (ffi.MIXED, lambda: W.plate(198, 33), 13), (ffi.MIXED, lambda: W.plate(209, 20), 20)])
def test_stepped_without_room_for_the_chains(gpu, monkeypatch, precision, model, nrhs):
    import torch

    m = model().full()
    b = torch.from_numpy(np.random.default_rng(nrhs).standard_normal((nrhs, m.n))).cuda()
    out = {}
    for chain in ("100000", "0"):
        monkeypatch.setenv("RFG_SOLVE_CHAIN", chain)
        h, _, _ = ffi.factor(m, precision=precision, refine_max_iter=0)
        assert h is not None, ffi.last_error()
        try:
            x, y = b.clone(), b.clone()
            torch.cuda.synchronize()
            assert ffi.lib().rfg_solve_device(h.ptr, nrhs, ctypes.c_void_p(x.data_ptr()), None) == 0, ffi.last_error()
            h.solve_device_noalloc(y.data_ptr(), nrhs)
            torch.cuda.synchronize()
            out[chain] = (x, y)
        finally:
            h.free()
    stepped = out["0"][0]
    assert torch.equal(out["0"][1], stepped)
    assert torch.equal(out["100000"][1], stepped)
    assert not torch.equal(out["100000"][0], stepped)
