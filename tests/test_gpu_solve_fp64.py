"""Sweeps of the FP64 factor with one to four right-hand sides: the prefetching step kernels
(diagonal blocks of one to four 64-pivot sub-blocks, 32-row CTAs) and the solve chains.

RFG_SOLVE_CHAIN = 0 steps every level (the full 256-pivot blocks stream their last four tiles
through the slots of the first), 100000 puts every level on chains, unset takes the plan's rule.
The bar is the FP64 parity bar against the oracle. The models' widest fronts per level cover
k = 3 (one element layer), blocks that end inside a sub-block, k just above 64, 128, 192 and
256, and fronts of several blocks."""
import numpy as np
import pytest

from oracle import refcpu
from rustyfem_b200 import ffi, workloads as W

pytestmark = pytest.mark.gpu

MODELS = {
    "plate 30x3": lambda: W.plate(30, 3),
    "cube 2": lambda: W.hex8_cube(2),
    "cube 7": lambda: W.hex8_cube(7),
    "cube 9": lambda: W.hex8_cube(9),
    "cube 15": lambda: W.hex8_cube(15),
    "hex20 4": lambda: W.hex20_cube(4),
}


@pytest.mark.parametrize("chain", [None, "0", "100000"])
@pytest.mark.parametrize("name", list(MODELS))
def test_sweep_against_oracle(gpu, monkeypatch, name, chain):
    if chain is None:
        monkeypatch.delenv("RFG_SOLVE_CHAIN", raising=False)
    else:
        monkeypatch.setenv("RFG_SOLVE_CHAIN", chain)
    m = MODELS[name]().full()
    ho, _, _ = refcpu.factor(m)
    h, _, _ = ffi.factor(m)
    assert h is not None, ffi.last_error()
    rng = np.random.default_rng(11)
    try:
        for nrhs in (1, 2, 3, 4):
            b = rng.standard_normal((nrhs, m.n)) * 1e3
            xo = np.stack([ho.solve(bb) for bb in b])
            for _ in range(3):  # launched, captured, replayed
                x = h.solve(b)
                assert np.linalg.norm(x - xo) <= 1e-10 * np.linalg.norm(xo), nrhs
    finally:
        h.free()
