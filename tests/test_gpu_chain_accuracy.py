"""The FP64 sweeps on the solve chains of the top levels round like the stepped sweeps: residuals in
extended precision of the same right-hand sides. Both substitute by blocks of 64 pivots with other
orders of the sums; the norm of 10⁵ rounding errors then agrees to a few parts in a hundred. A product
with the explicit inverse of a 256-pivot block gives a 2-norm 1.10 times as large on this model (six
right-hand sides); the bar lies in the middle."""
import numpy as np
import pytest

from rustyfem_b200 import ffi, workloads as W

pytestmark = pytest.mark.gpu


def residual_norms(m, b, x):
    d = m.data.astype(np.longdouble)
    out = []
    for j in range(len(b)):
        ax = np.add.reduceat(d * x[j][m.indices].astype(np.longdouble), m.indptr[:-1])
        out.append(np.linalg.norm((b[j] - ax).astype(float)) / np.linalg.norm(x[j]))
    return np.array(out)


@pytest.mark.parametrize("nrhs", [1, 6])
def test_residuals_of_the_stepped_sweeps(gpu, monkeypatch, nrhs):
    m = W.hex20_cube(20).full()
    rng = np.random.default_rng(3)
    b = rng.standard_normal((6, m.n))
    norms = []
    for chain in (True, False):
        if not chain:
            monkeypatch.setenv("RFG_SOLVE_CHAIN", "0")
        h, _, _ = ffi.factor(m)
        assert h is not None, ffi.last_error()
        try:
            x = h.solve(b) if nrhs > 1 else np.array([h.solve(v) for v in b])
        finally:
            h.free()
        norms.append(residual_norms(m, b, x))
    assert np.exp(np.log(norms[0] / norms[1]).mean()) <= 1.05
