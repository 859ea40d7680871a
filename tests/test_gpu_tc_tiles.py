"""The persistent tensor-core kernel when a CTA has more than 32 tiles of a launch (a warp decodes 32
at a time): the 60³ cube, whose two fronts below the root (16,500 rows each) make 8,000 tiles of
128 × 256 in one step, 55 per CTA on 148 SMs. A tile left out or decoded wrongly leaves entries of
the size of the matrix. Tolerance of the unrefined solve's normwise backward error: the rounding of
the FP32 factor, 2⁻²⁴ times the root of the largest front's rows, 129 × 6e-8 = 8e-6."""
import numpy as np
import pytest
import scipy.sparse as sp

from rustyfem_b200 import ffi, workloads as W

pytestmark = pytest.mark.gpu


def test_more_than_32_tiles_per_cta(gpu):
    model = W.hex8_cube(60).full()
    h, err, _ = ffi.factor(model, precision=ffi.MIXED, refine_max_iter=0)
    assert h is not None, ffi.last_error()
    x = h.solve(model.rhs)
    h.free()
    a = sp.csc_matrix((model.data, model.indices, model.indptr), shape=(model.n, model.n))
    norm = abs(a).sum(axis=0).max()  # symmetric: the row sums are the column sums
    eta = np.abs(model.rhs - a @ x).max() / (norm * np.abs(x).max() + np.abs(model.rhs).max())
    assert eta <= 8e-6
