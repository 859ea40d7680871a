"""The same FP64 factorization and solve many times over, from replayed graphs with the outer updates of
large fronts on the second stream: moduli over six decades, every solution bit for bit the first one. A
read that meets its writer by timing alone shows here as a run that differs (the numeric phase and the
sweeps add in a fixed order, so equal inputs give equal bits). And a pivot refused while an outer update
is on the second stream: the DOF is the one of the single-stream schedule, and the next good
factorization gives the bits of the first."""
import numpy as np
import pytest

from rustyfem_b200 import ffi, workloads as W

pytestmark = pytest.mark.gpu


def graded(n):
    return W.hex8_cube(n, emod=W.log_uniform_moduli(n, seed=0)).full()


@pytest.mark.parametrize("n,times,nrhs", [(33, 200, 1), (33, 60, 12), (45, 100, 1)])
def test_same_bits(gpu, n, times, nrhs):
    import torch

    m = graded(n)
    rhs = np.random.default_rng(n).standard_normal((nrhs, m.n))
    rhs[0] = m.rhs
    data, b0 = torch.from_numpy(m.data).cuda(), torch.from_numpy(rhs).cuda()
    h, _, _ = ffi.factor(m)
    assert h is not None, ffi.last_error()
    try:
        first = None
        for i in range(times):
            if i:
                assert h.refactor_device(data.data_ptr()) == -1, ffi.last_error()
            b = b0.clone()
            torch.cuda.synchronize()
            eta = h.solve_device(b.data_ptr(), nrhs)["backward_error"]
            assert eta <= 1e-12, i
            if first is None:
                first = b
            assert torch.equal(b, first), i
    finally:
        h.free()


def test_same_bits_beside_other_handles(gpu):
    # three threads with a handle each, so that launches, CTAs and warps meet in other orders
    import threading

    jobs = [(graded(25), ffi.FP64, 1), (graded(21), ffi.FP64, 6), (graded(21), ffi.MIXED, 1)]
    failed = []

    def run(m, precision, nrhs):
        rhs = np.random.default_rng(nrhs).standard_normal((nrhs, m.n))
        h, _, _ = ffi.factor(m, precision=precision)
        try:
            first = h.solve(rhs)
            for i in range(100):
                if h.refactor(m.data) != -1 or not np.array_equal(h.solve(rhs), first):
                    failed.append((m.name, precision, i, ffi.last_error()))
        finally:
            h.free()

    threads = [threading.Thread(target=run, args=job) for job in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed


@pytest.mark.parametrize("front", ["root", "largest below the root"])
def test_refused_beside_an_update(gpu, front):
    m = W.hex8_cube(27).full()
    h, _, _ = ffi.factor(m)
    assert h is not None, ffi.last_error()
    try:
        x = h.solve(m.rhs)
        k = h.fronts()[:, 1]
        big = np.argsort(k, kind="stable")[::-1]
        t = big[0] if front == "root" else big[1]
        assert k[t] > 3 * 256
        start = int(h.fronts()[t, 0])
        dof_of = np.argsort(h.order())
        for pos in (300, 511, 512, 600, 769):
            dof = int(dof_of[start + pos])
            bad = m.data.copy()
            col = m.indices[m.indptr[dof]:m.indptr[dof + 1]]
            bad[m.indptr[dof] + np.searchsorted(col, dof)] = -1.0
            for level in (0, 1, 0):
                h.set_profiling(level)
                assert h.refactor(bad) == dof, (pos, level)
            h.set_profiling(0)
            assert h.refactor(m.data) == -1
            assert np.array_equal(h.solve(m.rhs), x), pos
    finally:
        h.free()
