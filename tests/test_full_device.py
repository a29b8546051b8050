"""A device that is too full for default choices made for speed: what fits without them is factorised and solved.  The full
device is an allocation limit of the calling thread."""
import gc

import numpy as np
import pytest

from magla_gb300 import (DeviceOutOfMemoryError, FillReducingOrdering, Precision, SymmetricCSRMatrix, SymmetricUtduSolver,
                         UtduSolverOptions)

from .conftest import relative_residual

pytestmark = pytest.mark.gpu
NATURAL = FillReducingOrdering.Natural


def dense(n):
    i, j = np.triu_indices(n)
    rng = np.random.default_rng(n)
    v = np.where(i == j, 2.0 * n, rng.uniform(-1.0, 1.0, len(i)))
    return SymmetricCSRMatrix.from_triplets(n, i.astype(np.int32), j.astype(np.int32), v)


def solver(**kw):
    return SymmetricUtduSolver(UtduSolverOptions(Ordering=NATURAL, **kw))


@pytest.fixture
def limit(gpu_lib):
    """limit(bytes): the thread's allocation limit; returns the bytes held under the one before."""
    gc.collect()
    yield gpu_lib.uchol_check_allocation_limit
    gpu_lib.uchol_check_allocation_limit(-1)


def least_budget(sym, **kw):
    lo, hi = 1 << 20, 1 << 32
    while hi - lo > 1:
        mid = (lo + hi) // 2
        try:
            sym.EstimateDeviceBytes(UtduSolverOptions(Ordering=NATURAL, DeviceMemoryBudget=mid, **kw))
            hi = mid
        except DeviceOutOfMemoryError:
            lo = mid
    return hi


CASES = [dict(Precision=Precision.FP64), dict(Precision=Precision.TF32)]   # digits; inverse fronts past 2048 columns


@pytest.mark.parametrize("kw", CASES, ids=["fp64", "tf32"])
def test_the_rejected_plan_leaves_the_device(limit, kw):
    m = dense(2300)
    s = solver(**kw)
    sym = s.Analyze(m)
    sym.device_handle()
    # what the smallest configuration's plan and factor hold
    limit(1 << 40)
    f = solver(DeviceMemoryBudget=least_budget(sym, **kw), **kw).Factorize(m, sym)
    least = limit(-1)
    del f
    gc.collect()
    sym = s.Analyze(m)   # (its plans are another set)
    sym.device_handle()
    limit(least)
    f = s.Factorize(m, sym)
    limit(-1)
    b = np.random.default_rng(1).uniform(-1.0, 1.0, m.Size)
    assert relative_residual(m, b, f.SolveRefined(b, tolerance=1e-12)) <= 1e-12
    # the larger configuration is taken again once it fits
    limit(1 << 40)
    g = s.Factorize(m, sym)
    assert limit(-1) > least
    assert relative_residual(m, b, g.SolveRefined(b, tolerance=1e-12)) <= 1e-12


def held_with_a_solve(limit, s, m, sym, b):
    """Bytes of a factor and the workspace of its solve."""
    limit(1 << 40)
    f = s.Factorize(m, sym)
    f._apply(b)
    return limit(-1)


@pytest.mark.parametrize("kw,n,nrhs", [(dict(Precision=Precision.FP64), 1300, 1200), (dict(Precision=Precision.TF32), 2300, 300)],
                         ids=["fp64", "tf32"])
@pytest.mark.parametrize("call", ["apply", "refined", "residual"])
def test_the_factor_makes_room_for_a_solve(limit, kw, n, nrhs, call):
    """The device holds the default factor, but its solve only beside the smallest one."""
    m = dense(n)
    s = solver(**kw)
    b = np.asfortranarray(np.random.default_rng(2).uniform(-1.0, 1.0, (n, nrhs)))
    sym = s.Analyze(m)
    small = solver(DeviceMemoryBudget=least_budget(sym, **kw), **kw)
    sym.device_handle()
    least = held_with_a_solve(limit, small, m, sym, b)
    sym = s.Analyze(m)
    sym.device_handle()
    limit(1 << 40)
    f = s.Factorize(m, sym)
    whole = limit(-1)
    extra = 16 * n * nrhs if call == "refined" else 0   # its own right-hand sides and solutions
    assert whole <= least + extra
    del f
    gc.collect()
    sym = s.Analyze(m)
    sym.device_handle()
    limit(least + extra)
    f = s.Factorize(m, sym)
    d = f.Diagonal.copy()
    if call == "apply":
        x = f._apply(b)
    elif call == "refined":
        x = f.SolveRefined(b, tolerance=1e-12)
    else:
        f.DeviceResidualNorms(b, b)
        x = f._apply(b)
    limit(-1)
    ref = small.Factorize(m, sym)
    if call != "refined":
        assert np.array_equal(x, ref._apply(b))   # the smallest configuration's, bit for bit
    assert relative_residual(m, b[:, 7], f.SolveRefined(b[:, 7], tolerance=1e-12)) <= 1e-12
    assert np.allclose(f.Diagonal, d, rtol=1e-3 if kw["Precision"] == Precision.TF32 else 1e-13, atol=0)
    f.Refactorize(m)
    assert np.array_equal(f._apply(b[:, :5]), ref._apply(b[:, :5]))


@pytest.mark.parametrize("kw", CASES, ids=["fp64", "tf32"])
def test_a_solve_that_does_not_fit_leaves_the_factor(limit, kw):
    m = dense(1300)
    s = solver(**kw)
    b = np.asfortranarray(np.random.default_rng(4).uniform(-1.0, 1.0, (1300, 400)))
    sym = s.Analyze(m)
    sym.device_handle()
    whole = held_with_a_solve(limit, s, m, sym, b[:, :17])
    sym = s.Analyze(m)
    sym.device_handle()
    limit(whole)
    f = s.Factorize(m, sym)
    x = f._apply(b[:, :3])
    with pytest.raises(DeviceOutOfMemoryError):
        f._apply(np.asfortranarray(np.tile(b, (1, 40))))
    for k in (3, 1, 17):   # what fits is solved as before
        y = f._apply(b[:, :k])
        if k == 3:
            assert np.array_equal(x, y)
    limit(-1)
    assert np.array_equal(y, s.Factorize(m, sym)._apply(b[:, :17]))


def test_a_factor_that_cannot_be_put_back_waits_for_room(limit):
    """The memory that the factor gives up goes to others (here: was not counted), so that neither a smaller factor nor the
    one before can be allocated: calls are refused while there is no room, and answered once there is."""
    m = dense(1300)
    s = solver()
    b = np.asfortranarray(np.random.default_rng(5).uniform(-1.0, 1.0, (1300, 50)))
    sym = s.Analyze(m)
    f, g, h = (s.Factorize(m, sym) for _ in range(3))
    x = g._apply(b)
    d = f.Diagonal.copy()
    limit(1 << 20)
    for call in (lambda: f._apply(b), lambda: f._apply(b[:, 0]), lambda: f.SolveRefined(b), lambda: f.DeviceResidualNorms(b, b),
                 lambda: f.Refactorize(m), lambda: h._apply(b)):
        with pytest.raises(DeviceOutOfMemoryError):
            call()
    assert np.array_equal(f.Diagonal, d)
    limit(-1)
    assert np.array_equal(f._apply(b), x)
    h.Refactorize(m)
    assert np.array_equal(h._apply(b), x)
    assert np.array_equal(g._apply(b), x)
