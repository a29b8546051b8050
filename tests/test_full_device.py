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
