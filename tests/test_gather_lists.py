"""The lists of the children's entries that the forward solves read: counted by a device-memory budget, given up for it, and
without them (every front's vector gathered by a launch) the same sums in the same order."""
import gc

import numpy as np
import pytest

from magla_gb300 import (DeviceOutOfMemoryError, FillReducingOrdering, Precision, SymmetricUtduSolver, UtduSolverOptions)
from magla_gb300 import generators as G


def least_budget(sym, **kw):
    lo, hi = 1 << 10, 1 << 32
    while hi - lo > 1:
        mid = (lo + hi) // 2
        try:
            sym.EstimateDeviceBytes(UtduSolverOptions(DeviceMemoryBudget=mid, **kw))
            hi = mid
        except DeviceOutOfMemoryError:
            lo = mid
    return hi


# single-block fronts and inverse fronts; level kernels (no inverse fronts); fronts of up to one block only
@pytest.mark.gpu
@pytest.mark.parametrize("precision", [Precision.FP64, Precision.TF32])
@pytest.mark.parametrize("size,width", [((9, 9, 9, 2), 0), ((9, 9, 9, 2), -1), ((40, 40, 1, 1), 0)])
def test_without_the_lists(gpu_lib, precision, size, width):
    m = G.grid_matrix(*size)
    kw = dict(Precision=precision, InverseBlockWidth=width, Ordering=FillReducingOrdering.ApproximateMinimumDegree)
    solver = SymmetricUtduSolver(UtduSolverOptions(**kw))
    least = least_budget(solver.Analyze(m), **kw)
    b = np.random.default_rng(3).uniform(-1.0, 1.0, (m.Size, 17))
    held, x = [], []
    for budget in (0, least):
        sym = solver.Analyze(m)   # a device object, and plans, of its own
        sym.device_handle()
        gc.collect()
        gpu_lib.uchol_check_allocation_limit(1 << 40)
        f = SymmetricUtduSolver(UtduSolverOptions(DeviceMemoryBudget=budget, **kw)).Factorize(m, sym)
        held.append(gpu_lib.uchol_check_allocation_limit(-1))
        x.append([f._apply(np.asfortranarray(b[:, :k])) for k in (1, 5, 17)])
        del f
    assert held[1] < held[0]
    for a, c in zip(*x):
        assert np.array_equal(a, c)
