"""A device-memory budget that default choices made for speed alone exceed (wide inverse fronts, the digits of the FP64
tensor-core updates) is met without them: nothing that fits without them is refused (host-side plans, no GPU)."""
import numpy as np
import pytest

from magla_gb300 import (DeviceOutOfMemoryError, FillReducingOrdering, Precision, SymmetricCSRMatrix, SymmetricUtduSolver,
                         UtduSolverOptions)


def accepted(sym, budget, **kw):
    try:
        return sym.EstimateDeviceBytes(UtduSolverOptions(Ordering=FillReducingOrdering.Natural, DeviceMemoryBudget=budget, **kw))
    except DeviceOutOfMemoryError:
        return None


def smallest(sym, lo, hi, **kw):
    while hi - lo > 1 << 16:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if accepted(sym, mid, **kw) else (mid, hi)
    return hi


@pytest.fixture(scope="module")
def dense_symbolic():
    n = 2300
    i, j = np.triu_indices(n)
    v = np.where(i == j, 2.0 * n, 1.0)
    m = SymmetricCSRMatrix.from_triplets(n, i.astype(np.int32), j.astype(np.int32), v)
    return SymmetricUtduSolver(UtduSolverOptions(Ordering=FillReducingOrdering.Natural)).Analyze(m)


def test_wide_inverse_fronts_give_way(dense_symbolic):
    kw = dict(Precision=Precision.TF32)
    explicit = smallest(dense_symbolic, 1 << 20, 1 << 32, InverseBlockWidth=2048, **kw)
    assert accepted(dense_symbolic, explicit, **kw) is not None
    assert smallest(dense_symbolic, 1 << 20, 1 << 32, **kw) <= explicit + (1 << 16)


def test_digits_give_way(dense_symbolic):
    free = accepted(dense_symbolic, 0)
    least = smallest(dense_symbolic, 1 << 20, 1 << 32)
    assert free["staging"] > 0 and accepted(dense_symbolic, least)["staging"] == 0
    assert least < free["factor"] + free["contribution"] + free["staging"]
