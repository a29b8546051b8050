"""The inversion of the inverse fronts where the contribution arena is too small for its intermediate products: a budget
that holds everything else is met by forming them in their results' place, with the same sums."""
import numpy as np
import pytest

from magla_gb300 import (DeviceOutOfMemoryError, FillReducingOrdering, Precision, SymmetricCSRMatrix, SymmetricUtduSolver,
                         UtduSolverOptions)

NATURAL = FillReducingOrdering.Natural


def dense(n):
    rng = np.random.default_rng(n)
    G = rng.standard_normal((n, n + 8))
    A = G @ G.T / (n + 8) + np.eye(n)
    i, j = np.triu_indices(n)
    return A, SymmetricCSRMatrix.from_triplets(n, i.astype(np.int32), j.astype(np.int32), A[i, j])


def options(**kw):
    return UtduSolverOptions(Ordering=NATURAL, **kw)


def bare_budget(sym, m, kw):
    """Bytes of a factor of one dense front without the inversion's scratch, the gather lists and (FP64) the digits: panel,
    contribution, staging, pivots, two copies of the values and the inverse's blocks."""
    block, elem = (64, 8) if kw["Precision"] == Precision.FP64 else (128, 4)
    e = sym.EstimateDeviceBytes(options(**kw))
    staging = 0 if kw["Precision"] == Precision.FP64 else e["staging"]
    n, nb = m.Size, -(-m.Size // block)
    return (e["factor"] + e["contribution"] + staging + nb * (nb + 1) // 2 * block * block * elem +
            8 * (n + len(m.Values) + 2 * len(m.Values) - n))


CASES = [(dict(Precision=Precision.FP64), 700), (dict(Precision=Precision.FP64), 1987), (dict(Precision=Precision.TF32), 1300),
         (dict(Precision=Precision.TF32), 515)]


@pytest.mark.parametrize("kw,n", CASES)
def test_the_scratch_gives_way(kw, n):
    _, m = dense(n)
    sym = SymmetricUtduSolver(options(**kw)).Analyze(m)
    least = bare_budget(sym, m, kw)
    sym.EstimateDeviceBytes(options(DeviceMemoryBudget=least, **kw))
    with pytest.raises(DeviceOutOfMemoryError):
        sym.EstimateDeviceBytes(options(DeviceMemoryBudget=least - 1, **kw))


@pytest.mark.gpu
@pytest.mark.parametrize("kw,n", CASES)
def test_in_place(gpu_lib, kw, n):
    A, m = dense(n)
    s = SymmetricUtduSolver(options(**kw))
    b = np.random.default_rng(n).uniform(-1, 1, (n, 5))
    least = bare_budget(s.Analyze(m), m, kw)
    f = SymmetricUtduSolver(options(DeviceMemoryBudget=least, **kw)).Factorize(m)
    x = f._apply(b)
    if kw["Precision"] == Precision.TF32:   # one application of the factor; the scratch alone differs
        assert np.array_equal(x, s.Factorize(m)._apply(b))
    else:
        ref = np.linalg.solve(A, b)   # backward stable to a few n u; the condition number is below 6
        assert np.max(np.abs(x - ref)) <= 20 * n * 2.0 ** -53 * 6 * np.max(np.abs(ref))
