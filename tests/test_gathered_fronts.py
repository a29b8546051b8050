"""Fronts that read their children's and their ancestors' entries inside the solve kernels (up to 4096 rows), and larger
ones with launches of their own: three blocks of columns, each coupled to a common dense block and to none of the others,
so that the last front adds three children.  The matrix dominates its diagonal, so the solution is known to a few n u."""
import numpy as np
import pytest

from magla_gb300 import (FillReducingOrdering, Precision, SymmetricCSRMatrix, SymmetricUtduSolver,
                         UtduSolverOptions)


def _three_children(leaf, top):
    n = 3 * leaf + top
    rng = np.random.default_rng(n)
    i, j = [], []
    for k in range(3):
        a, b = np.triu_indices(leaf)
        i.append(a + k * leaf), j.append(b + k * leaf)
        i.append(np.repeat(np.arange(leaf) + k * leaf, top)), j.append(np.tile(np.arange(top) + 3 * leaf, leaf))
    a, b = np.triu_indices(top)
    i.append(a + 3 * leaf), j.append(b + 3 * leaf)
    i, j = np.concatenate(i), np.concatenate(j)
    v = rng.uniform(-1.0, 1.0, i.size)
    v[i == j] += n
    m = SymmetricCSRMatrix.from_triplets(n, i.astype(np.int32), j.astype(np.int32), v)
    x = rng.uniform(-1.0, 1.0, (n, 17))
    b = np.zeros((n, 17))
    for r in range(17):
        b[:, r] = np.bincount(i, v * x[j, r], n) + np.bincount(j, np.where(i == j, 0.0, v) * x[i, r], n)
    return m, x, b


# 3800 + 296 = 4096 rows: the largest front of the one kind, and one row more of the other; widths around the blocks'
@pytest.mark.gpu
@pytest.mark.parametrize("precision", [Precision.FP64, Precision.TF32])
@pytest.mark.parametrize("leaf,top", [(65, 130), (129, 64), (200, 1), (296, 3800), (297, 3800)])
def test_three_children(gpu_lib, precision, leaf, top):
    m, x, b = _three_children(leaf, top)
    n = x.shape[0]
    f = SymmetricUtduSolver(UtduSolverOptions(Precision=precision, Ordering=FillReducingOrdering.Natural)).Factorize(m)
    # the condition number is below 3 (Gershgorin: row sums of n uniform entries are about n / 2 around n)
    bound = 20 * n * 2.0 ** -53 * 3 if precision == Precision.FP64 else np.sqrt(n) * 2.0 ** -11 * 3
    for nrhs in (1, 5, 17):
        y = f.Solve(b[:, :nrhs]) if precision == Precision.FP64 else f._apply(np.asfortranarray(b[:, :nrhs]))
        assert np.max(np.abs(y - x[:, :nrhs])) <= bound
