"""FP64 fronts whose updates run on the tensor cores from 8-bit digits: dense matrices (one front), at the edges of the
digit chunks, tiles and super-blocks, with rows of very different scale, and with a row whose entries span many
exponents."""
import numpy as np
import pytest

from magla_gb300 import SymmetricCSRMatrix, SymmetricUtduSolver, UtduSolverOptions

pytestmark = pytest.mark.gpu


def dense(A):
    n = A.shape[0]
    i, j = np.triu_indices(n)
    return SymmetricCSRMatrix.from_triplets(n, i.astype(np.int32), j.astype(np.int32), A[i, j])


def cholesky_error(m, A, S):
    """max |(L D L^T - P A P^T)_ij| / sqrt(a_ii a_jj) by way of the solution of n columns: the residual of S^-1 A S^-1
    scaled systems, in units of the unit roundoff."""
    f = SymmetricUtduSolver(UtduSolverOptions(PivotTolerance=0.0)).Factorize(m)   # rows may be far below the largest
    rng = np.random.default_rng(0)
    b = S[:, None] * rng.uniform(-1, 1, (A.shape[0], 3))
    x = f.Solve(b)
    As = A / S[:, None] / S[None, :]
    xs = S[:, None] * x
    r = b / S[:, None] - As @ xs
    return f, np.max(np.linalg.norm(r, axis=0) / (np.linalg.norm(As, 2) * np.linalg.norm(xs, axis=0)))


@pytest.mark.parametrize("n", [383, 384, 385, 512, 640, 1024, 1025, 1087, 1151, 1153, 1300, 1537, 1700])
@pytest.mark.parametrize("decades", [0, 12])
def test_dense_fronts(gpu_lib, n, decades):
    rng = np.random.default_rng(n)
    G = rng.standard_normal((n, n + 8))
    C = G @ G.T / (n + 8) + 0.1 * np.eye(n)
    S = 10.0 ** rng.uniform(0, decades, n)   # (construction drops entries up to 1e-15)
    A = C * S[:, None] * S[None, :]
    A = (A + A.T) / 2
    f, err = cholesky_error(dense(A), A, S)
    # a backward stable factorisation and two substitutions: below 3 n u with a modest constant, sqrt(n) in practice
    assert err <= 8 * np.sqrt(n) * 2.0 ** -53
    assert f.RegularizedPivotCount == 0 and f.NegativePivotCount == 0
    # the pivots against an FP64 factorisation of the same (natural up to the order's permutation) matrix
    p = f.Symbolic.Permutation
    L = np.linalg.cholesky(C[np.ix_(p, p)])
    d = f.Diagonal / S[p] ** 2
    assert np.max(np.abs(d - np.diag(L) ** 2) / d) <= 100 * n * 2.0 ** -53


def test_entries_of_many_exponents(gpu_lib):
    """Off-diagonal entries from 1 to 1e-30 of their row's largest: the digits drop what FP64 sums drop."""
    n = 1200
    rng = np.random.default_rng(5)
    E = 10.0 ** -rng.uniform(0, 30, (n, n)) * rng.choice([-1.0, 1.0], (n, n))
    A = np.triu(E, 1)
    A = A + A.T
    A[np.arange(n), np.arange(n)] = np.sum(np.abs(A), axis=1) + 1.0
    S = np.sqrt(np.diag(A))
    _, err = cholesky_error(dense(A), A, S)
    assert err <= 8 * np.sqrt(n) * 2.0 ** -53


def test_not_finite_values_stay_visible(gpu_lib):
    n = 1100
    m = dense(np.eye(n) * 4.0 + 0.001)
    m.Values[7] = np.nan   # (construction drops entries that are not numbers)
    f = SymmetricUtduSolver(UtduSolverOptions()).Factorize(m)
    x = f.Solve(np.ones(n))
    assert not np.all(np.isfinite(x)) or f.RegularizedPivotCount > 0
