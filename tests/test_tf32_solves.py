"""The FP32 solve kernels of the mixed path, held to bounds that a missing block or child cannot pass: fronts that add three
children (at the 4096 rows where their vectors get launches of their own), coupled as strongly as the matrix allows, and inverse
fronts against the chain of block solves with the same factor.  The tests without a GPU plant the mistakes in the matrices."""
import numpy as np
import pytest

from magla_gb300 import FillReducingOrdering, Precision, SymmetricCSRMatrix, SymmetricUtduSolver, UtduSolverOptions

NATURAL = FillReducingOrdering.Natural
U = 2.0 ** -11   # TF32 operands, rounded to nearest


def dense_part(rng, n):
    """I + R, |R| of about 0.1 (entries of variance 0.05^2 / n: the norm of such a matrix is twice 0.05, far from 0.2)."""
    R = rng.uniform(-1.0, 1.0, (n, n)) * 0.05 * np.sqrt(3.0 / n)
    return np.eye(n) + np.triu(R) + np.triu(R, 1).T


def three_children(leaf, top):
    """Three blocks of columns, each coupled to a common block; the coupling's norm is 0.4: no eigenvalue below 0.4."""
    n, k = 3 * leaf + top, 3 * leaf
    rng = np.random.default_rng(n)
    A = np.zeros((n, n))
    for c in range(3):
        A[c * leaf:(c + 1) * leaf, c * leaf:(c + 1) * leaf] = dense_part(rng, leaf)
    A[k:, k:] = dense_part(rng, top)
    C = rng.uniform(-1.0, 1.0, (k, top))
    C *= 0.4 / np.linalg.norm(C, 2)
    A[:k, k:], A[k:, :k] = C, C.T
    return A, rng.uniform(-1.0, 1.0, (n, 17))


def bound(A, x):
    """Eight standard deviations of the largest error of x.  Every operand of an update, l_ik or l_ik d_k below the diagonal, is
    off by an independent U / sqrt 3 of itself at most; with G the Cholesky factor below its diagonal, s_i and t_k the deviations
    of the residual's two parts (roundings of row i; of column k's rows j), |A^-1| <= 1 / 0.4 and |G^-T| <= 0.4^-1/2.  FP32
    sums of n terms come on top."""
    G = np.tril(np.linalg.cholesky(A), -1)
    s = np.sqrt(np.max((G * G) @ (G.T @ x) ** 2))
    t = np.sqrt(np.max((G * G).T @ x ** 2))
    return 8 * U / np.sqrt(3) * np.hypot(s / 0.4, t / np.sqrt(0.4)) + 8 * np.sqrt(len(A)) * 2.0 ** -24 / 0.4


SIZES = [(65, 130), (129, 64), (200, 1), (296, 3800), (297, 3800)]


@pytest.mark.parametrize("leaf,top", SIZES)
def test_the_bound_sees_a_missing_child(leaf, top):
    A, x = three_children(leaf, top)
    k = 3 * leaf
    b = A @ x
    S = A[k:, k:] - A[k:, :k] @ np.linalg.solve(A[:k, :k], A[:k, k:])
    y = np.linalg.solve(A[:k, :k], b[:k])
    tol = bound(A, x)
    for c in range(3):   # the forward entries of child c never reach the common block
        y1 = y.copy()
        y1[c * leaf:(c + 1) * leaf] = 0.0
        z = np.linalg.solve(S, b[k:] - A[k:, :k] @ y1)
        error = np.max(np.abs(z - x[k:]), axis=0)
        for nrhs in (1, 5, 17):
            assert np.max(error[:nrhs]) > 3 * tol


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [Precision.TF32, Precision.FP64])
@pytest.mark.parametrize("leaf,top", SIZES)
def test_three_children(gpu_lib, precision, leaf, top):
    A, x = three_children(leaf, top)
    i, j = np.nonzero(np.triu(A))
    m = SymmetricCSRMatrix.from_triplets(len(A), i.astype(np.int32), j.astype(np.int32), A[i, j])
    b = A @ x
    f = SymmetricUtduSolver(UtduSolverOptions(Precision=precision, Ordering=NATURAL)).Factorize(m)
    tol = bound(A, x) if precision == Precision.TF32 else 20 * len(A) * 2.0 ** -53 / 0.4
    for nrhs in (1, 5, 17):
        assert np.max(np.abs(f._apply(np.asfortranarray(b[:, :nrhs])) - x[:, :nrhs])) <= tol


def dense_spd(n, seed):
    rng = np.random.default_rng(seed)
    G = rng.standard_normal((n, n + 8))
    A = G @ G.T / (n + 8) + np.eye(n)   # condition number below 6
    return A, rng.uniform(-1.0, 1.0, (n, 5))


BLOCKS = [2, 3, 4, 5, 8, 9, 13]


def inverse_bound(n, ref):
    """Two solves in FP32 with one factor, each within n u times the condition number (6) of its exact solution."""
    return 2 * 6 * n * 2.0 ** -24 * np.max(np.abs(ref))


@pytest.mark.parametrize("blocks", BLOCKS)
def test_the_bound_sees_a_missing_block(blocks):
    n = 128 * blocks - 5
    A, b = dense_spd(n, blocks)
    L = np.linalg.cholesky(A)
    X = np.linalg.inv(L)
    ref = np.linalg.solve(A, b)
    for i in range(1, blocks):
        for j in range(i):
            bad = X.copy()
            bad[128 * i:128 * (i + 1), 128 * j:128 * (j + 1)] = 0.0
            assert np.max(np.abs(X.T @ (bad @ b) - ref)) > 3 * inverse_bound(n, ref)
            assert np.max(np.abs(bad.T @ (X @ b) - ref)) > 3 * inverse_bound(n, ref)


@pytest.mark.gpu
@pytest.mark.parametrize("blocks", BLOCKS)
def test_inverse_fronts_and_block_solves_agree(gpu_lib, blocks):
    n = 128 * blocks - 5
    A, b = dense_spd(n, blocks)
    i, j = np.triu_indices(n)
    m = SymmetricCSRMatrix.from_triplets(n, i.astype(np.int32), j.astype(np.int32), A[i, j])
    ref = np.linalg.solve(A, b)
    f, g = (SymmetricUtduSolver(UtduSolverOptions(Precision=Precision.TF32, Ordering=NATURAL, InverseBlockWidth=w)).Factorize(m)
            for w in (0, -1))
    assert np.array_equal(f.Diagonal, g.Diagonal)   # one factor
    for nrhs in (1, 5):
        c = np.asfortranarray(b[:, :nrhs])
        assert np.max(np.abs(f._apply(c) - g._apply(c))) <= inverse_bound(n, ref)
