"""Inverses of the diagonal blocks and of the inverse fronts' diagonal blocks: dense matrices, whose factor is one
front of n columns, at the edges of the blocks (64 columns in FP64, 128 in the mixed path), of the 16-column
sub-blocks and of the doubling rounds.  A wrong inverse shows in the solution at once."""
import numpy as np
import pytest

from magla_gb300 import Precision, SymmetricCSRMatrix, SymmetricUtduSolver, UtduSolverOptions

pytestmark = pytest.mark.gpu


def dense_spd(n, seed):
    rng = np.random.default_rng(seed)
    G = rng.standard_normal((n, n + 8))
    A = G @ G.T / (n + 8) + np.eye(n)
    i, j = np.triu_indices(n)
    return A, SymmetricCSRMatrix.from_triplets(n, i.astype(np.int32), j.astype(np.int32), A[i, j])


@pytest.mark.parametrize("mask", [1, 0x1f])   # blocked fronts from 33 rows on; fronts up to 160 rows by one CTA
@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 32, 33, 48, 63, 64, 65, 100, 127, 128, 129, 160, 161])
def test_fp64_blocks(gpu_lib, n, mask):
    A, m = dense_spd(n, n)
    b = np.random.default_rng(n + 1).uniform(-1, 1, (n, 3))
    x = SymmetricUtduSolver(UtduSolverOptions(SmallFrontBuckets=mask)).Factorize(m).Solve(b)
    ref = np.linalg.solve(A, b)
    # both solves are backward stable to a few n u; the condition number is below 6
    assert np.max(np.abs(x - ref)) <= 20 * n * 2.0 ** -53 * 6 * np.max(np.abs(ref))


@pytest.mark.parametrize("precision,block", [(Precision.FP64, 64), (Precision.TF32, 128)])
@pytest.mark.parametrize("blocks", [2, 3, 4, 5, 8, 9, 13])
def test_inverse_fronts_by_halves(gpu_lib, precision, block, blocks):
    """Whole and ragged numbers of blocks; the same system without inverse fronts takes the chain of block solves."""
    n = block * blocks - 5
    A, m = dense_spd(n, blocks)
    b = np.random.default_rng(blocks).uniform(-1, 1, n)
    ref = np.linalg.solve(A, b)
    for width in (0, -1):
        f = SymmetricUtduSolver(UtduSolverOptions(Precision=precision, InverseBlockWidth=width)).Factorize(m)
        if precision == Precision.FP64:
            assert np.max(np.abs(f.Solve(b) - ref)) <= 20 * n * 2.0 ** -53 * 6 * np.max(np.abs(ref))
        else:
            # one application of the TF32 factor: operands rounded to 2^-11, sums of up to n of them
            x = f._apply(b)
            assert np.max(np.abs(x - ref)) <= np.sqrt(n) * 2.0 ** -11 * 6 * np.max(np.abs(ref))


@pytest.mark.parametrize("width", [64, 128])
def test_outer_block_of_64_columns(gpu_lib, width):
    """Outer blocks narrower than the solves' blocks keep their inverses in the workspace."""
    A, m = dense_spd(420, 3)
    b = np.random.default_rng(9).uniform(-1, 1, 420)
    f = SymmetricUtduSolver(UtduSolverOptions(Precision=Precision.TF32, BlockWidth=width)).Factorize(m)
    assert np.max(np.abs(f._apply(b) - np.linalg.solve(A, b))) <= np.sqrt(420) * 2.0 ** -11 * 6 * np.max(np.abs(b))
