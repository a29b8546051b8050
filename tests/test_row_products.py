"""The both-triangle product at the edges of its row handling: rows of one entry, of eight and nine (a lane group's
width), of the longest that a lane group takes and one more (a whole warp), and groups of right-hand sides."""
import numpy as np
import pytest

from magla_gb300 import DeviceSymmetricCSRMatrix, SymmetricCSRMatrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first_row", [1, 8, 9, 512, 513, 700])
@pytest.mark.parametrize("nrhs", [1, 3, 4, 5])
def test_row_lengths(gpu_lib, first_row, nrhs):
    n = 703
    rng = np.random.default_rng(first_row)
    rows = np.concatenate([np.arange(n), np.zeros(first_row - 1, int), np.arange(5, n - 1)]).astype(np.int32)
    cols = np.concatenate([np.arange(n), np.arange(1, first_row), np.arange(6, n)]).astype(np.int32)
    m = SymmetricCSRMatrix.from_triplets(n, rows, cols, rng.uniform(0.5, 1.5, len(rows)))
    x = rng.uniform(-1, 1, (n, nrhs))
    y = DeviceSymmetricCSRMatrix(m).Multiply(x)
    ref = m.to_dense() @ x
    # each sum: at most first_row + 2 terms below 1.5 in magnitude
    assert np.max(np.abs(y - ref)) <= 2 * (first_row + 2) * 2.0 ** -53 * 1.5 * (first_row + 2)
