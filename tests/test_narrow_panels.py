"""Rows below an outer block by tiles of 64: the same products in the same order as by tiles of 128, so the same bits."""
import ctypes as C

import numpy as np
import pytest

from magla_gb300 import _native
from magla_gb300.errors import raise_for_status

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,nb", [(129, 128), (128 + 63, 128), (128 + 64, 128), (128 + 65, 128), (517, 96), (400, 1), (261, 33)])
def test_panel_tiles_agree(gpu_lib, m, nb):
    rng = np.random.default_rng(m)
    G = rng.standard_normal((m, m + 8))
    A = np.asfortranarray((G @ G.T / (m + 8) + np.eye(m))[:, :nb].astype(np.float32))
    lib = _native.gpu()
    results = []
    for rows in (128, 64):
        L, W = (np.zeros((m, nb), np.float32, order="F") for _ in range(2))
        D, counts = np.zeros(nb), (C.c_int * 3)()
        st = lib.uchol_check_diag_panel_rows(rows, m, nb, A.ctypes.data, 0.0, 0.0, 0, L.ctypes.data, D.ctypes.data,
                                             W.ctypes.data, counts)
        raise_for_status(st, lib.uchol_last_error())
        results.append((L, W, D, list(counts)))
    assert all(np.array_equal(a, b) for a, b in zip(*results))
    L64 = np.linalg.cholesky(A[:nb].astype(np.float64) if nb > 1 else A[:1].astype(np.float64))
    W64 = np.linalg.solve(L64 / np.diag(L64), A[nb:].astype(np.float64).T).T
    assert np.max(np.abs(results[1][0][nb:] * D - W64)) <= 1e-4 * max(1.0, np.max(np.abs(W64)))
