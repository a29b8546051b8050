"""Tensor-core updates by row tiles of 64 and 128 rows, which launches of up to one tile an SM take, against the FP64
product of the same operands, with the bounds of the 256-row tiles."""
import ctypes as C

import numpy as np
import pytest

from magla_gb300 import _native
from magla_gb300.errors import raise_for_status
from tests.test_kernel_checks import BF16_U, TF32_U, bf16_round, check_update

pytestmark = pytest.mark.gpu


# one column; one column tile; ragged columns and rows with a K range inside the operands; contribution columns, by one
# CTA a tile and by three CTAs in all; K long enough to be split
@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("rows", [64, 128])
@pytest.mark.parametrize("m,w,c0,cend,kbeg,kn,max_ctas", [(129, 129, 0, 1, 0, 64, 0), (640, 640, 128, 256, 0, 128, 0),
                                                          (577, 400, 256, 400, 128, 70, 0), (703, 300, 300, 703, 0, 300, 0),
                                                          (703, 300, 300, 703, 0, 300, 3), (450, 450, 320, 448, 0, 2112, 0)])
def test_narrow_row_tiles(gpu_lib, bf16, rows, m, w, c0, cend, kbeg, kn, max_ctas):
    ld = -(-(kbeg + kn) // 64) * 64
    rng = np.random.default_rng(m + rows)
    front = np.asfortranarray(np.tril(rng.uniform(-1.0, 1.0, (m, m))).astype(np.float32))
    W, L = (rng.uniform(-1.0, 1.0, (m, ld)).astype(np.float32) for _ in range(2))
    W[:, kbeg + kn:] = 0.0
    L[:, kbeg + kn:] = 0.0
    out = np.zeros((m, m), np.float32, order="F")
    tiles, split = C.c_int64(), C.c_int()
    lib = _native.gpu()
    st = lib.uchol_check_schur_update_rows(rows, int(bf16), m, w, c0, cend, kbeg, kn, front.ctypes.data, W.ctypes.data,
                                           L.ctypes.data, ld, max_ctas, out.ctypes.data, C.byref(tiles), C.byref(split))
    raise_for_status(st, lib.uchol_last_error())
    assert tiles.value == sum(-(-(m - c) // rows) for c in range(c0, cend, 128))
    assert split.value == (kn > 2000)
    Wr, Lr = (bf16_round(W), bf16_round(L)) if bf16 else (W, L)
    Wk, Lk = (X[:, kbeg:kbeg + kn].astype(np.float64) for X in (Wr, Lr))
    ref = front.astype(np.float64)
    ref[:, c0:cend] -= Wk @ Lk[c0:cend].T
    check_update(front, out, ref, np.abs(Wk) @ np.abs(Lk[c0:cend]).T, c0, cend, BF16_U if bf16 else TF32_U)
