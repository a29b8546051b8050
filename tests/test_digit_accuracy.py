"""Entries of the FP64 update from 8-bit digits (uchol_check_digit_update) against the same sums in extended precision, for
rows of one large entry, in a column of its own choice, and others 2^-g of it."""
import numpy as np
import pytest

from magla_gb300 import _native
from magla_gb300.errors import raise_for_status

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def digit_update(front, pivots, w, c0, cend, kbeg, kn):
    lib = _native.gpu()
    m = front.shape[0]
    front, out = np.asfortranarray(front), np.zeros((m, m), order="F")
    pivots = np.ascontiguousarray(pivots)
    st = lib.uchol_check_digit_update(m, w, c0, cend, kbeg, kn, front.ctypes.data, pivots.ctypes.data, out.ctypes.data)
    raise_for_status(st, lib.uchol_last_error())
    return out


def graded_front(m, w, g, seed):
    """Unit L times the pivots' square roots: entries of about 2^-g, one a row and block of 128 columns of about 1; C of the
    size of those products."""
    rng = np.random.default_rng(seed)
    X = rng.uniform(0.5, 1.0, (m, w)) * rng.choice([-1.0, 1.0], (m, w)) * 2.0 ** -g
    for k in range(0, w, 128):
        X[np.arange(m), k + rng.integers(0, min(128, w - k), m)] *= 2.0 ** g
    pivots = 10.0 ** rng.uniform(-3, 3, w)
    front = np.tril(rng.uniform(-1.0, 1.0, (m, m)) * 2.0 ** -g)
    front[:, :w] = np.tril(X / np.sqrt(pivots))
    return front, pivots, X


# one chunk; ragged columns and rows; a super-block's first columns; a K range inside the panel; one tile in all
SHAPES = [(300, 128, 128, 300, 0, 128), (517, 300, 300, 517, 0, 300), (700, 650, 384, 650, 0, 384),
          (900, 700, 640, 700, 512, 128), (65, 64, 64, 65, 0, 64)]


@pytest.mark.parametrize("m,w,c0,cend,kbeg,kn", SHAPES)
@pytest.mark.parametrize("g", [0, 4, 7, 16])
def test_entries_of_graded_rows(gpu_lib, m, w, c0, cend, kbeg, kn, g):
    front, pivots, _ = graded_front(m, w, g, m + g)
    out = digit_update(front, pivots, w, c0, cend, kbeg, kn)
    K = np.arange(kbeg, kbeg + kn)
    L, W = front[:, K], front[:, K] * pivots[K]
    lower = np.tril(np.ones((m, m), bool))
    lower[:, :c0] = lower[:, cend:] = False
    assert np.array_equal(out[~lower], front[~lower])
    ext = np.longdouble
    ref = front.astype(ext) - (L.astype(ext) * pivots[K]) @ L.astype(ext).T
    size = np.abs(L) @ np.abs(W).T
    # what the digits leave out: a column scaled by s (L) and 1 / s (W), about sqrt(d); the largest scaled entries of a row
    # and chunk are at least half of their power of two, the mean loss of random digits is 2^-60.7 of the powers' product,
    # and no entry of these fronts is more than five times the mean (10^5 of them): 2^(2 - 60.7 + 2.3) < 2^-56
    s = 2.0 ** ((((pivots[K].view(np.int64) >> 52) & 0x7ff) - 1023) >> 1)
    loss = np.zeros((m, m))
    for k in range(0, kn, 128):
        a, b = (np.max(np.abs(x[:, k:k + 128]), axis=1) for x in (L * s, W / s))
        loss += 2.0 ** -56 * a[:, None] * b[None, :]
    chunks = -(-kn // 128)
    # FP64 roundings: W, every chunk's sum, their additions, the subtraction from C
    bound = loss + U * ((chunks + 2) * size + np.abs(front) + np.abs(ref).astype(float))
    err = np.abs((out - ref).astype(float))
    assert np.all(err[lower] <= bound[lower]), f"{np.max((err / bound)[lower]):.2f}"
    if g <= 7 and kn > 1:
        # no less accurate than the sums on the FP64 pipe: 32 columns at a time, each subtracted from C
        plain = front.copy()
        for k in range(0, kn, 32):
            plain -= L[:, k:k + 32] @ W[:, k:k + 32].T
        fp64 = np.abs((plain - ref).astype(float))
        rms = [float(np.sqrt(np.mean((e[lower] / (size[lower] + 1e-300)) ** 2))) for e in (err, fp64)]
        if lower.sum() > 1000:   # (a mean of enough entries)
            assert rms[0] <= rms[1], rms


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("where", ["row", "column", "pivot"])
def test_not_finite_entries_reach_their_rows_and_columns_only(gpu_lib, value, where):
    """A staged entry that is not finite makes its row's and its column's entries of C NaN, a pivot every one; all others are
    those of the finite front."""
    m, w, c0, cend, kbeg, kn = 420, 300, 300, 420, 0, 300
    front, pivots, _ = graded_front(m, w, 0, 8)
    clean = digit_update(front, pivots, w, c0, cend, kbeg, kn)
    i, k = (330, 200) if where == "row" else (419, 17)   # in the middle of a tile; the last row, the first chunk
    if where == "pivot":
        pivots[k] = value
    else:
        front[i, k] = value
    out = digit_update(front, pivots, w, c0, cend, kbeg, kn)
    rows, cols = np.tril_indices(m)
    hit = np.zeros((m, m), bool)
    updated = (cols >= c0) & (cols < cend)
    reached = updated & ((rows == i) | (cols == i) | (where == "pivot"))
    hit[rows[reached], cols[reached]] = True
    low = np.tril(np.ones((m, m), bool))
    low[:, :w] = False
    assert np.all(np.isnan(out[hit])) and hit.sum() > 0
    assert np.array_equal(out[low & ~hit], clean[low & ~hit])


@pytest.mark.parametrize("exponent", [-1000, -1021, -1030])
def test_subnormal_products(gpu_lib, exponent):
    """Pivots at the lower end of the range: products l d, and entries of C, that are subnormal count like any others."""
    m, w, c0, cend, kbeg, kn = 300, 200, 200, 300, 0, 200
    rng = np.random.default_rng(-exponent)
    front = np.tril(rng.uniform(-1.0, 1.0, (m, m)) * 2.0 ** exponent)
    front[:, :w] = np.tril(rng.uniform(0.5, 1.0, (m, w)) * 2.0 ** -rng.integers(0, 30, (m, w)))
    pivots = rng.uniform(1.0, 2.0, w) * 2.0 ** exponent
    out = digit_update(front, pivots, w, c0, cend, kbeg, kn)
    ext = np.longdouble
    L = front[:, :kn]
    ref = front.astype(ext) - (L.astype(ext) * pivots) @ L.astype(ext).T
    size = np.abs(L) @ np.abs(L * pivots).T
    # the digits' loss (test_entries_of_graded_rows) against rows whose largest entry is at most 1, sqrt(d) being in both, and
    # roundings to the smallest subnormal: each product l d, each chunk's sum (twice) and addition, the subtraction
    tiny = 2.0 ** -1074
    bound = 2 * 2.0 ** (exponent + 1 - 56) + U * (4 * size + np.abs(front) + np.abs(ref).astype(float)) + (kn + 8) * tiny
    lower = np.tril(np.ones((m, m), bool))
    lower[:, :c0] = False
    assert np.all(np.abs((out - ref).astype(float))[lower] <= bound[lower])
