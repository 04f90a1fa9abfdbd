"""Products and windows of many short rows (a lane a row): entry counts around
the lane's eight, the warp's and the CTA's limits, alone in their warp and
next to one another, with B rows that are empty."""
import numpy as np
import pytest

import dbd_gb300 as dbd
import oracle

pytestmark = pytest.mark.gpu
SPECIAL = [0, 7, 8, 9, 15, 16, 17, 63, 64, 65, 66, 255, 256, 257, 300]


@pytest.mark.parametrize("rows", [(1 << 19) - 1, 1 << 19, (1 << 19) + 37])
@pytest.mark.parametrize("together", [False, True])
def test_row_products(rows, together):
    rng = np.random.default_rng(rows)
    inner, cols = 512, 700
    lens = rng.integers(0, 3, rows)
    at = np.arange(len(SPECIAL)) if together else np.linspace(31, rows - 1, len(SPECIAL)).astype(int)
    lens[at] = SPECIAL
    ptr = np.r_[0, np.cumsum(lens)].astype(np.int32)
    # Ascending distinct columns: a start and steps of one.
    start = rng.integers(0, inner - lens + 1)
    idx = (np.repeat(start - ptr[:-1], lens) + np.arange(ptr[-1])).astype(np.int32)
    A = dbd.CSR(rows, inner, ptr, idx, rng.integers(-3, 4, idx.size).astype(np.float64))
    blen = rng.integers(0, 3, inner)
    bptr = np.r_[0, np.cumsum(blen)].astype(np.int32)
    bidx = np.concatenate([np.sort(rng.choice(cols, n, replace=False)) for n in blen]).astype(np.int32)
    B = dbd.CSR(inner, cols, bptr, bidx, rng.integers(-3, 4, bidx.size).astype(np.float64))
    with dbd.Context(cpu_gib=4, gpu_gib=8) as ctx:
        res = ctx.spgemm(A, B)
    assert res.stats["products"] == int(blen[idx].sum())
    Cp, Ci, Cv = oracle.spgemm(A, B)[:3]
    np.testing.assert_array_equal(res.C.row_ptr, Cp)
    np.testing.assert_array_equal(res.C.col_idx, Ci)
    np.testing.assert_array_equal(res.C.val, Cv)  # whole numbers: exact in any order
