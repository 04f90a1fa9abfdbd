"""Dense rows (windows of more than 2^18 columns): spans around the kernel's
windows of 16384 words and its groups of 128 and 256 words, thin and full
rows."""
import numpy as np
import pytest

import dbd_gb300 as dbd
import oracle

pytestmark = pytest.mark.gpu
DENSE = 8


@pytest.mark.parametrize("words", [8193, 8319, 16257, 16383, 16384, 16385, 16513, 32768, 32769])
@pytest.mark.parametrize("entries", [4200, 70000])
def test_wide_windows(words, entries):
    rng = np.random.default_rng(words + entries)
    lo, hi = 32 + 19, 32 * words + 31 - 3  # words 1 .. words
    # A full stretch at the window's end, the rest thin.
    run = np.arange(max(lo, hi - entries // 2), hi + 1)
    pool = np.unique(np.r_[lo, lo + rng.choice(hi - lo, entries - run.size, replace=False), run])
    part = rng.integers(0, 3, pool.size)
    rows = [pool[(part == q) | ((part == (q + 1) % 3) & (rng.random(pool.size) < 0.3))] for q in range(3)]
    ptr = np.cumsum([0] + [r.size for r in rows]).astype(np.int32)
    idx = np.concatenate(rows).astype(np.int32)
    B = dbd.CSR(3, hi + 2, ptr, idx, rng.standard_normal(idx.size))
    A = dbd.CSR(2, 3, np.array([0, 3, 6], np.int32), np.array([0, 1, 2, 2, 0, 1], np.int32), rng.standard_normal(6))
    with dbd.Context(cpu_gib=1, gpu_gib=8) as ctx:
        res = ctx.spgemm(A, B)
    assert res.stats["rows_per_bin"][DENSE] == 2
    Cp, Ci, Cv, Ca = oracle.spgemm(A, B, with_abs=True)
    np.testing.assert_array_equal(res.C.row_ptr, Cp)
    np.testing.assert_array_equal(res.C.col_idx, Ci)
    assert np.all(np.abs(res.C.val - Cv) <= 1e-12 * Ca)
