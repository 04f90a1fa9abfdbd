"""Long runs of columns in narrow rows, whose products few rows take six steps
at a time: run lengths around the groups, and row counts on both sides of where
the groups end (16 rows an SM).  Every row sums in A's entry order either way:
values within 1e-12 * sum |terms|, the same bits from both."""
import numpy as np
import pytest

import dbd_gb300 as dbd
import oracle

pytestmark = pytest.mark.gpu
DENSEW = 9
LAST_FEW = 16 * 152


def _runs(starts, length, n_cols, seed):
    k = len(starts)
    idx = (np.asarray(starts)[:, None] + np.arange(length)).astype(np.int32).ravel()
    return dbd.CSR(k, n_cols, (np.arange(k + 1) * length).astype(np.int32), idx,
                   np.random.default_rng(seed).standard_normal(idx.size))


@pytest.mark.parametrize("length", [95, 96, 191, 192, 193, 223, 224, 225, 384, 400])
@pytest.mark.parametrize("step", [0, 1, 3])
def test_long_runs(length, step):
    entries = 34
    B = _runs(5 + step * np.arange(entries), length, 512, 1)
    rng = np.random.default_rng(2)
    few, many = 7, LAST_FEW + 1
    rows = [np.sort(rng.choice(entries, e, replace=False)) for e in (entries, entries, 33, 32, 31, 5, 1)]
    got = {}
    for m in (few, LAST_FEW, many):
        use = [rows[r % few] for r in range(m)]
        vals = [np.random.default_rng(10 + r % few).standard_normal(rows[r % few].size) for r in range(m)]
        A = dbd.CSR(m, entries, np.r_[0, np.cumsum([r.size for r in use])].astype(np.int32),
                    np.concatenate(use).astype(np.int32), np.concatenate(vals))
        with dbd.Context(cpu_gib=1, gpu_gib=4) as ctx:
            res = ctx.spgemm(A, B)
        assert res.stats["rows_per_bin"][DENSEW] == m
        if m == few:
            Cp, Ci, Cv, Ca = oracle.spgemm(A, B, with_abs=True)
            np.testing.assert_array_equal(res.C.row_ptr, Cp)
            np.testing.assert_array_equal(res.C.col_idx, Ci)
            assert np.all(np.abs(res.C.val - Cv) <= 1e-12 * Ca)
        got[m] = [res.C.val[res.C.row_ptr[r]:res.C.row_ptr[r + 1]] for r in range(m)]
    for m in (LAST_FEW, many):
        for r in range(m):
            np.testing.assert_array_equal(got[m][r].view(np.uint64), got[few][r % few].view(np.uint64))
