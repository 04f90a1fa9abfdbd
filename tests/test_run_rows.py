"""Symbolic sizes of narrow rows over column runs: unions counted without
per-column work where the runs' ends ascend, by prefix maxima where only their
starts do, and per column otherwise; around steps of 32 entries."""
import numpy as np
import pytest

import dbd_gb300 as dbd
import oracle

pytestmark = pytest.mark.gpu
FLAGW = 2


@pytest.mark.parametrize("entries", [3, 31, 32, 33, 64, 65, 97])
@pytest.mark.parametrize("kind", ["band", "nested", "equal starts", "empty rows among them", "descending", "a gap"])
def test_unions_of_runs(entries, kind):
    rng = np.random.default_rng(entries)
    start = 10 + 3 * np.arange(entries)
    length = np.full(entries, 40)
    if kind == "nested":
        length = rng.integers(17, 90, entries)
    elif kind == "equal starts":
        start = 10 + 20 * (np.arange(entries) // 5)
        length = 20 + np.arange(entries) % 7
    elif kind == "empty rows among them":
        length[rng.random(entries) < 0.3] = 0
        length[1] = 500  # its end stays the largest for a while
    elif kind == "descending":
        start = start[::-1].copy()
    rows = [np.arange(s, s + l) for s, l in zip(start, length)]
    if kind == "a gap":
        rows[entries // 2] = np.delete(rows[entries // 2], 7)
    n = int(max(r[-1] for r in rows if len(r))) + 3
    ptr = np.r_[0, np.cumsum([len(r) for r in rows])].astype(np.int32)
    B = dbd.CSR(entries, n, ptr, np.concatenate(rows).astype(np.int32), rng.standard_normal(int(ptr[-1])))
    cols = [np.arange(entries), np.arange(3), np.arange(entries)]
    ptr = np.r_[0, np.cumsum([len(c) for c in cols])].astype(np.int32)
    A = dbd.CSR(3, entries, ptr, np.concatenate(cols).astype(np.int32), rng.standard_normal(int(ptr[-1])))
    with dbd.Context(cpu_gib=1, gpu_gib=4) as ctx:
        res = ctx.spgemm(A, B)
    assert res.stats["sym_rows_per_bin"][FLAGW] >= 2
    Cp, Ci, Cv, Ca = oracle.spgemm(A, B, with_abs=True)
    np.testing.assert_array_equal(res.C.row_ptr, Cp)
    np.testing.assert_array_equal(res.C.col_idx, Ci)
    assert np.all(np.abs(res.C.val - Cv) <= 1e-12 * Ca)
