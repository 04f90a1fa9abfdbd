"""Symbolic wide rows of 2^18 products and more, launched on their own, and of 2^19 and
more, cut into column slabs: at both thresholds, over windows of two slabs up
to several windows, with B's rows ascending (cut) and not (whole)."""
import numpy as np
import pytest

import dbd_gb300 as dbd
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entries", [63, 64, 127, 128, 300])
@pytest.mark.parametrize("cols", [70_000, 1 << 18, (1 << 18) + 70_000, 1_300_000])
@pytest.mark.parametrize("order", ["ascending", "shuffled"])
def test_heavy_rows(entries, cols, order):
    rng = np.random.default_rng(entries + cols)
    per = 4096  # products an entry
    k = 300
    # Columns crowd towards 0, as a power-law graph's do, and reach the last one.
    draw = lambda: np.unique((cols * rng.random(3 * per) ** 2).astype(np.int64))
    rows = []
    for _ in range(k):
        c = rng.permutation(draw())[:per]
        c[0] = cols - 1 if cols - 1 not in c else c[0]
        rows.append(np.sort(c) if order == "ascending" else c)
    assert all(len(r) == per for r in rows)
    idx = np.concatenate(rows).astype(np.int32)
    B = dbd.CSR(k, cols, (np.arange(k + 1) * per).astype(np.int32), idx, rng.standard_normal(idx.size))
    a_cols = [np.arange(entries), np.arange(3), np.arange(k - entries, k), np.arange(1)]
    ptr = np.r_[0, np.cumsum([len(c) for c in a_cols])].astype(np.int32)
    A = dbd.CSR(4, k, ptr, np.concatenate(a_cols).astype(np.int32), rng.standard_normal(int(ptr[-1])))
    with dbd.Context(cpu_gib=1, gpu_gib=8) as ctx:
        res = ctx.spgemm(A, B)
    Cp, Ci, Cv, Ca = oracle.spgemm(A, B, with_abs=True)
    np.testing.assert_array_equal(res.C.row_ptr, Cp)
    np.testing.assert_array_equal(res.C.col_idx, Ci)
    assert np.all(np.abs(res.C.val - Cv) <= 1e-12 * Ca)
