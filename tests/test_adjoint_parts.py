"""Adjoint of rows heavy enough to be cut into parts: parts that start inside
a batch, empty ones (one B row holds nearly all products), batches of fewer
products than parts, narrow and wide rows of C.  |d - oracle| <= 1e-12 * sum
of |terms|, and the same bits on every run where that is promised."""
import ctypes

import numpy as np
import pytest

import dbd_gb300 as dbd
import oracle

pytestmark = pytest.mark.gpu


def _lens(case, rng):
    if case == "even":
        return np.full(1300, 230)
    if case == "one entry":
        return np.r_[rng.integers(0, 3, 300), 90000, rng.integers(0, 3, 300)]
    if case == "just cut":
        return np.full(64, 128)  # 8192 products, the least that is cut
    assert case == "thin last batch"
    return np.r_[np.full(512, 900), np.zeros(30, int), 1, 1]


def _adjoint(ctx, A, B, g, flags):
    va, ka = A.view()
    vb, kb = B.view()
    da, db = np.full(A.nnz, np.nan), np.full(B.nnz, np.nan)
    dbd._check(ctx._lib.dbd_spgemm_adjoint(ctx.handle, ctypes.byref(va), ctypes.byref(vb), g.ctypes.data,
                                           da.ctypes.data, db.ctypes.data, 0, flags), ctx.handle)
    del ka, kb
    return da, db


@pytest.mark.parametrize("n_cols", [100000, 1 << 19])
@pytest.mark.parametrize("case", ["even", "one entry", "just cut", "thin last batch"])
def test_adjoint_parts(case, n_cols):
    rng = np.random.default_rng(5)
    lens = _lens(case, rng)
    ptr = np.r_[0, np.cumsum(lens)].astype(np.int32)
    idx = np.concatenate([np.sort(rng.choice(n_cols, l, replace=False)) for l in lens]).astype(np.int32)
    B = dbd.CSR(lens.size, n_cols, ptr, idx, rng.standard_normal(idx.size))
    # The whole of B twice among rows that are not cut.
    rows = [np.arange(3), np.arange(lens.size), np.arange(lens.size // 4), np.arange(lens.size), np.arange(1)]
    aptr = np.r_[0, np.cumsum([r.size for r in rows])].astype(np.int32)
    A = dbd.CSR(len(rows), lens.size, aptr, np.concatenate(rows).astype(np.int32), rng.standard_normal(aptr[-1]))
    with dbd.Context(cpu_gib=1, gpu_gib=8) as ctx:
        C = ctx.spgemm(A, B).C
        g = rng.standard_normal(C.nnz)
        got = [_adjoint(ctx, A, B, g, flags) for flags in (0, 0, 2, 2)]
    da, db = oracle.adjoint(A, B, C.row_ptr, C.col_idx, g)
    absA = dbd.CSR(A.n_rows, A.n_cols, A.row_ptr, A.col_idx, np.abs(A.val))
    absB = dbd.CSR(B.n_rows, B.n_cols, B.row_ptr, B.col_idx, np.abs(B.val))
    sa, sb = oracle.adjoint(absA, absB, C.row_ptr, C.col_idx, np.abs(g))
    for a, b in got:
        assert np.all(np.abs(a - da) <= 1e-12 * sa)
        assert np.all(np.abs(b - db) <= 1e-12 * sb)
        np.testing.assert_array_equal(a, got[0][0])
    np.testing.assert_array_equal(got[2][1], got[3][1])
