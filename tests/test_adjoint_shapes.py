"""Adjoint of many rows of more than 256 entries, which are told apart by their
shape: rows of C around the kernels' sizes (512, 1024 and 2048 entries), entries
of A around the steps' groups, one product an entry up to a whole row in one, and
rows of uneven entries.  |d - oracle| <= 1e-12 * sum of |terms|; dA, and with
DBD_ADJ_DETERMINISTIC dB, are the same bits on every run."""
import ctypes

import numpy as np
import pytest

import dbd_gb300 as dbd
import oracle

pytestmark = pytest.mark.gpu
ROWS = 1600  # told apart from 1520 on (152 SMs)


def _adjoint(ctx, A, B, g, flags):
    va, ka = A.view()
    vb, kb = B.view()
    da, db = np.full(A.nnz, np.nan), np.full(B.nnz, np.nan)
    dbd._check(ctx._lib.dbd_spgemm_adjoint(ctx.handle, ctypes.byref(va), ctypes.byref(vb), g.ctypes.data,
                                           da.ctypes.data, db.ctypes.data, 0, flags), ctx.handle)
    del ka, kb
    return da, db


def _check(A, B, rng):
    with dbd.Context(cpu_gib=2, gpu_gib=8) as ctx:
        C = ctx.spgemm(A, B).C
        g = rng.standard_normal(C.nnz)
        got = [_adjoint(ctx, A, B, g, flags) for flags in (0, 2, 2)]
    da, db = oracle.adjoint(A, B, C.row_ptr, C.col_idx, g)
    absA = dbd.CSR(A.n_rows, A.n_cols, A.row_ptr, A.col_idx, np.abs(A.val))
    absB = dbd.CSR(B.n_rows, B.n_cols, B.row_ptr, B.col_idx, np.abs(B.val))
    sa, sb = oracle.adjoint(absA, absB, C.row_ptr, C.col_idx, np.abs(g))
    for a, b in got:
        assert np.all(np.abs(a - da) <= 1e-12 * sa)
        assert np.all(np.abs(b - db) <= 1e-12 * sb)
        np.testing.assert_array_equal(a, got[0][0])
    np.testing.assert_array_equal(got[1][1], got[2][1])
    return np.diff(C.row_ptr)


@pytest.mark.parametrize("entries, products", [
    (1, 512), (1, 513), (1, 1024), (1, 2049), (3, 171), (4, 128), (5, 103), (8, 64), (9, 57), (9, 113), (16, 32),
    (17, 31), (17, 121), (33, 9), (64, 8), (65, 9), (100, 4), (100, 5), (300, 1), (300, 3), (512, 1), (513, 1),
    (1024, 1), (1025, 1), (2048, 1), (2049, 1)])
def test_even_rows(entries, products):
    rng = np.random.default_rng(entries * 31 + products)
    k = max(2 * entries, 40)  # rows of B, over columns of their own
    n = k * products
    B = dbd.CSR(k, n, (np.arange(k + 1) * products).astype(np.int32), np.arange(n, dtype=np.int32),
                rng.standard_normal(n))
    idx = np.concatenate([np.sort(rng.choice(k, entries, replace=False)) for _ in range(ROWS)]).astype(np.int32)
    A = dbd.CSR(ROWS, k, (np.arange(ROWS + 1) * entries).astype(np.int32), idx, rng.standard_normal(idx.size))
    assert np.all(_check(A, B, rng) == entries * products)


def test_uneven_rows():
    """Entries of 0 to 1500 products, most of them short, some columns shared; rows of every kind at once."""
    rng = np.random.default_rng(3)
    k, n = 4000, 60000
    lens = np.minimum(rng.zipf(1.5, k) - 1, 1500)
    B = dbd.CSR(k, n, np.r_[0, np.cumsum(lens)].astype(np.int32),
                np.concatenate([np.sort(rng.choice(n, l, replace=False)) for l in lens]).astype(np.int32),
                rng.standard_normal(int(lens.sum())))
    rows = [np.sort(rng.choice(k, e, replace=False)) for e in rng.integers(20, 400, 2 * ROWS)]
    A = dbd.CSR(len(rows), k, np.r_[0, np.cumsum([r.size for r in rows])].astype(np.int32),
                np.concatenate(rows).astype(np.int32), rng.standard_normal(sum(r.size for r in rows)))
    nnz = _check(A, B, rng)
    assert (nnz > 256).sum() >= ROWS and (nnz > 2048).any() and ((nnz > 256) & (nnz <= 512)).any()
