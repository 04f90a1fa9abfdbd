"""Warp rows of at most 512 products (expand, sort, compress in registers) at
the edges of the sort sizes, with no, few and many equal columns (runs within
a lane, over a lane's edge and over many lanes), and column spans around the
32-bit keys' ranges."""
import numpy as np
import pytest

import dbd_gb300 as dbd
import oracle

pytestmark = pytest.mark.gpu
HWARP = 3


def _from_rows(n_cols, rows, seed):
    ptr = np.zeros(len(rows) + 1, np.int64)
    np.cumsum([len(r) for r in rows], out=ptr[1:])
    idx = np.concatenate([np.asarray(r, np.int64) for r in rows]).astype(np.int32)
    return dbd.CSR(len(rows), n_cols, ptr.astype(np.int32), idx, np.random.default_rng(seed).standard_normal(idx.size))


@pytest.mark.parametrize("products", [33, 64, 128, 191, 192, 193, 255, 256, 257, 400, 511, 512, 513])
@pytest.mark.parametrize("distinct", [1, 2, 7, 60, 250, 10**9])
def test_sorted_rows(products, distinct):
    """Every B row holds `per` of the columns; a row of C over them has min(distinct, products) or fewer."""
    rng = np.random.default_rng(products * 7 + min(distinct, 1000))
    n = 70000  # spans over 2048 words: warp rows, hashed or sorted
    pool = np.sort(rng.choice(n, min(distinct, 250), replace=False))
    pool[0], pool[-1] = 0, n - 1
    pool = np.unique(pool)
    if pool.size == 1:
        pool = np.array([0, n - 1])
    per = min(8, pool.size)
    lens = [per] * (products // per) + ([products % per] if products % per else [])
    B = _from_rows(n, [rng.choice(pool, l, replace=False) for l in lens] + [[]], 1)
    order = np.arange(len(lens) + 1)
    A = _from_rows(len(lens) + 1, [order, order[::-1], order], 2)
    with dbd.Context(cpu_gib=1, gpu_gib=4) as ctx:
        res = ctx.spgemm(A, B)
    Cp, Ci, Cv, Ca = oracle.spgemm(A, B, with_abs=True)
    assert res.stats["rows_per_bin"][HWARP] == 3
    np.testing.assert_array_equal(res.C.row_ptr, Cp)
    np.testing.assert_array_equal(res.C.col_idx, Ci)
    assert np.all(np.abs(res.C.val - Cv) <= 1e-12 * Ca)


@pytest.mark.parametrize("products", [128, 192, 256, 512])
@pytest.mark.parametrize("span", [(1 << 23) - 1, 1 << 23, (1 << 23) + 1, 1 << 25])
def test_sorted_rows_over_wide_spans(products, span):
    """The row's first and last column are 5 and 5 + span - 1."""
    rng = np.random.default_rng(span % 1000 + products)
    pool = np.unique(np.r_[5, 5 + span - 1, 5 + rng.choice(span, 200, replace=False)])
    n = (1 << 25) + 10
    lens = [16] * (products // 16)
    rows = [np.sort(rng.choice(pool, 16, replace=False)) for _ in lens]
    rows[0] = np.unique(np.r_[pool[0], pool[-1], rng.choice(pool[1:-1], 14, replace=False)])
    B = _from_rows(n, rows, 1)
    A = _from_rows(len(lens), [np.arange(len(lens))], 2)
    with dbd.Context(cpu_gib=1, gpu_gib=4) as ctx:
        res = ctx.spgemm(A, B)
    assert res.stats["rows_per_bin"][HWARP] == 1
    ref, size = {}, {}
    for e in range(A.nnz):
        for f in range(B.row_ptr[e], B.row_ptr[e + 1]):
            c, x = int(B.col_idx[f]), A.val[e] * B.val[f]
            ref[c] = ref.get(c, 0.0) + x
            size[c] = size.get(c, 0.0) + abs(x)
    assert res.C.col_idx.tolist() == sorted(ref)
    want, tol = (np.array([d[c] for c in sorted(ref)]) for d in (ref, size))
    assert np.all(np.abs(res.C.val - want) <= 1e-12 * tol)
