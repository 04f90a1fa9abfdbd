"""Rows whose sums are fused multiply-adds, by their error against exact sums.

Every column of C has two products, both in [1, 2).  A fused sum rounds the
first product (by at most 2^-53) and then the sum, which lies in [2, 4) (by at
most 2^-52): 3 * 2^-53 in all.  Products rounded one by one before they are
added may be off by 4 * 2^-53, and one column in sixteen is by more than 3."""
import numpy as np
import pytest

import dbd_gb300 as dbd

pytestmark = pytest.mark.gpu
HWARP, RANKS = 3, 4


def _exact(x):
    """The number as an integer multiple of 2^-52 (for x in [1, 2))."""
    return [int(v) for v in np.ldexp(x, 52).astype(np.int64)]


# Columns of a row, the columns they are drawn from, and the bin that takes them.
@pytest.mark.parametrize("columns, n, bin_of", [(129, 70000, HWARP), (200, 70000, HWARP), (256, 70000, HWARP),
                                                (256, 1 << 26, HWARP), (257, 70000, RANKS), (1000, 4000, RANKS),
                                                (3960, 250000, RANKS), (3961, 250000, RANKS), (4096, 250000, RANKS)])
def test_two_products_a_column(columns, n, bin_of):
    rng = np.random.default_rng(columns)
    rows = max(8, 3000 // columns)
    # Rows 2r and 2r + 1 of B have the same columns, and row r of A takes both.
    cols = [np.unique(np.r_[0, rng.choice(n - 2, columns - 2, replace=False) + 1, n - 1]) for _ in range(rows)]
    idx = np.concatenate([c for c in cols for _ in "ab"]).astype(np.int32)
    B = dbd.CSR(2 * rows, n, (np.arange(2 * rows + 1) * columns).astype(np.int32), idx, rng.uniform(1.0, 1.4, idx.size))
    A = dbd.CSR(rows, 2 * rows, (2 * np.arange(rows + 1)).astype(np.int32), np.arange(2 * rows, dtype=np.int32),
                rng.uniform(1.0, 1.4, 2 * rows))
    with dbd.Context(cpu_gib=1, gpu_gib=4) as ctx:
        res = ctx.spgemm(A, B)
    assert res.stats["rows_per_bin"][bin_of] == rows
    np.testing.assert_array_equal(res.C.col_idx, np.concatenate(cols))
    a, b = _exact(A.val), _exact(B.val)
    got = [int(v) for v in np.ldexp(res.C.val, 51).astype(np.int64)]  # in [2, 4): multiples of 2^-51
    for r in range(rows):
        for j in range(columns):
            want = sum(a[2 * r + h] * b[(2 * r + h) * columns + j] for h in (0, 1))  # multiples of 2^-104
            assert abs((got[r * columns + j] << 53) - want) <= 3 << 51


@pytest.mark.parametrize("products", [257, 300, 480, 511, 512])
@pytest.mark.parametrize("distinct", [2, 3, 9, 70, 240])
@pytest.mark.parametrize("per", [1.2, 3, 12])
def test_warp_rows_are_chains_in_order(products, distinct, per):
    """Warp rows of 257 to 512 products of at most 256 entries: every sum is the fused multiply-adds of its
    products in A's entry order, bit for bit; with more entries a row takes the table, which adds in any order."""
    from fractions import Fraction
    rng = np.random.default_rng(products + distinct)
    n = 70000
    pool = np.unique(np.r_[0, rng.choice(n - 2, distinct - 2, replace=False) + 1, n - 1])
    lens = []
    while sum(lens) < products:
        top = min(pool.size, products - sum(lens))
        lens.append(int(min(top, 1 + rng.poisson(per - 1))))
    cols = [np.sort(rng.choice(pool, l, replace=False)) for l in lens]
    cols[0][:1], cols[-1][-1:] = pool[0], pool[-1]  # the window's ends
    cols = [np.unique(c) for c in cols]
    idx = np.concatenate(cols).astype(np.int32)
    if not 256 < idx.size <= 512:
        pytest.skip("another class of rows")
    B = dbd.CSR(len(cols), n, np.r_[0, np.cumsum([c.size for c in cols])].astype(np.int32), idx,
                rng.standard_normal(idx.size))
    A = dbd.CSR(2, len(cols), (np.arange(3) * len(cols)).astype(np.int32), np.tile(np.arange(len(cols)), 2).astype(np.int32),
                rng.standard_normal(2 * len(cols)))
    with dbd.Context(cpu_gib=1, gpu_gib=4) as ctx:
        res = ctx.spgemm(A, B)
    assert res.stats["rows_per_bin"][HWARP] == 2
    for r in range(2):
        want, size = {}, {}
        for e in range(len(cols)):
            x = A.val[r * len(cols) + e]
            for f in range(B.row_ptr[e], B.row_ptr[e + 1]):
                c = int(B.col_idx[f])
                want[c] = float(Fraction(x) * Fraction(B.val[f]) + Fraction(want.get(c, 0.0)))
                size[c] = size.get(c, 0.0) + abs(x * B.val[f])
        s, t = res.C.row_ptr[r], res.C.row_ptr[r + 1]
        assert res.C.col_idx[s:t].tolist() == sorted(want)
        exact = np.array([want[c] for c in sorted(want)])
        if len(cols) <= 256:
            np.testing.assert_array_equal(res.C.val[s:t], exact)
        else:
            assert np.all(np.abs(res.C.val[s:t] - exact) <= 1e-12 * np.array([size[c] for c in sorted(want)]))
