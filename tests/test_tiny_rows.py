"""Rows of at most 32 products: one lane each, sorted in registers by 8, 16 or
32 keys.  Bit for bit equal to the oracle (Gustavson order), at the edges of
the sort sizes, of a warp's 32 rows and of the 2^27-column key range."""
import numpy as np
import pytest

import dbd_gb300 as dbd
import oracle

pytestmark = pytest.mark.gpu


def _matrix(n_rows, n_cols, rows, seed):
    """rows[r]: the columns of row r; values with signed zeros among them."""
    rng = np.random.default_rng(seed)
    ptr = np.zeros(n_rows + 1, np.int64)
    np.cumsum([len(r) for r in rows], out=ptr[1:])
    idx = np.concatenate([np.asarray(r, np.int64) for r in rows] + [np.zeros(0, np.int64)]).astype(np.int32)
    val = rng.standard_normal(idx.size)
    val[rng.random(idx.size) < 0.1] = -0.0
    return dbd.CSR(n_rows, n_cols, ptr.astype(np.int32), idx, val)


def _check(A, B, want):
    with dbd.Context(cpu_gib=1, gpu_gib=4) as ctx:
        res = ctx.spgemm(A, B)
    assert res.stats["sym_rows_per_bin"][1] == want and res.stats["rows_per_bin"][1] == want
    return res.C


@pytest.mark.parametrize("rows", [1, 31, 33, 64, 65, 200])
@pytest.mark.parametrize("products", [1, 8, 9, 16, 17, 31, 32])
@pytest.mark.parametrize("order", ["ascending", "shuffled"])
def test_tiny_rows_bit_exact(rows, products, order):
    rng = np.random.default_rng(rows * 100 + products)
    k, n = 97, 41  # few columns: most are hit several times
    lens = rng.integers(0, 6, k)
    lens[0], lens[1] = 1, 0
    brows = [rng.choice(n, l, replace=False) for l in lens]
    if order == "ascending":
        brows = [np.sort(r) for r in brows]
    B = _matrix(k, n, brows, 1)
    arows = []
    for _ in range(rows):
        left, cols = products, []
        for c in rng.permutation(np.arange(2, k)):
            if lens[c] <= left and len(cols) < 30:
                cols.append(c)
                left -= lens[c]
        arows.append(np.sort(np.asarray(cols + ([0] if left else []), np.int64)))
    A = _matrix(rows, k, arows, 2)
    live = sum(1 for r in arows if sum(lens[c] for c in r))
    C = _check(A, B, live)
    Cp, Ci, Cv = oracle.spgemm(A, B)
    np.testing.assert_array_equal(C.row_ptr, Cp)
    np.testing.assert_array_equal(C.col_idx, Ci)
    np.testing.assert_array_equal(C.val.view(np.uint64), Cv.view(np.uint64))


@pytest.mark.parametrize("span", [(1 << 27) - 1, 1 << 27, (1 << 27) + 1, (1 << 31) - 2])
def test_tiny_rows_over_wide_spans(span):
    """Columns 0 and `span` among a row's columns: around the 32-bit keys' range."""
    low = [0, 3, 5]
    B = _matrix(4, (1 << 31) - 1, [low, [3, span], [5, 7, span], [0, span - 1]], 3)
    A = _matrix(3, 4, [[0, 1, 2, 3], [1, 3], [0]], 4)
    C = _check(A, B, 3)
    for r in range(3):
        ref = {}
        for e in range(A.row_ptr[r], A.row_ptr[r + 1]):
            k = A.col_idx[e]
            for f in range(B.row_ptr[k], B.row_ptr[k + 1]):
                c = int(B.col_idx[f])
                ref[c] = ref.get(c, 0.0) + A.val[e] * B.val[f]
        s = slice(C.row_ptr[r], C.row_ptr[r + 1])
        assert C.col_idx[s].tolist() == sorted(ref)
        np.testing.assert_array_equal(C.val[s], [ref[c] for c in sorted(ref)])
