"""Adjoint kernels at the edges of their row classes: rows of C around the
warp kernel's bins, rows staged in several batches, entries whose products
span several warps, many one-product entries in a step, empty B rows and rows
of C too wide for the bitmap.  |d - oracle| <= 1e-12 * sum of |terms|; dA, and
with DBD_ADJ_DETERMINISTIC dB, are the same bits on every run."""
import ctypes

import numpy as np
import pytest

import dbd_gb300 as dbd
import oracle

pytestmark = pytest.mark.gpu


def _from_rows(n_cols, rows, seed):
    ptr = np.zeros(len(rows) + 1, np.int64)
    np.cumsum([len(r) for r in rows], out=ptr[1:])
    idx = np.concatenate([np.asarray(r, np.int64) for r in rows]).astype(np.int32)
    return dbd.CSR(len(rows), n_cols, ptr.astype(np.int32), idx, np.random.default_rng(seed).standard_normal(idx.size))


def _spread(n_cols, lens, rng):
    return [np.sort(rng.choice(n_cols, l, replace=False)) for l in lens]


def _operands(case):
    rng = np.random.default_rng(7)
    if case == "around 256 entries":
        # Row r of A takes one B row of 200 + r entries: rows of C of 200 to 320.
        B = _from_rows(40000, _spread(40000, range(200, 321), rng), 1)
        A = _from_rows(121, [[r] for r in range(121)], 2)
    elif case == "narrow windows":
        # Up to 512 columns: the dense-window bin.
        B = _from_rows(512, _spread(512, rng.integers(1, 300, 400), rng), 1)
        A = _from_rows(400, _spread(400, rng.integers(1, 200, 50), rng), 2)
    elif case == "long entries":
        # One entry of 30000 products among short and empty ones.
        lens = np.r_[30000, 0, 3, 1, 700, np.zeros(5, int), rng.integers(0, 40, 200)]
        B = _from_rows(60000, _spread(60000, lens, rng), 1)
        A = _from_rows(lens.size, [np.arange(lens.size), [0], [0, 1, 2], [3, 4], np.arange(1, lens.size)], 2)
    elif case == "one-product entries":
        # 3000 entries of one or two products: several batches, many entries a step.
        B = _from_rows(9000, _spread(9000, rng.integers(1, 3, 4000), rng), 1)
        A = _from_rows(4000, _spread(4000, [3000, 513, 512, 511, 1], rng), 2)
    else:
        assert case == "wide rows"
        n = 1 << 20  # over 2^18 columns: binary search
        B = _from_rows(n, _spread(n, rng.integers(0, 400, 60), rng), 1)
        A = _from_rows(60, _spread(60, [60, 30, 5, 1], rng), 2)
    return A, B


def _products(A, B):
    return int(np.diff(B.row_ptr)[A.col_idx].sum())


def _adjoint(ctx, A, B, g, flags):
    va, ka = A.view()
    vb, kb = B.view()
    da, db = np.full(A.nnz, np.nan), np.full(B.nnz, np.nan)
    dbd._check(ctx._lib.dbd_spgemm_adjoint(ctx.handle, ctypes.byref(va), ctypes.byref(vb), g.ctypes.data,
                                           da.ctypes.data, db.ctypes.data, 0, flags), ctx.handle)
    del ka, kb
    return da, db


@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("case", ["around 256 entries", "narrow windows", "long entries", "one-product entries",
                                  "wide rows"])
def test_adjoint_row_classes(case, shuffled):
    A, B = _operands(case)
    if shuffled:  # columns inside a row need not ascend
        rng = np.random.default_rng(3)
        for M in (A, B):
            for r in range(M.n_rows):
                s = slice(M.row_ptr[r], M.row_ptr[r + 1])
                M.col_idx[s] = rng.permutation(M.col_idx[s])
    got = []
    # An eighth of the second budget is less than the products take.
    for gib, runs in ((8, (0, 2, 2, 1)), (0.9 * 64 * _products(A, B) / 2**30, (0, 2))):
        with dbd.Context(cpu_gib=1, gpu_gib=gib) as ctx:
            C = ctx.spgemm(A, B).C
            g = np.random.default_rng(4).standard_normal(C.nnz)
            got += [_adjoint(ctx, A, B, g, flags) for flags in runs]
    da, db = oracle.adjoint(A, B, C.row_ptr, C.col_idx, g)
    absA = dbd.CSR(A.n_rows, A.n_cols, A.row_ptr, A.col_idx, np.abs(A.val))
    absB = dbd.CSR(B.n_rows, B.n_cols, B.row_ptr, B.col_idx, np.abs(B.val))
    sa, sb = oracle.adjoint(absA, absB, C.row_ptr, C.col_idx, np.abs(g))
    for x, y in got:
        assert np.all(np.abs(x - da) <= 1e-12 * sa)
        assert np.all(np.abs(y - db) <= 1e-12 * sb)
        np.testing.assert_array_equal(x.view(np.uint64), got[0][0].view(np.uint64))
    np.testing.assert_array_equal(got[1][1].view(np.uint64), got[2][1].view(np.uint64))
    np.testing.assert_array_equal(got[1][1].view(np.uint64), got[5][1].view(np.uint64))
