"""Infinities and NaN among the values, through every numeric bin and the
adjoint's kernels: they land where the oracle has them, with its signs, and
leave every other entry alone."""
import ctypes

import numpy as np
import pytest

import dbd_gb300 as dbd
import oracle

pytestmark = pytest.mark.gpu

# Entries of a row of A, of a row of B, C's columns, how many of them are used, and the bin that takes the rows.
SHAPES = {
    "tiny": (3, 5, 1000, 1000, 1),
    "warp ranks": (40, 8, 1500, 250, 2),
    "sorted": (20, 8, 90000, 90000, 3),
    "sorted, fused": (40, 10, 90000, 200, 3),
    "table": (80, 10, 90000, 200, 3),
    "ranks in shared memory": (60, 20, 90000, 90000, 4),
    "ranks in place": (600, 20, 90000, 90000, 5),
    "hashed, small": (40, 20, 1 << 24, 1 << 24, 6),
    "hashed, large": (150, 20, 1 << 24, 1 << 24, 7),
    "windows": (600, 20, 1 << 24, 1 << 24, 8),
    "runs": (40, 65, 500, 500, 9),
}


def _operands(shape, rows, rng):
    entries, per, n, used, _ = SHAPES[shape]
    k = entries + 7
    if shape == "runs":
        cols = [np.arange(s, s + per) for s in rng.integers(0, n - per, k)]
    elif used == n:
        cols = [np.unique(rng.integers(0, n, per)) for _ in range(k)]
    else:
        pool = np.unique(np.r_[0, rng.choice(n, used, replace=False), n - 1])
        cols = [np.sort(rng.choice(pool, per, replace=False)) for _ in range(k)]
        cols = [np.unique(np.r_[c, pool[[0, -1]]]) for c in cols]  # every row as wide as the pool
    def csr(n_cols, rs):
        idx = np.concatenate(rs).astype(np.int32)
        val = rng.standard_normal(idx.size)
        odd = rng.random(idx.size) < 3.0 / idx.size ** 0.75
        val[odd] = rng.choice([np.inf, -np.inf, np.nan, 0.0, -0.0], odd.sum())
        val[rng.integers(idx.size, size=2)] = np.inf, np.nan
        return dbd.CSR(len(rs), n_cols, np.r_[0, np.cumsum([r.size for r in rs])].astype(np.int32), idx, val)
    B = csr(n, cols)
    return csr(k, [np.sort(rng.choice(k, entries, replace=False)) for _ in range(rows)]), B


def _same(got, want, size):
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
    inf = np.isinf(want)
    np.testing.assert_array_equal(got[inf], want[inf])
    fine = np.isfinite(want)
    assert inf.any() or np.isnan(want).any()
    assert np.all(np.abs(got[fine] - want[fine]) <= 1e-12 * size[fine])


def _abs(m):
    return dbd.CSR(m.n_rows, m.n_cols, m.row_ptr, m.col_idx, np.abs(m.val))


@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_multiply(shape):
    A, B = _operands(shape, 6, np.random.default_rng(len(shape)))
    with dbd.Context(cpu_gib=1, gpu_gib=8) as ctx:
        res = ctx.spgemm(A, B)
    assert res.stats["rows_per_bin"][SHAPES[shape][4]] == 6
    Cp, Ci, Cv, Ca = oracle.spgemm(A, B, with_abs=True)
    np.testing.assert_array_equal(res.C.col_idx, Ci)
    _same(res.C.val, Cv, Ca)


@pytest.mark.parametrize("rows", [6, 1600])
@pytest.mark.parametrize("shape", ["sorted", "ranks in shared memory", "hashed, small", "runs"])
@pytest.mark.parametrize("flags", [0, 2])
def test_adjoint(shape, rows, flags):
    rng = np.random.default_rng(rows + len(shape))
    A, B = _operands(shape, rows, rng)
    with dbd.Context(cpu_gib=1, gpu_gib=8) as ctx:
        C = ctx.spgemm(A, B).C
        g = rng.standard_normal(C.nnz)
        g[rng.integers(C.nnz, size=3)] = np.inf, -np.inf, np.nan
        va, ka = A.view()
        vb, kb = B.view()
        da, db = np.zeros(A.nnz), np.zeros(B.nnz)
        dbd._check(ctx._lib.dbd_spgemm_adjoint(ctx.handle, ctypes.byref(va), ctypes.byref(vb), g.ctypes.data,
                                               da.ctypes.data, db.ctypes.data, 0, flags), ctx.handle)
    with np.errstate(invalid="ignore"):
        wa, wb = oracle.adjoint(A, B, C.row_ptr, C.col_idx, g)
        sa, sb = oracle.adjoint(_abs(A), _abs(B), C.row_ptr, C.col_idx, np.abs(g))
    _same(da, wa, sa)
    _same(db, wb, sb)
