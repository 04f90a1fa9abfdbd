"""Narrow rows whose B rows are runs of columns, taken as one flat sequence of
products: run lengths around a step of 32, runs starting at every distance
from the run before (overlapping steps must fall back), descending and repeated
runs, A rows around a chunk of 32 entries.  Values within 1e-12 * sum |terms|
and the same bits on every run."""
import numpy as np
import pytest

import dbd_gb300 as dbd
import oracle

pytestmark = pytest.mark.gpu
DENSEW = 9


def _check(A, B):
    got = []
    with dbd.Context(cpu_gib=1, gpu_gib=4) as ctx:
        for _ in range(2):
            got.append(ctx.spgemm(A, B))
    assert got[0].stats["rows_per_bin"][DENSEW] == A.n_rows
    Cp, Ci, Cv, Ca = oracle.spgemm(A, B, with_abs=True)
    C = got[0].C
    np.testing.assert_array_equal(C.row_ptr, Cp)
    np.testing.assert_array_equal(C.col_idx, Ci)
    assert np.all(np.abs(C.val - Cv) <= 1e-12 * Ca)
    np.testing.assert_array_equal(C.val.view(np.uint64), got[1].C.val.view(np.uint64))


def _runs(starts, lens, n_cols, seed):
    idx = np.concatenate([np.arange(s, s + l) for s, l in zip(starts, lens)]).astype(np.int32)
    ptr = np.zeros(len(lens) + 1, np.int64)
    np.cumsum(lens, out=ptr[1:])
    return dbd.CSR(len(lens), n_cols, ptr.astype(np.int32), idx, np.random.default_rng(seed).standard_normal(idx.size))


def _all_entries(rows, k, seed):
    """`rows` rows over all k entries, 0 .. k - 1 in order; the last row without its last entry from the third on."""
    cols = [np.arange(k)] * (rows - 1) + [np.arange(min(k, max(2, k - 1)))]
    ptr = np.zeros(rows + 1, np.int64)
    np.cumsum([len(c) for c in cols], out=ptr[1:])
    idx = np.concatenate(cols).astype(np.int32)
    return dbd.CSR(rows, k, ptr.astype(np.int32), idx, np.random.default_rng(seed).standard_normal(idx.size))


@pytest.mark.parametrize("entries", [2, 31, 32, 33, 64, 65])
@pytest.mark.parametrize("length", [31, 32, 33, 63, 64, 65, 129])
@pytest.mark.parametrize("step", [0, 1, 2])
def test_bands(entries, length, step):
    B = _runs(7 + step * np.arange(entries), np.full(entries, length), 7 + step * entries + length, 1)
    _check(_all_entries(3, entries, 2), B)


@pytest.mark.parametrize("distance", [-40, -1, 0, 1, 7, 8, 9, 32, 39, 40, 41, 60])
@pytest.mark.parametrize("length", [32, 40, 41])
def test_distances_between_runs(distance, length):
    """Six runs of `length`, each `distance` behind the one before."""
    starts = 300 + distance * np.arange(6) - min(0, 5 * distance) - (200 if distance > 20 else 0)
    starts = starts - starts.min() + 3
    B = _runs(starts, np.full(6, length), int(starts.max()) + length + 2, 1)
    _check(_all_entries(2, 6, 2), B)


def test_mixed_rows():
    """Runs beside rows with a gap, short rows and empty ones, 40 entries in random order."""
    rng = np.random.default_rng(5)
    starts = rng.integers(0, 200, 40)
    lens = rng.choice([0, 1, 20, 33, 64, 100], 40, p=[0.1, 0.1, 0.1, 0.2, 0.3, 0.2])
    B = _runs(starts, lens, 310, 1)
    keep = np.ones(B.nnz, bool)
    keep[B.row_ptr[:-1][lens == 64] + 30] = False  # a gap in the runs of 64
    ptr = np.zeros(41, np.int64)
    ptr[1:] = np.cumsum(np.add.reduceat(np.append(keep, False).astype(int), B.row_ptr[:-1]) * (lens > 0))
    B = dbd.CSR(40, 310, ptr.astype(np.int32), B.col_idx[keep], B.val[keep])
    _check(_all_entries(5, 40, 2), B)
