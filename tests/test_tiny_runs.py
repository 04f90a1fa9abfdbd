"""Tiny rows of C that do not follow each other in a warp's run of rows: longer
rows between them, empty ones, pairs of a batch; bit for bit the oracle's."""
import numpy as np
import pytest

import dbd_gb300 as dbd
import oracle

pytestmark = pytest.mark.gpu


def _matrices(kind, rows, seed):
    """A whose rows are tiny except where `kind` puts a longer or an empty one."""
    rng = np.random.default_rng(seed)
    inner, cols = 60, 300
    blen = rng.integers(1, 4, inner)
    blen[0], blen[1] = 90, 0
    bptr = np.r_[0, np.cumsum(blen)].astype(np.int32)
    bidx = np.concatenate([np.sort(rng.choice(cols, n, replace=False)) for n in blen]).astype(np.int32)
    B = dbd.CSR(inner, cols, bptr, bidx, rng.standard_normal(bidx.size))
    arows = [np.sort(2 + rng.choice(inner - 2, rng.integers(1, 9), replace=False)) for _ in range(rows)]
    at = {"alternating": range(0, rows, 2), "one": [rows // 2], "none": [], "empty": []}[kind]
    for r in at:
        arows[r] = np.array([0, 5])
    if kind == "empty":
        for r in range(1, rows, 3):
            arows[r] = np.array([1])
    aptr = np.r_[0, np.cumsum([r.size for r in arows])].astype(np.int32)
    aidx = np.concatenate(arows).astype(np.int32)
    return dbd.CSR(rows, inner, aptr, aidx, rng.standard_normal(aidx.size)), B


def _same(C, A, B):
    Cp, Ci, Cv = oracle.spgemm(A, B)[:3]
    np.testing.assert_array_equal(C.row_ptr, Cp)
    np.testing.assert_array_equal(C.col_idx, Ci)
    tiny = np.repeat([np.diff(B.row_ptr)[A.col_idx[A.row_ptr[r]:A.row_ptr[r + 1]]].sum() <= 32
                      for r in range(A.n_rows)], np.diff(Cp))
    np.testing.assert_array_equal(C.val.view(np.uint64)[tiny], Cv.view(np.uint64)[tiny])


@pytest.mark.parametrize("rows", [1, 31, 32, 33, 64, 200])
@pytest.mark.parametrize("kind", ["alternating", "one", "none", "empty"])
def test_tiny_runs(rows, kind):
    A, B = _matrices(kind, rows, rows)
    with dbd.Context(cpu_gib=1, gpu_gib=4) as ctx:
        _same(ctx.spgemm(A, B).C, A, B)


def test_tiny_runs_of_a_batch():
    pairs = [_matrices(k, n, n) for k, n in (("none", 20), ("alternating", 45), ("empty", 13), ("none", 70))]
    with dbd.Context(cpu_gib=1, gpu_gib=4) as ctx:
        for C, (A, B) in zip(ctx.spgemm_batched([a for a, _ in pairs], [b for _, b in pairs]).C, pairs):
            _same(C, A, B)
