"""CTA rank rows (windows of at most 2^18 columns): window sizes around the
threads' quads of words and the kernel's limits, small and large rows, sorted
and unsorted B, with the symbolic pass's bitmap kept (dbd_spgemm) and rebuilt
(dbd_spgemm_noalloc)."""
import ctypes

import numpy as np
import pytest

import dbd_gb300 as dbd
import oracle
from dbd_gb300 import _ffi

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
RANKS, RANKL = 4, 5


def _from_rows(n_cols, rows, seed):
    ptr = np.zeros(len(rows) + 1, np.int64)
    np.cumsum([len(r) for r in rows], out=ptr[1:])
    idx = np.concatenate([np.asarray(r, np.int64) for r in rows]).astype(np.int32)
    return dbd.CSR(len(rows), n_cols, ptr.astype(np.int32), idx, np.random.default_rng(seed).standard_normal(idx.size))


def _noalloc(A, B, nnz):
    def dev(m):
        t = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (m.row_ptr, m.col_idx, m.val)]
        return t, dbd.CSR.from_device(m.n_rows, m.n_cols, m.nnz, *(x.data_ptr() for x in t)).view()[0]
    (ka, va), (kb, vb) = dev(A), dev(B)
    ptr = torch.empty(A.n_rows + 1, dtype=torch.int64, device="cuda")
    idx = torch.empty(nnz, dtype=torch.int32, device="cuda")
    val = torch.empty(nnz, dtype=torch.float64, device="cuda")
    got = ctypes.c_int64()
    torch.cuda.synchronize()
    dbd._check(_ffi.load().dbd_spgemm_noalloc(ctypes.byref(va), ctypes.byref(vb), ptr.data_ptr(), idx.data_ptr(),
                                              val.data_ptr(), nnz, ctypes.byref(got), None))
    return ptr.cpu().numpy(), idx.cpu().numpy(), val.cpu().numpy()


@pytest.mark.parametrize("words", [65, 66, 67, 1023, 1024, 1025, 2047, 2050, 4097, 8190, 8191, 8192])
@pytest.mark.parametrize("entries", [300, 4096, 4097, 60000])
@pytest.mark.parametrize("order", ["ascending", "shuffled"])
def test_rank_rows(words, entries, order):
    rng = np.random.default_rng(words + entries)
    off = 37  # the window starts inside a word
    lo, hi = 32 + off % 32, 32 * words + 31 - off % 7  # words 1 .. words
    want = min(entries, hi - lo - 1)
    pool = np.unique(np.r_[lo, hi, lo + rng.choice(hi - lo, want, replace=False)])
    # Three B rows that cover the pool, each column in one or two of them.
    part = rng.integers(0, 3, pool.size)
    rows = [pool[(part == q) | ((part == (q + 1) % 3) & (rng.random(pool.size) < 0.3))] for q in range(3)]
    if order == "shuffled":
        rows = [rng.permutation(r) for r in rows]
    B = _from_rows(hi + 1 + rng.integers(0, 3), rows + [rows[0][:0]], 1)
    A = _from_rows(4, [[0, 1, 2, 3], [2, 1, 0]], 2)
    with dbd.Context(cpu_gib=1, gpu_gib=8) as ctx:
        res = ctx.spgemm(A, B)
    Cp, Ci, Cv, Ca = oracle.spgemm(A, B, with_abs=True)
    if Cp[1] > 256:
        assert res.stats["rows_per_bin"][RANKS if Cp[1] <= 4096 else RANKL] == 2
    for ptr, idx, val in ((res.C.row_ptr, res.C.col_idx, res.C.val), _noalloc(A, B, int(Cp[-1]))):
        np.testing.assert_array_equal(ptr, Cp)
        np.testing.assert_array_equal(idx, Ci)
        assert np.all(np.abs(val - Cv) <= 1e-12 * Ca)
