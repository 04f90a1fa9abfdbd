"""Assembly of a batch at the edges of the gather's tiles (2048 elements) and
of its 32-wide pair search: host and device pairs, empty ones among them."""
import numpy as np
import pytest

import dbd_gb300 as dbd

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _diagonal(n, seed):
    return dbd.CSR(n, n, np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32),
                   np.random.default_rng(seed).standard_normal(n))


@pytest.mark.parametrize("count", [1, 2, 31, 32, 33, 65, 300])
@pytest.mark.parametrize("where", ["host", "device"])
def test_pairs_land_where_they_belong(count, where):
    sizes = np.resize([2048, 0, 1, 2047, 2049, 4096, 5, 0, 0, 9000, 100], count)
    A = [_diagonal(int(n), q) for q, n in enumerate(sizes)]
    B = [_diagonal(int(n), q + 1000) for q, n in enumerate(sizes)]
    want = [a.val * b.val for a, b in zip(A, B)]
    keep = []
    if where == "device":
        def dev(m):
            t = [torch.from_numpy(x).cuda() for x in (m.row_ptr, m.col_idx, m.val)]
            keep.append(t)
            return dbd.CSR.from_device(m.n_rows, m.n_cols, m.val.size, *(x.data_ptr() or t[0].data_ptr() for x in t))
        A, B = [dev(m) for m in A], [dev(m) for m in B]
        torch.cuda.synchronize()
    with dbd.Context(cpu_gib=1, gpu_gib=8) as ctx:
        res = ctx.spgemm_batched(A, B)
    assert res.row_off.tolist() == np.r_[0, np.cumsum(sizes)].tolist() == res.nnz_off.tolist()
    for n, C, val in zip(sizes, res.C, want):
        np.testing.assert_array_equal(C.row_ptr, np.arange(n + 1))
        np.testing.assert_array_equal(C.col_idx, np.arange(n))
        np.testing.assert_array_equal(C.val, val)
