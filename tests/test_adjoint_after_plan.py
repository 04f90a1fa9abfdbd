"""An adjoint behind a planned batch: the plan takes C's arrays over, so the
last multiply's pattern is computed again, for rows that a warp takes and for
rows that a CTA does."""
import ctypes

import numpy as np
import pytest

import dbd_gb300 as dbd
import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _device(m):
    t = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (m.row_ptr, m.col_idx, m.val)]
    torch.cuda.synchronize()
    return dbd.CSR.from_device(m.n_rows, m.n_cols, m.nnz, *(x.data_ptr() for x in t)), t


@pytest.mark.parametrize("per_row", [4, 40])
def test_adjoint_after_batch_plan(per_row):
    rng = np.random.default_rng(per_row)
    n = 3000
    idx = np.concatenate([np.sort(rng.choice(n, per_row, replace=False)) for _ in range(n)]).astype(np.int32)
    A = dbd.CSR(n, n, (np.arange(n + 1) * per_row).astype(np.int32), idx, rng.standard_normal(idx.size))
    Cp, Ci, Cv = oracle.spgemm(A)[:3]
    g = rng.standard_normal(Ci.size)
    dev, keep = _device(A)
    dg, da, db = torch.from_numpy(g).cuda(), *(torch.zeros(A.nnz, dtype=torch.float64, device="cuda") for _ in "ab")
    torch.cuda.synchronize()
    view = dev.view()[0]
    with dbd.Context(cpu_gib=1, gpu_gib=8) as ctx:
        ctx.spgemm(dev, scope="kernel", fetch=False)
        ctx.batch_plan([dev], capacity=8 * Ci.size)
        dbd._check(ctx._lib.dbd_spgemm_adjoint(ctx.handle, ctypes.byref(view), None, dg.data_ptr(), da.data_ptr(),
                                               db.data_ptr(), 1, 0), ctx.handle)
    wa, wb = oracle.adjoint(A, A, Cp, Ci, g)
    big = dbd.CSR(n, n, A.row_ptr, A.col_idx, np.abs(A.val))
    sa, sb = oracle.adjoint(big, big, Cp, Ci, np.abs(g))
    assert np.all(np.abs(da.cpu().numpy() - wa) <= 1e-12 * sa)
    assert np.all(np.abs(db.cpu().numpy() - wb) <= 1e-12 * sb)
    del keep
