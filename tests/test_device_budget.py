"""A context stays within its GPU budget when a deterministic adjoint, which
keeps its products between calls, and a multiply whose C nearly fills the
budget meet, in either order; the multiply keeps C on the device."""
import ctypes

import pytest

import dbd_gb300 as dbd
from dbd_gb300 import _ffi

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
GIB = 1 << 30


def _device(m, n, per_row, seed):
    """m x n with per_row columns a row, spread evenly."""
    g = torch.Generator("cuda").manual_seed(seed)
    first = torch.randint(n, (m, 1), device="cuda", generator=g)
    cols = ((first + torch.arange(per_row, device="cuda") * (n // per_row)) % n).sort(1).values
    t = [torch.arange(0, m * per_row + 1, per_row, dtype=torch.int32, device="cuda"), cols.flatten().to(torch.int32),
         torch.rand(m * per_row, dtype=torch.float64, device="cuda", generator=g)]
    torch.cuda.synchronize()
    return dbd.CSR.from_device(m, n, m * per_row, *(x.data_ptr() for x in t)), t


def _adjoint(ctx, a, g, flags):
    out = [torch.zeros(a.nnz, dtype=torch.float64, device="cuda") for _ in "ab"]
    v = a.view()[0]
    dbd._check(ctx._lib.dbd_spgemm_adjoint(ctx.handle, ctypes.byref(v), None, g.data_ptr(), out[0].data_ptr(),
                                           out[1].data_ptr(), 1, flags), ctx.handle)
    return out


def _nnz(ctx):
    """Entries of C, which is on the device."""
    o = _ffi.CsrOut()
    dbd._check(ctx._lib.dbd_result(ctx.handle, ctypes.byref(o)), ctx.handle)
    assert o.on_device
    return o.nnz


def _held(order):
    small, k1 = _device(8192, 8192, 44, 1)  # 15.9M products: 127 MB of them kept
    big, k2 = _device(9220, 2, 2, 2)  # a full C of 85M entries, 0.95 GiB
    wide, k3 = _device(2, 9220, 9220, 3)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    with dbd.Context(cpu_gib=1, gpu_gib=1) as ctx:
        grads = []
        for what in order:
            if what == "multiply":
                r = ctx.spgemm(big, wide, scope="kernel", fetch=False)
                assert r.stats["n_chunks"] == 1 and _nnz(ctx) == 9220 * 9220
            else:
                ctx.spgemm(small, scope="kernel", fetch=False)
                g = torch.ones(_nnz(ctx), dtype=torch.float64, device="cuda")
                torch.cuda.synchronize()
                grads = [_adjoint(ctx, small, g, f) for f in (2, 0)]
                for x, y in zip(*grads):
                    assert torch.all((x - y).abs() <= 1e-12 * y.abs())
                del g
        del grads
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        held = free - torch.cuda.mem_get_info()[0]
    del k1, k2, k3
    return held


@pytest.mark.parametrize("order", [("adjoint", "multiply"), ("multiply", "adjoint")])
def test_adjoint_and_multiply_share_the_budget(order):
    _held(order)  # kernels loaded, torch's own pools grown
    # Work arrays that the budget does not count, and the allocator's blocks.
    held = _held(order)
    assert held <= GIB + 48 * (1 << 20)
