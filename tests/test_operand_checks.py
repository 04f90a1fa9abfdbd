"""Checks of device-resident operands before a multiply: sizes around the
check kernel's block, empty rows, one entry out of order anywhere, and every
malformed row_ptr or column refused."""
import numpy as np
import pytest

import dbd_gb300 as dbd
import oracle
from dbd_gb300 import generators as gen

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _device(m, offset=0):
    """The matrix on the device, its columns `offset` entries past an aligned address."""
    idx = np.concatenate([np.zeros(offset, np.int32), m.col_idx])
    t = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (m.row_ptr, idx, m.val)]
    t[1] = t[1][offset:]
    torch.cuda.synchronize()
    return dbd.CSR.from_device(m.n_rows, m.n_cols, m.nnz, *(x.data_ptr() for x in t)), t


def _square(n, lens, seed):
    """n x n with lens[r] columns in row r, ascending."""
    rng = np.random.default_rng(seed)
    idx = [np.sort(rng.choice(n, k, replace=False)) for k in lens]
    ptr = np.zeros(n + 1, np.int64)
    np.cumsum(lens, out=ptr[1:])
    return dbd.CSR(n, n, ptr.astype(np.int32), np.concatenate(idx).astype(np.int32), rng.standard_normal(int(ptr[-1])))


def _swap(m, row, at):
    """Entries at and at + 1 of a row exchanged (its order broken there)."""
    s = int(m.row_ptr[row]) + at
    for x in (m.col_idx, m.val):
        x[s], x[s + 1] = x[s + 1], x[s]


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("case", ["ascending", "first row", "last row", "long row's end", "row after empty rows"])
def test_order_of_every_row_is_seen(case, offset):
    n = 700
    lens = np.full(n, 3)
    lens[5:40] = 0
    lens[300] = 600  # longer than a block
    A = _square(n, lens, 1)
    if case == "first row":
        _swap(A, 0, 0)
    elif case == "last row":
        _swap(A, n - 1, 1)
    elif case == "long row's end":
        _swap(A, 300, 598)
    elif case == "row after empty rows":
        _swap(A, 40, 0)
    Cp, Ci, Cv, Ca = oracle.spgemm(A, with_abs=True)
    dev, keep = _device(A, offset)
    with dbd.Context(cpu_gib=1, gpu_gib=4) as ctx:
        C = ctx.spgemm(dev).C
    del keep
    np.testing.assert_array_equal(C.row_ptr, Cp)
    np.testing.assert_array_equal(C.col_idx, Ci)
    assert np.all(np.abs(C.val - Cv) <= 1e-12 * Ca)


@pytest.mark.parametrize("n", [1, 255, 256, 257])
@pytest.mark.parametrize("fault", ["first", "last", "decreases", "negative", "past the end", "column low", "column high"])
def test_malformed_device_operands_are_refused(n, fault):
    A = _square(n, np.full(n, 1), n)
    if fault == "first":
        A.row_ptr[0] = 1
    elif fault == "last":
        A.row_ptr[n] -= 1
    elif fault == "decreases":
        if n == 1:
            pytest.skip("one row cannot decrease without breaking its ends")
        A.row_ptr[n // 2] = n
    elif fault == "negative":
        A.row_ptr[n // 2] = -1
    elif fault == "past the end":
        A.row_ptr[(n + 1) // 2] = n + 7
    elif fault == "column low":
        A.col_idx[n - 1] = -1
    else:
        A.col_idx[n - 1] = n
    bad, keep = _device(A, n % 4)
    good, keep2 = _device(gen.banded(n, 1, 0))
    with dbd.Context(cpu_gib=1, gpu_gib=1) as ctx:
        for a, b in ((bad, None), (bad, good), (good, bad)):
            with pytest.raises(dbd.DBDError) as e:
                ctx.spgemm(a, b)
            assert "DBD_ERR_INVALID" in str(e.value)
            assert ("column" if "column" in fault else "row_ptr") in str(e.value)
        assert ctx.spgemm(good).C.n_rows == n
    del keep, keep2


def _bad(n):
    A = gen.banded(n, 1, 0)
    A.col_idx[-1] = n
    return A


def test_checks_are_read_with_the_first_results():
    """The operands' checks are waited for with the work estimate: A's fault is
    reported ahead of B's and of mismatched sizes, nothing is multiplied, and
    the context goes on working; the stage functions report them at once."""
    bad, keep = _device(_bad(300))
    good, keep2 = _device(gen.banded(300, 1, 0))
    other, keep3 = _device(gen.banded(200, 1, 0))
    with dbd.Context(cpu_gib=1, gpu_gib=1) as ctx:
        for a, b, text in ((bad, bad, "A: column"), (bad, other, "A: column"), (good, other, "inner dimensions"),
                           (good, bad, "B: column")):
            with pytest.raises(dbd.DBDError, match=text):
                ctx.spgemm(a, b)
        for load, name in ((ctx.initialize_A, "A"), (ctx.initialize_B, "B")):
            with pytest.raises(dbd.DBDError, match=f"{name}: column"):
                load(bad)
        with pytest.raises(dbd.DBDError, match="load A and B"):
            ctx.divide_Blocks()
        with pytest.raises(dbd.DBDError, match="a pair's column"):
            ctx.spgemm_batched([good, bad, good])
        ctx.initialize_A(good)
        ctx.initialize_B(good)
        ctx.divide_Blocks()
        ctx.distribute_Workload("kernel")
        first = ctx.result()
        np.testing.assert_array_equal(first.val, ctx.spgemm(good).C.val)
        assert ctx.spgemm_batched([good, good]).C[1].nnz == first.nnz
    del keep, keep2, keep3


def test_noalloc_refuses_malformed_operands():
    import ctypes
    from dbd_gb300 import _ffi
    bad, keep = _device(_bad(300))
    good, keep2 = _device(gen.banded(300, 1, 0))
    ptr = torch.empty(301, dtype=torch.int64, device="cuda")
    idx = torch.empty(3000, dtype=torch.int32, device="cuda")
    val = torch.empty(3000, dtype=torch.float64, device="cuda")
    nnz = ctypes.c_int64()
    for a, b, rc in ((bad, None, -1), (bad, good, -1), (good, bad, -1), (good, good, 0), (good, None, 0)):
        va, vb = a.view()[0], None if b is None else b.view()[0]
        got = _ffi.load().dbd_spgemm_noalloc(ctypes.byref(va), None if vb is None else ctypes.byref(vb), ptr.data_ptr(),
                                             idx.data_ptr(), val.data_ptr(), 3000, ctypes.byref(nnz), None)
        assert got == rc
        assert rc or nnz.value == 300 * 5 - 6
    del keep, keep2
