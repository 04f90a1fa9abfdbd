"""Float32 values rounded on their way to the host: chunk sizes and
destinations off the 128-byte lines they are written in, and products of several
chunks, equal to rounding the FP64 product."""
import numpy as np
import pytest

import dbd_gb300 as dbd
from dbd_gb300 import generators as gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 33, 127, 1000, 4095, 70001])
def test_sizes(n):
    A = gen.banded(n, 1, n)
    with dbd.Context(cpu_gib=1, gpu_gib=4) as ctx:
        want = ctx.spgemm(A).C
    with dbd.Context(cpu_gib=1, gpu_gib=4, out_val_fp32=True) as ctx:
        got = ctx.spgemm(A, scope="d2h").C
    np.testing.assert_array_equal(got.row_ptr, want.row_ptr)
    np.testing.assert_array_equal(got.col_idx, want.col_idx)
    assert got.val.dtype == np.float32
    np.testing.assert_array_equal(got.val, want.val.astype(np.float32))


@pytest.mark.parametrize("fp32", [False, True])
def test_several_chunks(fp32):
    """A product of over 128 MiB of host bytes: more than one chunk, each at an odd offset."""
    A = gen.banded(150_001, 40, 7)
    with dbd.Context(cpu_gib=2, gpu_gib=8) as ctx:
        want = ctx.spgemm(A).C
    with dbd.Context(cpu_gib=2, gpu_gib=8, out_val_fp32=fp32) as ctx:
        res = ctx.spgemm(A, scope="d2h")
    assert res.stats["n_chunks"] > 1
    np.testing.assert_array_equal(res.C.row_ptr, want.row_ptr)
    np.testing.assert_array_equal(res.C.col_idx, want.col_idx)
    np.testing.assert_array_equal(res.C.val, want.val.astype(np.float32) if fp32 else want.val)
