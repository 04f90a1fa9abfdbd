"""Device slots of the +D2H scope with float32 values: 12 bytes an entry, as
with FP64 values, unless a device digest reads the floats there too."""
import numpy as np
import pytest

import dbd_gb300 as dbd

pytestmark = pytest.mark.gpu


def test_float32_chunks_are_as_large_as_fp64_ones():
    rng = np.random.default_rng(1)
    m, n = 65536, 64  # C is full: 4.2M entries, 50 MB, of which a 16 MiB budget holds a part
    A = dbd.CSR(m, 1, np.arange(m + 1, dtype=np.int32), np.zeros(m, np.int32), rng.standard_normal(m))
    B = dbd.CSR(1, n, np.array([0, n], np.int32), np.arange(n, dtype=np.int32), rng.standard_normal(n))
    want = np.outer(A.val, B.val)
    chunks = {}
    for fp32 in (False, True):
        with dbd.Context(cpu_gib=1, gpu_gib=1 / 64, out_val_fp32=fp32) as ctx:
            for digest in ((False, True, False) if fp32 else (False,)):
                ctx._lib.dbd_set_digest(ctx.handle, 1 if digest else 0)
                res = ctx.spgemm(A, B, scope="d2h")
                np.testing.assert_array_equal(res.C.val.reshape(m, n), want.astype(np.float32) if fp32 else want)
                chunks.setdefault((fp32, digest), set()).add(res.stats["n_chunks"])
    assert all(len(x) == 1 for x in chunks.values())
    plain, floats, digested = (chunks[k].pop() for k in ((False, False), (True, False), (True, True)))
    assert 4 <= plain == floats < digested
