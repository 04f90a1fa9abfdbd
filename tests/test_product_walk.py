"""Products of a CTA row placed 32 a step: B rows of one entry (32 starts a
step), around a step's length, longer than several steps, and empty ones
between them, over batches of entries around the CTAs' sizes."""
import numpy as np
import pytest

import dbd_gb300 as dbd
import oracle

pytestmark = pytest.mark.gpu
LENGTHS = {
    "ones": [1],
    "around a step": [31, 32, 33],
    "uneven": [1, 0, 2, 70, 1, 1, 0, 0, 5, 31, 1, 200, 32, 3],
    "long": [700, 1, 64],
}


@pytest.mark.parametrize("lengths", list(LENGTHS))
@pytest.mark.parametrize("entries", [31, 255, 256, 257, 511, 513, 1300])
@pytest.mark.parametrize("n_cols", [60000, 600000])  # one window, and several
def test_product_walk(lengths, entries, n_cols):
    rng = np.random.default_rng(entries)
    pat = LENGTHS[lengths]
    lens = np.array([pat[i % len(pat)] for i in range(entries)])
    rows = [np.sort(rng.choice(n_cols, n, replace=False)) for n in lens]
    ptr = np.r_[0, np.cumsum(lens)].astype(np.int32)
    B = dbd.CSR(entries, n_cols, ptr, np.concatenate(rows).astype(np.int32), rng.standard_normal(ptr[-1]))
    A = dbd.CSR(2, entries, np.array([0, entries, 2 * entries], np.int32),
                np.r_[rng.permutation(entries), np.arange(entries)].astype(np.int32), rng.standard_normal(2 * entries))
    with dbd.Context(cpu_gib=1, gpu_gib=8) as ctx:
        res = ctx.spgemm(A, B)
    Cp, Ci, Cv, Ca = oracle.spgemm(A, B, with_abs=True)
    np.testing.assert_array_equal(res.C.row_ptr, Cp)
    np.testing.assert_array_equal(res.C.col_idx, Ci)
    assert np.all(np.abs(res.C.val - Cv) <= 1e-12 * Ca)
