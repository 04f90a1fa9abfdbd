"""Products of a warp row placed 32 a step: B rows that are empty among A's
entries (the owner is searched) or not (it is counted), around a step's
length, chunks of 31 to 33 and 65 entries, in the hashed, sorted, ranked and
flagged bins."""
import numpy as np
import pytest

import dbd_gb300 as dbd
import oracle

pytestmark = pytest.mark.gpu
LENGTHS = {"ones": [1], "twos and threes": [2, 3], "empty first": [0, 3], "empty between": [4, 0, 0, 1, 2],
           "empty last": [5, 1, 0], "a step": [33, 1, 31, 32]}


@pytest.mark.parametrize("lengths", list(LENGTHS))
@pytest.mark.parametrize("entries", [12, 31, 32, 33, 65])
@pytest.mark.parametrize("n_cols", [400, 2000, 300000])
def test_warp_walk(lengths, entries, n_cols):
    rng = np.random.default_rng(entries)
    pat = LENGTHS[lengths]
    lens = np.array([pat[i % len(pat)] for i in range(entries)])
    rows = [np.sort(rng.choice(n_cols, n, replace=False)) for n in lens]
    ptr = np.r_[0, np.cumsum(lens)].astype(np.int32)
    B = dbd.CSR(entries, n_cols, ptr, np.concatenate(rows).astype(np.int32), rng.standard_normal(ptr[-1]))
    A = dbd.CSR(3, entries, np.array([0, entries, 2 * entries, 3 * entries], np.int32),
                np.r_[rng.permutation(entries), np.arange(entries), np.arange(entries)[::-1]].astype(np.int32),
                rng.standard_normal(3 * entries))
    with dbd.Context(cpu_gib=1, gpu_gib=4) as ctx:
        res = ctx.spgemm(A, B)
    Cp, Ci, Cv, Ca = oracle.spgemm(A, B, with_abs=True)
    np.testing.assert_array_equal(res.C.row_ptr, Cp)
    np.testing.assert_array_equal(res.C.col_idx, Ci)
    assert np.all(np.abs(res.C.val - Cv) <= 1e-12 * Ca)
