"""Row lists per bin, row blocks' products and C's row pointers at the edges
of the 256-row tiles and of the tile scan's step (4096 tiles)."""
import numpy as np
import pytest

import dbd_gb300 as dbd
import oracle

pytestmark = pytest.mark.gpu


def _rows(m, n, seed):
    """Empty, tiny, warp and CTA rows mixed: lengths 0 to 40 over n columns."""
    rng = np.random.default_rng(seed)
    lens = rng.choice([0, 1, 2, 9, 40], m, p=[0.3, 0.4, 0.2, 0.08, 0.02])
    ptr = np.zeros(m + 1, np.int64)
    np.cumsum(lens, out=ptr[1:])
    step = n // 41
    pos = np.arange(ptr[-1]) - np.repeat(ptr[:-1], lens)
    idx = (pos * step + rng.integers(0, step, pos.size)).astype(np.int32)  # ascending and distinct in a row
    return dbd.CSR(m, n, ptr.astype(np.int32), idx, rng.standard_normal(idx.size))


@pytest.mark.parametrize("m", [1, 255, 256, 257, 8191, 8193, 4096 * 256, 4096 * 256 + 1])
@pytest.mark.parametrize("block", [256, 4096])
def test_lists_blocks_and_row_pointers(m, block):
    A, B = _rows(m, 1500, m), _rows(1500, 700, 1)
    with dbd.Context(cpu_gib=1, gpu_gib=8, rows_per_block=block) as ctx:
        ctx.initialize_A(A)
        ctx.initialize_B(B)
        nb = ctx.divide_Blocks()
        got, _ = ctx.block_info(nb)
        st = ctx.distribute_Workload("kernel")
        C = ctx.result()
    lens = np.diff(B.row_ptr)[A.col_idx]
    prod = np.add.reduceat(np.append(lens, 0), np.minimum(A.row_ptr[:-1], lens.size)) * (np.diff(A.row_ptr) > 0)
    assert nb == -(-m // block)
    np.testing.assert_array_equal(got, np.add.reduceat(prod, np.arange(0, m, block)))
    assert sum(st["rows_per_bin"]) == m and sum(st["sym_rows_per_bin"]) == m
    Cp, Ci, Cv, Ca = oracle.spgemm(A, B, with_abs=True)
    np.testing.assert_array_equal(C.row_ptr, Cp)
    np.testing.assert_array_equal(C.col_idx, Ci)
    assert np.all(np.abs(C.val - Cv) <= 1e-12 * Ca)
