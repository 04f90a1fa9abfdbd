"""No check of a device operand reads outside its columns, whatever its
row_ptr holds.  The check kernels' own text is built for the host, where the
columns end at pages that cannot be read; on the GPU every entry point refuses
the same operands."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

import dbd_gb300 as dbd
from dbd_gb300 import generators as gen

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FENCED = r"""
#include "kernel_on_host.h"
#include <cstdio>
#include <cstdlib>
#include <sys/mman.h>
#include <vector>
// `n` columns with an unreadable page right behind them, or (front) before them.
static int32_t *fenced(long n, bool front) {
    const long page = 65536, bytes = (4 * n + page - 1) / page * page;
    char *p = (char *)mmap(nullptr, bytes + 2 * page, PROT_NONE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    mprotect(p + page, bytes, PROT_READ | PROT_WRITE);
    return (int32_t *)(front ? p + page : p + page + bytes - 4 * n);
}
"""

HARNESS = FENCED + r"""
%s
// argv: rows, columns that there are, front; then row_ptr.
int main(int argc, char **argv) {
    const int m = atoi(argv[1]), have = atoi(argv[2]);
    std::vector<int32_t> ptr;
    for (int i = 4; i < argc; ++i) ptr.push_back(atoi(argv[i]));
    CsrDev M;
    M.m = m;
    M.n = 1000;
    M.nnz = atoi(getenv("NNZ"));
    int32_t *idx = fenced(have, atoi(argv[3]));
    for (int i = 0; i < have; ++i) idx[i] = (have - i) %% 7;
    M.ptr = ptr.data();
    M.idx = idx;
    std::vector<int2> range(m);
    int badPtr = 0, badIdx = 0, unsorted = 0;
    each_thread(2, 256, [&] { k_check_operand(M, range.data(), &badPtr, &badIdx, &unsorted); });
    unsorted = 1;
    each_thread(2, 256, [&] { k_row_minmax(M, range.data(), &badPtr, &unsorted); });
    each_thread(2, 256, [&] { k_row_minmax(M, range.data(), nullptr, &unsorted); });
    std::vector<double> wide(M.nnz);
    each_thread(2, 256, [&] { k_f32_to_f64((const float *)idx, wide.data(), M.nnz, &badPtr); });
    printf("%%d %%d", badPtr, badIdx);
}
"""

# Two pairs of `have` entries; the second one's row_ptr does not end at its nnz.
GATHER = FENCED + r"""
struct BatchPair {
    int64_t m, nnz, ncols, nnzOff, colOff;
    int32_t shift;
    const int32_t *ptr, *idx;
    const double *val;
};
constexpr int kGatherThreads = 256, kGatherPerThread = 8, kGatherTile = 2048;
static int64_t first_pair(const int64_t *off, int64_t count, int64_t x) {
    int64_t q = count - 1;
    while (off[q] > x) --q;
    return q;
}
%s
int main(int argc, char **argv) {
    const int have = atoi(argv[1]), given = atoi(argv[2]);
    BatchPair p[2] = {};
    for (int q = 0; q < 2; ++q) {
        p[q].ncols = 7;
        p[q].nnz = q ? given : have;
        p[q].nnzOff = q ? have : 0;
        int32_t *idx = fenced(have, false);
        for (int i = 0; i < have; ++i) idx[i] = i %% 7;
        p[q].idx = idx;
        p[q].val = (const double *)fenced(2 * have, false);
    }
    const int64_t off[3] = {0, have, have + given};
    std::vector<int32_t> outIdx(off[2]);
    std::vector<double> outVal(off[2]);
    int bad = have != given;
    each_thread((int)((off[2] + kGatherTile - 1) / kGatherTile), kGatherThreads,
                [&] { k_batch_entries(p, off, 2, off[2], outIdx.data(), outVal.data(), &bad); });
    printf("%%d", bad);
}
"""


def _kernel(text, name):
    """A kernel's definition out of the source."""
    at = text.index("__global__", text.rindex("\n\n", 0, re.search(rf"\b{name}\(", text).start()))
    depth, i = 0, text.index("{", at)
    while True:
        depth += (text[i] == "{") - (text[i] == "}")
        i += 1
        if depth == 0:
            return text[at:i]


def _program(tmp, harness, source, kernels):
    with open(os.path.join(ROOT, "dbd_gb300", "csrc", source)) as f:
        text = f.read()
    src, exe = str(tmp / "kernels.cpp"), str(tmp / "kernels")
    with open(src, "w") as f:
        f.write(harness % "\n".join(_kernel(text, k) for k in kernels))
    subprocess.run(["g++", "-O1", "-std=c++17", "-w", "-I", os.path.join(ROOT, "tests", "helpers"), src, "-o", exe],
                   check=True)
    return exe


@pytest.fixture(scope="module")
def checks(tmp_path_factory):
    return _program(tmp_path_factory.mktemp("checks"), HARNESS, "k_analysis.cu",
                    ("k_check_operand", "k_row_minmax", "k_f32_to_f64"))


@pytest.fixture(scope="module")
def gather(tmp_path_factory):
    return _program(tmp_path_factory.mktemp("gather"), GATHER, "k_batch.cu", ("k_batch_entries",))


# Five rows over 20 entries; what a fault leaves of them.
GOOD = [0, 4, 8, 12, 16, 20]
FAULTS = {
    "well formed": GOOD,
    "far past the end": [0, 4, 1 << 30, 12, 16, 20],
    "far below": [0, 4, -(1 << 30), 12, 16, 20],
    "least": [0, 4, -(1 << 31), 12, 16, 20],
    "largest": [0, 4, (1 << 31) - 1, 12, 16, 20],
    "all far": [0, 1 << 30, 1 << 30, 1 << 30, 1 << 30, 20],
    "decreasing": [0, 20, 0, 20, 0, 20],
    "first": [1 << 20, 4, 8, 12, 16, 20],
    "last": [0, 4, 8, 12, 16, 1 << 30],
    "last negative": [0, 4, 8, 12, 16, -5],
}


@pytest.mark.parametrize("front", [0, 1])
@pytest.mark.parametrize("fault", sorted(FAULTS))
def test_checks_stay_inside_the_columns(checks, fault, front):
    ptr = FAULTS[fault]
    run = subprocess.run([checks, "5", "20", str(front)] + [str(x) for x in ptr], capture_output=True, text=True,
                         env=dict(os.environ, NNZ="20"))
    assert run.returncode == 0, f"ended by signal {-run.returncode}"
    assert run.stdout == ("0 0" if fault == "well formed" else "1 0")


@pytest.mark.parametrize("front", [0, 1])
@pytest.mark.parametrize("nnz", [19, 21, 24, 5000, 1 << 21])
def test_checks_read_no_more_entries_than_row_ptr_ends_at(checks, nnz, front):
    """Columns (and float32 values) are read only where row_ptr's end is the number of entries that was given."""
    run = subprocess.run([checks, "5", "20", str(front)] + [str(x) for x in GOOD], capture_output=True, text=True,
                         env=dict(os.environ, NNZ=str(nnz)))
    assert run.returncode == 0, f"ended by signal {-run.returncode}"
    assert run.stdout == "1 0"


@pytest.mark.parametrize("have, given", [(20, 20), (3000, 3000), (20, 21), (20, 4096), (3000, 9000), (3000, 2999)])
def test_gather_reads_no_more_entries_than_row_ptr_ends_at(gather, have, given):
    run = subprocess.run([gather, str(have), str(given)], capture_output=True, text=True)
    assert run.returncode == 0, f"ended by signal {-run.returncode}"
    assert run.stdout == str(int(have != given))


def _device(torch, m, row_ptr, nnz=None, fp32=False):
    val = m.val.astype(np.float32) if fp32 else m.val
    t = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (row_ptr.astype(np.int32), m.col_idx, val)]
    torch.cuda.synchronize()
    return dbd.CSR.from_device(m.n_rows, m.n_cols, nnz or m.nnz, *(x.data_ptr() for x in t), val_fp32=fp32), t


@pytest.mark.gpu
@pytest.mark.parametrize("fault", sorted(set(FAULTS) - {"well formed"}))
def test_entry_points_refuse_far_row_pointers(fault):
    """B's rows do not ascend, so that the unsorted operand's path is taken."""
    torch = pytest.importorskip("torch")
    from dbd_gb300 import _ffi
    rng = np.random.default_rng(1)
    ptr = np.array(GOOD, np.int32)
    idx = np.concatenate([rng.permutation(5)[:4] for _ in range(5)]).astype(np.int32)
    M = dbd.CSR(5, 5, ptr, idx, rng.standard_normal(20))
    good, keep = _device(torch, M, ptr)
    bad, keep2 = _device(torch, M, np.array(FAULTS[fault], np.int64))
    out = [torch.empty(n, dtype=t, device="cuda") for n, t in
           ((6, torch.int64), (25, torch.int32), (25, torch.float64))]
    grads = torch.zeros(2, 25, dtype=torch.float64, device="cuda")
    nnz = ctypes.c_int64()
    with dbd.Context(cpu_gib=1, gpu_gib=1) as ctx:
        want = ctx.spgemm(good).C
        for a, b in ((bad, None), (good, bad), (bad, good)):
            for call in (lambda: ctx.spgemm(a, b),
                         lambda: ctx.spgemm_batched([good, a], [good, b] if b is not None else None)):
                with pytest.raises(dbd.DBDError, match="row_ptr"):
                    call()
            va, vb = a.view()[0], None if b is None else b.view()[0]
            assert _ffi.load().dbd_spgemm_noalloc(
                ctypes.byref(va), None if vb is None else ctypes.byref(vb), out[0].data_ptr(), out[1].data_ptr(),
                out[2].data_ptr(), 25, ctypes.byref(nnz), None) == -1
        for load in (ctx.initialize_A, ctx.initialize_B):
            with pytest.raises(dbd.DBDError, match="row_ptr"):
                load(bad)
        ctx.spgemm(good, good)  # an adjoint on the kept pattern
        va, vb = bad.view()[0], good.view()[0]
        for x, y in ((va, vb), (vb, va)):
            assert ctx._lib.dbd_spgemm_adjoint(ctx.handle, ctypes.byref(x), ctypes.byref(y), out[2].data_ptr(),
                                               grads[0].data_ptr(), grads[1].data_ptr(), 1, 0) == -1
        again = ctx.spgemm(good).C
    np.testing.assert_array_equal(again.col_idx, want.col_idx)
    np.testing.assert_array_equal(again.val, want.val)
    del keep, keep2


@pytest.mark.gpu
@pytest.mark.parametrize("nnz", [19, 21, 1 << 21])
@pytest.mark.parametrize("fp32", [False, True])
def test_entry_points_refuse_another_number_of_entries(nnz, fp32):
    torch = pytest.importorskip("torch")
    from dbd_gb300 import _ffi
    M = gen.banded(7, 1, 0)
    M = dbd.CSR(7, 7, M.row_ptr, M.col_idx, np.ones(M.nnz))
    good, keep = _device(torch, M, M.row_ptr, fp32=fp32)
    bad, keep2 = _device(torch, M, M.row_ptr, nnz=nnz if nnz != M.nnz else nnz + 1, fp32=fp32)
    out = [torch.empty(n, dtype=t, device="cuda") for n, t in
           ((8, torch.int64), (49, torch.int32), (49, torch.float64))]
    count = ctypes.c_int64()
    with dbd.Context(cpu_gib=1, gpu_gib=1) as ctx:
        for a, b in ((bad, None), (good, bad), (bad, good)):
            with pytest.raises(dbd.DBDError, match="malformed row_ptr"):
                ctx.spgemm(a, b)
            if not fp32:
                va, vb = a.view()[0], None if b is None else b.view()[0]
                assert _ffi.load().dbd_spgemm_noalloc(
                    ctypes.byref(va), None if vb is None else ctypes.byref(vb), out[0].data_ptr(), out[1].data_ptr(),
                    out[2].data_ptr(), 49, ctypes.byref(count), None) == -1
        for load in (ctx.initialize_A, ctx.initialize_B):
            with pytest.raises(dbd.DBDError, match="malformed row_ptr"):
                load(bad)
        if not fp32:
            for b in (None, [good, good], [good, bad]):
                with pytest.raises(dbd.DBDError, match="a pair's row_ptr"):
                    ctx.spgemm_batched([good, bad], b)
            ctx.batch_plan([good, bad], [good, good], capacity=98)
            ctx.batch_enqueue()
            torch.cuda.synchronize()
            with pytest.raises(dbd.DBDError, match="a pair's row_ptr"):
                ctx.batch_result(fetch=False)
        assert ctx.spgemm(good).C.val.sum() == 5 * 9 + 2 * 4
    del keep, keep2
