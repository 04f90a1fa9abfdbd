"""The allocation-free entry point's first call in a process, which sets the
device up: on a capturing stream it is refused and the capture goes on."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = r"""
import ctypes, sys
import torch
import dbd_gb300 as dbd
from dbd_gb300 import _ffi, generators as gen

M = gen.banded(300, 1, 0)
t = [torch.from_numpy(x).cuda() for x in (M.row_ptr, M.col_idx, M.val)]
view = dbd.CSR.from_device(300, 300, M.nnz, *(x.data_ptr() for x in t)).view()[0]
out = [torch.empty(n, dtype=d, device="cuda") for n, d in
       ((301, torch.int64), (3000, torch.int32), (3000, torch.float64))]
held = torch.zeros(4, device="cuda")
lib = _ffi.load()
nnz = ctypes.c_int64()
stream = torch.cuda.Stream()
torch.cuda.synchronize()

def call(s):
    return lib.dbd_spgemm_noalloc(ctypes.byref(view), None, out[0].data_ptr(), out[1].data_ptr(), out[2].data_ptr(),
                                  3000, ctypes.byref(nnz), s.cuda_stream)

graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph, stream=stream, capture_error_mode="MODE"):
    held.add_(1)  # the capture holds something
    first = call(stream)
graph.replay()
torch.cuda.synchronize()
assert held.tolist() == [1.0] * 4, held
assert first == -1, first
assert call(stream) == 0 and nnz.value == 300 * 5 - 6
print("done")
"""


@pytest.mark.parametrize("mode", ["global", "thread_local"])
def test_first_call_during_a_capture(mode):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    text = PROGRAM.replace("MODE", mode)
    run = subprocess.run([sys.executable, "-c", text], cwd=root, capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and run.stdout.endswith("done\n"), run.stderr[-2000:]
