"""The first call of ps_fit_batch_noalloc in a process takes no device memory
either: not for its buffers, and not for a larger local-memory arena, which the
runtime would take at the first launch of a kernel with a deep stack."""
from __future__ import annotations

import subprocess
import sys

import pytest

from conftest import GOLDEN, ROOT

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes as C, sys
import torch
from periodsearch_gb300 import FIT_DTYPE, Engine, _abi, read_input

eng = Engine(read_input(sys.argv[1]))
n, dev = 10, torch.device("cuda", 0)
p = torch.arange(1, n + 1, dtype=torch.int64, device=dev)
m = torch.arange(1, n + 1, dtype=torch.int32, device=dev)
out = torch.zeros(n * FIT_DTYPE.itemsize, dtype=torch.uint8, device=dev)
torch.cuda.synchronize()
before = torch.cuda.mem_get_info(0)[0]
st = eng._L.ps_fit_batch_noalloc(eng._ctx, eng.info.conw_r0, n, C.c_void_p(p.data_ptr()), C.c_void_p(m.data_ptr()),
                                 C.c_void_p(out.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream))
_abi.check(st, "ps_fit_batch_noalloc", eng._ctx)
torch.cuda.synchronize()
print("taken", before - torch.cuda.mem_get_info(0)[0])
"""


def test_first_call_takes_no_device_memory(engine_lib):
    r = subprocess.run([sys.executable, "-c", CHILD, str(GOLDEN / "tiny_mix" / "period_search_in")], cwd=ROOT,
                       capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split() == ["taken", "0"]
