"""The TMA-staged transpose: its first use under capture, and a wait that runs out."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FIRST_USE = """
import ctypes
import numpy as np, torch
from cytnx_b200 import _lib
from cytnx_b200.core import Type
m, n = 1024, 2056
x = torch.arange(m * n, device="cuda", dtype=torch.int32).to(torch.int16)
y = torch.zeros_like(x)
lib, shp, mp, off = _lib.lib(), np.array([m, n], dtype=np.uint64), np.array([1, 0], dtype=np.uint64), np.zeros(1, dtype=np.int64)
P, I = _lib.P_u64, _lib.P_i64
h = ctypes.c_void_p()
_lib.check(lib.ctn_permute_plan_create(Type.from_torch(x.dtype), 2, 1, shp.ctypes.data_as(P), off.ctypes.data_as(I),
                                       off.ctypes.data_as(I), mp.ctypes.data_as(P), ctypes.byref(h)))
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    _lib.check(lib.ctn_permute_plan_run(h, x.data_ptr(), y.data_ptr(), _lib.stream_ptr()))
g.replay()
torch.cuda.synchronize()
lib.ctn_permute_plan_destroy(h)
assert torch.equal(y.view(n, m), x.view(m, n).T)
print("captured")
"""


def test_first_use_in_a_process_may_be_captured():
    r = subprocess.run([sys.executable, "-c", FIRST_USE], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "captured" in r.stdout, r.stderr[-2000:]


def test_a_wait_that_runs_out_is_reported_once():
    """ctn_selftest_permute_timeout: waits that probe nothing; the copies in flight are waited for all the same."""
    import cytnx_b200 as c
    from cytnx_b200 import _lib

    lib = _lib.lib()
    for _ in range(2):
        rc = lib.ctn_selftest_permute_timeout(_lib.stream_ptr())
        assert rc == 4, (rc, lib.ctn_last_error())
        assert b"gave up waiting" in lib.ctn_last_error()
    x = torch.arange(1024 * 1040, device="cuda", dtype=torch.int32).to(torch.int16).view(1024, 1040)
    got = c.Tensor.from_torch(x).permute([1, 0]).contiguous().to_torch()
    assert torch.equal(got, x.T)
