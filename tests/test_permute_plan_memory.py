"""Preparing a block permutation without the memory for it is an error status, not an abort."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
RUN = """
import ctypes, resource, sys
import numpy as np
from cytnx_b200 import _lib
lib, n = _lib.lib(), 1_000_000  # about 96 MB of descriptors
shp, off = np.tile(np.array([3, 5], dtype=np.uint64), n), np.zeros(n, dtype=np.int64)
mp, h = np.array([1, 0], dtype=np.uint64), ctypes.c_void_p()
P, I = _lib.P_u64, _lib.P_i64
args = (3, 2, n, shp.ctypes.data_as(P), off.ctypes.data_as(I), off.ctypes.data_as(I), mp.ctypes.data_as(P))
vm = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (vm + (16 << 20), resource.RLIM_INFINITY))
one = lib.ctn_permute_plan_create(*args, ctypes.byref(h))
two = lib.ctn_permute_blocks(None, None, *args, None)  # fails before it looks at the tensors
resource.setrlimit(resource.RLIMIT_AS, (resource.RLIM_INFINITY, resource.RLIM_INFINITY))
text = lib.ctn_last_error()
print("status", one, two, h.value, text.decode())
"""


def test_out_of_host_memory():
    r = subprocess.run([sys.executable, "-c", RUN], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stderr[-1000:])
    assert "status 1 1 None" in r.stdout and "bad_alloc" in r.stdout, r.stdout
