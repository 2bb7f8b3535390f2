"""A device reset between two engines of one process: the second one works,
whether the first was closed before the reset or not (a child process each;
the reset ends that process's own GPU context only)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes, os, sys
import numpy as np
from rtspmspm_b200 import Engine, gen

A = gen.erdos_renyi(9000, 9000, 40.0, 1)

def products(e):
    out = []
    for algo in ("plain", "learned"):
        C, _ = e.multiply(A, A, algo=algo)
        out.append(C.to_host())
        C.free()
    return out

e = Engine(0)
before = products(e)
if sys.argv[1] == "closed":
    e.close()
cu = ctypes.CDLL("libcuda.so.1")
dev = ctypes.c_int()
assert cu.cuDeviceGet(ctypes.byref(dev), 0) == 0
assert cu.cuDevicePrimaryCtxReset(dev) == 0
for _ in range(2):
    e2 = Engine(0)
    for x, y in zip(before, products(e2)):
        assert np.array_equal(x.row_ptr, y.row_ptr) and np.array_equal(x.col_idx, y.col_idx)
        assert np.array_equal(x.val.view(np.uint32), y.val.view(np.uint32))
    e2.close()
print("same", flush=True)
os._exit(0)  # nothing of the ended context is freed
"""


@pytest.mark.parametrize("first", ["closed", "open"])
def test_engine_after_a_device_reset(first):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CHILD, first], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("same"), r.stdout + r.stderr
