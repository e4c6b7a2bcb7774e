"""Planning needs the number of SMs and nothing else of a device: the same plan (and so the same order of sums) with and without one, and no
context on the device that a process only plans for."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import ctypes
from dandan_ops_b200 import _native
lib = _native.load()
shapes = [(m, n, k) for m in (1, 8, 16, 33, 64, 128, 200, 1000) for n in (48, 512, 1000, 2048, 4096, 5000, 6144, 12304) for k in (64, 776, 2048, 4096, 12288)]
print([(tuple(_native.plan(*s).values()), lib.b2_w4a16_workspace_bytes(*s)) for s in shapes])
driver = ctypes.CDLL("libcuda.so.1")
flags, active = ctypes.c_uint(), ctypes.c_int()
if driver.cuInit(0) == 0:
    assert driver.cuDevicePrimaryCtxGetState(0, ctypes.byref(flags), ctypes.byref(active)) == 0
assert active.value == 0, "planning made a context"
"""


def test_the_same_plans_without_a_device():
    outs = []
    for hidden in (False, True):
        env = dict(os.environ, CUDA_VISIBLE_DEVICES="" if hidden else os.environ.get("CUDA_VISIBLE_DEVICES", "0"))
        done = subprocess.run([sys.executable, "-c", CODE], env=env, capture_output=True, text=True, timeout=300)
        assert done.returncode == 0, done.stderr[-2000:]
        outs.append(done.stdout)
    assert outs[0] == outs[1] and len(outs[0]) > 1000
