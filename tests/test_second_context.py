"""A mixed-precision case in a second CUDA context of one process: kernel
attributes (the int8-slice product's 223 KB of shared memory among them) belong
to a context, so each case has to set them for its own.  In a child process,
without torch, so that no other library's state lives in the second context."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes, math
import numpy as np
import turbid_b200 as tb
from turbid_b200 import synthetic

P = dict(nx=24, ny=18, nz=33, nphase=2, precision="mixed", lx=4 * math.pi, ly=2 * math.pi, dt=2 * math.pi / 2000,
         reynolds=800.0, froude=1.0, averaged_concentration=1e-3, specific_gravity=2.65, bc_u=[1, 0, 0, 1, 0],
         bc_v=[1, 0, 0, 1, 0], schmidt=0.5, settling=5e-4, erosion_rate=1e-4, critical_shear=2e-4)

def fields():
    gc = tb.ChannelCase(**P)
    gc.upload_state(*synthetic.initial_state(seed=3, **P))
    assert gc.run_steps(2) == 2
    out = gc.download_state()
    gc.close()
    return out

first = fields()          # the primary context
cuda = ctypes.CDLL("libcuda.so.1")
dev, ctx, old = ctypes.c_int(), ctypes.c_void_p(), ctypes.c_void_p()
assert cuda.cuDeviceGet(ctypes.byref(dev), 0) == 0
assert cuda.cuCtxCreate_v2(ctypes.byref(ctx), 0, dev) == 0   # and current
second = fields()
assert cuda.cuCtxPopCurrent_v2(ctypes.byref(old)) == 0
assert cuda.cuCtxDestroy_v2(ctx) == 0
for a, b in zip(first, second):
    assert np.array_equal(a, b)
print("same fields")
"""


@pytest.mark.gpu
def test_mixed_case_in_a_second_context(cuda):
    env = dict(os.environ, PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same fields" in r.stdout, r.stderr[-2000:]
