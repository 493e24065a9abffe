"""The standalone calls after a cudaDeviceReset: their scratch pool went with the context, and they go on with
another. In a process of its own, which holds nothing else on the GPU."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import ctypes
import torch                                   # maps the runtime library that resets the device
from bug_defense_b200 import _lib
rt = ctypes.CDLL([l.split()[-1] for l in open("/proc/self/maps") if "libcudart" in l][0])

def field(n):
    p = ctypes.c_void_p()
    assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(4 * n)) == 0
    assert rt.cudaMemset(p, 0, ctypes.c_size_t(4 * n)) == 0
    return p

def advance():
    from bug_defense_b200.ablation import plume_params_struct
    shape = (8, 8, 8)
    p = plume_params_struct(shape, 0.03, 0.03, 0.03, 1e-5, 1.0, 1.0, 0.0, 0.0, "as_given")
    a, b, flags = field(512), field(512), field(128)
    in_b = ctypes.c_int(0)
    for _ in range(3):
        _lib.call("bd_plume_advance", ctypes.byref(p), a, b, 3, flags, ctypes.byref(in_b), None)

advance()
for _ in range(2):
    assert rt.cudaDeviceReset() == 0
    advance()
print("done")
"""


def test_plume_advance_after_a_device_reset(gpu):
    r = subprocess.run([sys.executable, "-c", SCRIPT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("done"), (r.returncode, r.stdout, r.stderr[-2000:])
