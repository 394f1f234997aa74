"""The entry points after cudaDeviceReset, which ends the context that their scratch memory came
from: in a process of its own, through the C ABI alone."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

PROGRAM = r"""
import ctypes, sys
import numpy as np
from riptide_b200 import _lib
from oracle import oracle as O

lib = _lib.load()
rt = ctypes.CDLL([l.split()[-1] for l in open("/proc/self/maps") if "libcudart" in l][0])
x = np.random.default_rng(0).standard_normal((300, 251)).astype(np.float32)
y = np.random.default_rng(1).standard_normal(50003).astype(np.float32)

def call(fn, a, out, *args):
    d_in, d_out = ctypes.c_void_p(), ctypes.c_void_p()
    assert rt.cudaMalloc(ctypes.byref(d_in), ctypes.c_size_t(a.nbytes)) == 0
    assert rt.cudaMalloc(ctypes.byref(d_out), ctypes.c_size_t(out.nbytes)) == 0
    assert rt.cudaMemcpy(d_in, a.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(a.nbytes), 1) == 0
    _lib.check(fn(d_in, *args, d_out, None))
    assert rt.cudaMemcpy(out.ctypes.data_as(ctypes.c_void_p), d_out, ctypes.c_size_t(out.nbytes), 2) == 0
    assert rt.cudaFree(d_in) == 0 and rt.cudaFree(d_out) == 0
    return out

for turn in range(3):
    assert np.array_equal(call(lib.rt_ffa2, x, np.empty_like(x), 300, 251), O.C().ffa2(x))
    got = call(lib.rt_fast_running_median, y, np.empty(y.size), y.size, 2001, 101)
    assert np.array_equal(got, O.fast_running_median(y, 2001, 101))
    if turn == 1:
        _lib.check(lib.rt_release_scratch())
    assert rt.cudaDeviceReset() == 0
print("done")
"""


def test_scratch_after_a_reset():
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True,
                       timeout=120, env=dict(os.environ, PYTHONPATH=ROOT))
    assert r.returncode == 0 and "done" in r.stdout, r.stdout + r.stderr
