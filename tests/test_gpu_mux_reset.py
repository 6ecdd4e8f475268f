"""fxb_vdif_mux on a thread that has called it before, after the program has reset
its own CUDA context: in a process of its own, buffers made anew, the same
bytes."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = r"""
import ctypes, glob, os, sys
import numpy as np
import torch
from fxb200 import synth
from fxb200.native import vdif_mux_device
path = glob.glob(os.path.join(os.path.dirname(torch.__file__), "..", "nvidia", "cuda_runtime", "lib", "libcudart.so*"))
rt = ctypes.CDLL(path[0] if path else "libcudart.so")
data = synth.interlaced_vdif(nthreads=4, nframes=6, payload=1000, nbits=2, fps=1000, seed=5)
cap = 6 * (4 * 1000 + 32)

def mux():
    din, dout = ctypes.c_void_p(0), ctypes.c_void_p(0)
    assert rt.cudaSetDevice(0) == 0
    assert rt.cudaMalloc(ctypes.byref(din), ctypes.c_size_t(data.size)) == 0
    assert rt.cudaMalloc(ctypes.byref(dout), ctypes.c_size_t(cap)) == 0
    assert rt.cudaMemcpy(din, ctypes.c_void_p(data.ctypes.data), ctypes.c_size_t(data.size), 1) == 0
    for _ in range(2):
        n = vdif_mux_device(din.value, data.size, range(4), 1032, 1000, 2, dout.value, cap)
    out = np.zeros(cap, dtype=np.uint8)
    assert rt.cudaMemcpy(ctypes.c_void_p(out.ctypes.data), dout, ctypes.c_size_t(cap), 2) == 0
    assert n == cap
    return out

first = mux()
assert rt.cudaDeviceReset() == 0
assert np.array_equal(first, mux())
print("same")
"""


def test_mux_after_a_reset_of_the_own_context():
    env = dict(os.environ, PYTHONPATH=os.pathsep.join(p for p in sys.path if p))
    r = subprocess.run([sys.executable, "-c", PROGRAM], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr
