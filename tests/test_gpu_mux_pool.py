"""fxb_vdif_mux keeps its tables' memory mapped between calls: the device's free
memory does not grow at a synchronisation after a call (in a process of its own)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = r"""
import torch
from fxb200 import synth
from fxb200.native import vdif_mux_device
data = torch.from_numpy(synth.interlaced_vdif(nthreads=4, nframes=6, payload=1000, nbits=2, fps=1000, seed=5)).cuda()
out = torch.empty(6 * (4 * 1000 + 32), dtype=torch.uint8, device="cuda")
for _ in range(3):
    torch.cuda.synchronize()
    assert vdif_mux_device(data.data_ptr(), data.numel(), range(4), 1032, 1000, 2, out.data_ptr(), out.numel()) == out.numel()
    before = torch.cuda.mem_get_info()[0]
    torch.cuda.synchronize()
    after = torch.cuda.mem_get_info()[0]
    print("given back", after - before)
    assert after - before < 1 << 20
"""


def test_memory_stays_mapped():
    env = dict(os.environ, PYTHONPATH=os.pathsep.join(p for p in sys.path if p))
    r = subprocess.run([sys.executable, "-c", PROGRAM], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
