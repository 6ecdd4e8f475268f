"""Device memory that a context holds."""
import ctypes
import glob
import os

import pytest
import torch

from fxb200.native import Correlator
from helpers import small_job

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _cudart():
    for p in glob.glob(os.path.join(os.path.dirname(torch.__file__), "..", "nvidia", "cuda_runtime", "lib", "libcudart.so*")):
        return ctypes.CDLL(p)
    return ctypes.CDLL("libcudart.so")


def used(rt) -> int:
    """bytes allocated from the device's default pool"""
    pool, v = ctypes.c_void_p(0), ctypes.c_uint64(0)
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    assert rt.cudaMemPoolGetAttribute(pool, 7, ctypes.byref(v)) == 0        # cudaMemPoolAttrUsedMemCurrent
    return v.value


def test_tensor_core_fft_holds_no_pair_constants(monkeypatch):
    # 64 two-band items x 4000 FFTs: 33 MB of constants in the CUDA-core F stage; the
    # tensor-core FFT's unit records (two items each) take about as much in one slot
    job = small_job(nstation=16, nchan=1024, bw=32.0, nfreq=4, subint_ns=128_000_000)
    rt = _cudart()
    assert rt.cudaSetDevice(0) == 0
    torch.cuda.synchronize()
    held = {}
    for env in ("0", "1"):
        monkeypatch.setenv("FXB_TC_FFT", env)
        before = used(rt)
        corr = Correlator(job, xmac="fp16", inflight=1)
        held[env] = used(rt) - before
        assert ("tensor-core FFT" in corr.tuning_report()) == (env == "1")
        corr.close()
    assert held["1"] - held["0"] < 16 * MB, held
