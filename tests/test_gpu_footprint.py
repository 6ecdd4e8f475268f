"""fxb_job_footprint against the device memory that a context holds once its
staging slots have been used: never below it, and not far above.  Odd row counts
(padded rows of the tensor-core layout), time-sliced cross-multiplication, the
tensor-core FFT's records, two-subband items, FP8, phase cal, raw reads."""
import ctypes
import glob
import os

import numpy as np
import pytest
import torch

from fxb200 import serving, synth
from fxb200.native import Correlator
from fxb200.job import Freq, full_job
from helpers import mux_job, pcal_job, small_job, zoom_job

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


def one_pol(nstation, nfreq, nchan, bw, subint_ns):
    job = full_job(nstation, [Freq(8400.0 + bw * k, bw, nchan) for k in range(nfreq)], pols="R", full_pol=False,
                   subint_ns=subint_ns)
    synth.make_delay_polys(job, seed=1)
    job.validate()
    return job


JOBS = {
    "three_inputs": (lambda: one_pol(3, 16, 64, 8.0, 320_000_000), "fp16"),
    "two_inputs_fp32": (lambda: one_pol(2, 16, 32, 8.0, 64_000_000), "fp32"),
    "array_sliced": (lambda: small_job(nstation=32, nchan=32, bw=16.0, nfreq=1, full_pol=True, subint_ns=64_000_000), "fp16"),
    "one_row": (lambda: small_job(nstation=2, nchan=256, bw=16.0, nfreq=8, subint_ns=64_000_000), "fp16"),
    "three_rows": (lambda: small_job(nstation=3, nchan=512, bw=16.0, nfreq=4, subint_ns=64_000_000), "fp16"),
    "25_rows": (lambda: small_job(nstation=25, nchan=256, bw=16.0, nfreq=1, subint_ns=32_000_000), "bf16"),
    "sliced": (lambda: small_job(nstation=10, nchan=64, bw=16.0, nfreq=2, full_pol=True, subint_ns=64_000_000), "fp16"),
    "tc_fft": (lambda: small_job(nstation=8, nchan=1024, bw=32.0, nfreq=4, full_pol=True, subint_ns=32_000_000), "fp16"),
    "fp32": (lambda: small_job(nstation=8, nchan=64, bw=16.0, nfreq=4, full_pol=True, subint_ns=32_000_000), "fp32"),
    "fp8": (lambda: small_job(nstation=7, nchan=128, bw=16.0, nfreq=4, full_pol=True, subint_ns=32_000_000), "fp8"),
    "zoom": (lambda: zoom_job(subint_ns=65_536_000), "fp16"),
    "pcal": (lambda: pcal_job(nstation=3, nfreq=2, full_pol=True, subint_ns=32_768_000), "fp32"),
    "mux": (lambda: mux_job(subint_ns=32_768_000), "fp16"),
}


@pytest.mark.parametrize("name", sorted(JOBS))
@pytest.mark.parametrize("inflight", [2, 8])
def test_footprint_covers_the_context(name, inflight):
    make, xmac = JOBS[name]
    job = make()
    rt = _cudart()
    assert rt.cudaSetDevice(0) == 0
    torch.cuda.synchronize()
    # the sizes of a subint's windows count, not what is in them
    sub = []
    for s, st in enumerate(job.stations):
        nf, dsec, dns = synth.subint_window(job, s, 0, job.subint_ns)[1:4]
        sub.append((np.zeros(nf * (st.payload_bytes + st.header_bytes), dtype=np.uint8), dsec, dns))
    before = used(rt)
    corr = Correlator(job, xmac=xmac, inflight=inflight)
    for _ in range(inflight):
        corr.submit(sub, 0, job.subint_ns)
    corr.results()
    held = used(rt) - before
    corr.close()
    told = serving.job_footprint(job, xmac=xmac, inflight=inflight)
    assert held <= told <= 1.3 * held + 24 * MB, (held / MB, told / MB)


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
