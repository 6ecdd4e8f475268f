"""An error that is pending in the runtime when a subint is submitted is the
submit's to report, on a device that keeps up and on one that lags the caller;
a device that lags is no error."""
import ctypes

import pytest
import torch

from fxb200 import synth
from fxb200.native import Correlator, FxbError, lib
from helpers import small_job

pytestmark = pytest.mark.gpu

SUBINT = 32_000_000


@pytest.mark.parametrize("xmac", ["fp16", "fp32"])
@pytest.mark.parametrize("queued", [1, 3])
def test_pending_error_is_reported(xmac, queued):
    job = small_job(nstation=6, nfreq=2, nchan=1024, full_pol=True, subint_ns=SUBINT)
    sub = synth.subint_inputs(job, 0, SUBINT, rho=0.05, seed=13)
    bufs = [torch.from_numpy(b).cuda() for b, _, _ in sub]
    args = ([b.data_ptr() for b in bufs], [b.numel() for b in bufs], [d for _, d, _ in sub], [n for _, _, n in sub], 0,
            SUBINT)
    torch.cuda.synchronize()
    corr = Correlator(job, xmac=xmac, inflight=3)
    for _ in range(8):
        corr.submit_device(*args)
    corr.sync()
    for _ in range(queued):
        corr.submit_device(*args)
    # more page-locked memory than any host has: refused, and left pending
    st = ctypes.c_int32(0)
    assert not lib().fxb_host_alloc(1 << 60, ctypes.byref(st)) and st.value != 0
    with pytest.raises(FxbError):
        corr.submit_device(*args)
    corr.submit_device(*args)                    # reported once
    corr.sync()
    corr.close()
