"""fxb_last_timing's total is the device time of the subint's own kernels: of a
subint at the end of a queue of eight as of one alone, not the wait behind the
others."""
import pytest
import torch

from fxb200 import synth
from fxb200.native import Correlator
from helpers import small_job

pytestmark = pytest.mark.gpu

SUBINT = 32_000_000


def test_total_leaves_the_queue_out():
    job = small_job(nstation=10, nfreq=4, nchan=1024, full_pol=True, subint_ns=SUBINT)
    sub = synth.subint_inputs(job, 0, SUBINT, rho=0.05, seed=13)
    bufs = [torch.from_numpy(b).cuda() for b, _, _ in sub]
    args = ([b.data_ptr() for b in bufs], [b.numel() for b in bufs], [d for _, d, _ in sub], [n for _, _, n in sub], 0,
            SUBINT)
    torch.cuda.synchronize()
    corr = Correlator(job, xmac="fp16", inflight=8)
    for _ in range(24):                          # every slot's graphs are there
        corr.submit_device(*args)
    corr.sync()
    corr.submit_device(*args)
    alone = corr.timing()
    for _ in range(16):
        corr.submit_device(*args)
    f, x, total = corr.timing()
    corr.close()
    assert total >= f + x
    # a queue of eight: without the wait the preparation is all that is left over,
    # which beside other kernels takes at most about one subint's time
    assert total < 3 * alone[2], (alone, (f, x, total))
