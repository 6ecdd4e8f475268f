"""Preparation kernels beside the last subints' F stage and XMAC.

A context whose device lags the caller runs a subint's preparation on a second
stream, against the slot's own parameters.  Forty subints queued without a wait,
a delay model changed on the way, must give what one kernel after the other gives,
bit for bit: with two and three slots, with longer buffers than the arrays were
sized for, and with the context's stream in the caller's hands.  The context's
report tells how many subints took which way: enough of them, on both sides of the
new delay model, that every slot's graph without the preparation was replayed."""
import ctypes
import re

import numpy as np
import pytest
import torch

from fxb200 import synth
from fxb200.native import Correlator, check, lib, poly_arrays
from helpers import small_job

pytestmark = pytest.mark.gpu

SUBINT = 32_000_000
NSUB, CHANGE = 40, 20


def beside(corr):
    n, of = re.search(r"preparation: (\d+) of (\d+) subints", corr.tuning_report()).groups()
    return int(n), int(of)


@pytest.mark.parametrize("inflight,exposed,extra", [(2, False, 0), (3, False, 0), (3, True, 0), (3, False, 1)])
def test_queued_subints_match_serial(inflight, exposed, extra):
    # 24 stations, four recordings among them: about 0.4 ms of kernels a subint, several
    # times what a submit takes
    job = small_job(nstation=24, nfreq=4, nchan=1024, full_pol=True, subint_ns=SUBINT)
    four = small_job(nstation=4, nfreq=4, nchan=1024, full_pol=True, subint_ns=SUBINT)
    inputs = [synth.subint_inputs(four, 0, SUBINT * k, rho=0.05, seed=13 + k) for k in (1, 2)]
    npoly, order, p0, interval, coeffs = poly_arrays(job, 2)
    moved = np.ascontiguousarray(coeffs).copy()
    moved.reshape(npoly, -1)[:, 0] += 0.25

    def run(graphs):
        corr = Correlator(job, xmac="fp16", inflight=inflight)
        corr.set_graphs(graphs)
        if exposed:
            assert corr.stream()
        dev = []
        for sub in inputs:
            bufs = [torch.from_numpy(np.ascontiguousarray(b)).cuda() for b, _, _ in sub]
            if extra:       # each station's buffer three times over: more frames than a subint's
                bufs = [torch.cat([b, b, b]) for b in bufs]
            dev.append(([bufs[s % 4] for s in range(24)], [sub[s % 4][1] for s in range(24)],
                        [sub[s % 4][2] for s in range(24)]))
        torch.cuda.synchronize()
        count = []
        for i in range(NSUB):
            if i == CHANGE:
                count.append(beside(corr)[0])
                check(lib().fxb_set_delay_poly(corr.ctx, 2, npoly, order, p0, interval,
                                               moved.ctypes.data_as(ctypes.POINTER(ctypes.c_double))), corr.ctx, "delay")
            bufs, dsec, dns = dev[i & 1]
            corr.submit_device([b.data_ptr() for b in bufs], [b.numel() for b in bufs], dsec, dns, 0,
                               SUBINT * (1 + (i & 1)))
        n, of = beside(corr)
        assert of == NSUB
        count.append(n - count[0])
        out, weights = corr.results(), corr.fft_weights()
        times = corr.timing()
        corr.close()
        return out, weights, times, count

    a, wa, _, none = run(False)
    b, wb, times, count = run(True)
    assert none == [0, 0]
    if exposed:
        assert count == [0, 0]
    else:
        assert min(count) >= 2 * inflight, count
    assert np.abs(a).max() > 0
    assert np.array_equal(a, b)
    assert np.array_equal(wa, wb)
    assert all(t > 0 for t in times)
