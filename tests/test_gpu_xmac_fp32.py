"""The FP32 XMAC's tilings and time slices (csrc/fxb_xmac.cu) against the FP64
oracle: rows around its tiles of 3, 4 and 5 and around a CTA's share of the tile
pairs, few channels (slices over a cluster and over the warps of a CTA), fewer
times than slices, and channel counts below a CTA's 32.

Tolerance: FP32_TOL (1e-5, norm-wise; each sum has at most T products, every
addition within 2^-24).  The result is also the same on a second run, bit for
bit: the slices are added in a fixed order."""
import numpy as np
import pytest

from fxb200 import synth
from fxb200.native import Correlator
from helpers import compare_core, small_job

import fxoracle

pytestmark = pytest.mark.gpu

# stations (x 2 polarisations = rows), channels, subbands, FFTs
CASES = [(2, 16, 1, 5), (2, 64, 1, 400), (3, 32, 2, 97), (4, 256, 1, 64), (5, 128, 1, 3), (7, 64, 2, 33), (10, 64, 1, 40),
         (11, 32, 1, 21), (16, 16, 1, 12)]


@pytest.mark.parametrize("nstation,nchan,nfreq,nfft", CASES)
def test_slices_and_tiles_match_oracle(nstation, nchan, nfreq, nfft):
    job = small_job(nstation=nstation, nchan=nchan, nfreq=nfreq, full_pol=True, subint_ns=nfft * nchan * 1000 // 16)
    when = (0, 4_000_000)
    inputs = synth.subint_inputs(job, *when, rho=0.05, seed=8)
    corr = Correlator(job)
    corr.submit(inputs, *when)
    got = corr.results()
    corr.reset()
    corr.submit(inputs, *when)
    again = corr.results()
    layout, n = corr.layout(), corr.corelen
    corr.close()
    ref = fxoracle.OracleCorrelator(job).process_subint(inputs, *when)
    compare_core(job, layout, n, got, ref)
    assert np.array_equal(got, again)
