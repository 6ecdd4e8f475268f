"""Weight sums (k_weights) against the oracle's sequential float sums, bit for
bit: runs of whole and of invalid FFTs (added by their count), runs with partly
valid FFTs (added one by one) at the start, at the end and around the runs' 32 and
128 FFTs, and several subints."""
import numpy as np
import pytest

from fxb200 import synth
from fxb200.native import Correlator
from helpers import regions, small_job

import fxoracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nfft", [1, 31, 33, 128, 129, 300])
@pytest.mark.parametrize("bad", [(), (0,), (1, 2), (-1,), (0, 3, -2)])
def test_weight_sums_are_exact(nfft, bad):
    job = small_job(nstation=3, nchan=512, bw=16.0, full_pol=True, subint_ns=nfft * 32_000)
    for st in job.stations:
        st.payload_bytes = 1000                  # frames of 2000 samples, about two windows
    job.validate()
    corr, orc, ref = Correlator(job), fxoracle.OracleCorrelator(job), None
    for k in (1, 2):
        sec, ns = divmod(4_000_000 + k * job.subint_ns, 1_000_000_000)
        f0, nf = synth.subint_window(job, 1, sec, ns)[:2]
        inputs = synth.subint_inputs(job, sec, ns, rho=0.05, seed=5, invalid={1: [f0 + b % nf for b in bad]})
        flags = [None, None, synth.valid_flags(job, invalid_ffts=[nfft // 2])]
        corr.submit(inputs, sec, ns, validflags=flags)
        full = [synth.valid_flags(job) if f is None else f for f in flags]
        ref = orc.process_subint(inputs, sec, ns, validflags=full, coreresult=ref)
    got, layout, n = corr.results(), corr.layout(), corr.corelen
    corr.close()
    for name, sl in regions(job, layout, n):
        if "weight" in name:
            assert np.array_equal(got[sl], ref[sl].astype(np.float32)), name
