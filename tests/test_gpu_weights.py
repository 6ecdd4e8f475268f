"""Weight sums (k_weights) against the oracle's sequential float sums, bit for
bit.  The kernel takes 2048 FFTs at a time: a chunk of whole and invalid FFTs, or a
run of 32 of them, is added by its count, other runs one by one.  Partly valid FFTs
at the start, at the end and between, in the first, a middle and the last chunk, FFT
counts around the runs' 32 and the chunks' 2048, several subints (a sum that is no
whole number carried into clean chunks), and stations of several threads, whose sums
are per band and read with a stride."""
import numpy as np
import pytest

from fxb200 import synth
from fxb200.native import Correlator
from helpers import mux_job, regions, small_job

import fxoracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nfft", [1, 31, 33, 128, 129, 300])
@pytest.mark.parametrize("bad", [(), (0,), (1, 2), (-1,), (0, 3, -2)])
def test_weight_sums_are_exact(nfft, bad):
    job = small_job(nstation=3, nchan=512, bw=16.0, full_pol=True, subint_ns=nfft * 32_000)
    for st in job.stations:
        st.payload_bytes = 1000                  # frames of 2000 samples, about two windows
    job.validate()
    check_sums(job, nfft, lambda nf: {1: [b % nf for b in bad]})


# invalid frames by the part of the subint that they lie in: first, middle, last chunk
PARTS = {"none": (), "first": (0.01,), "middle": (0.5,), "last": (0.995,), "all": (0.01, 0.4, 0.5, 0.6, 0.995)}


@pytest.mark.parametrize("nfft", [2047, 2048, 2049, 4100])
@pytest.mark.parametrize("part", sorted(PARTS))
@pytest.mark.parametrize("threads", [False, True])
def test_chunks_of_many_ffts(nfft, part, threads):
    make = mux_job if threads else small_job
    job = make(nstation=3, nchan=16, bw=16.0, nfreq=1, full_pol=True, subint_ns=nfft * 1000)
    for st in job.stations:
        st.payload_bytes = 40                    # frames of 80 samples, two and a half windows of 32
    job.validate()
    frames = lambda nf: [int(f * nf) for f in PARTS[part]]
    check_sums(job, nfft, lambda nf: {0: frames(nf)[:1], 1: frames(nf)})


def check_sums(job, nfft, bad):
    corr, orc, ref = Correlator(job), fxoracle.OracleCorrelator(job), None
    for k in (1, 2):
        sec, ns = divmod(4_000_000 + k * job.subint_ns, 1_000_000_000)
        f0, nf = synth.subint_window(job, 1, sec, ns)[:2]
        invalid = {s: [f0 + b for b in frames] for s, frames in bad(nf).items()}
        inputs = synth.subint_inputs(job, sec, ns, rho=0.05, seed=5, invalid=invalid)
        flags = [None, None, synth.valid_flags(job, invalid_ffts=[nfft // 2])]
        corr.submit(inputs, sec, ns, validflags=flags)
        full = [synth.valid_flags(job) if f is None else f for f in flags]
        ref = orc.process_subint(inputs, sec, ns, validflags=full, coreresult=ref)
    got, layout, n = corr.results(), corr.layout(), corr.corelen
    corr.close()
    for name, sl in regions(job, layout, n):
        if "weight" in name:
            assert np.array_equal(got[sl], ref[sl].astype(np.float32)), name
