"""Stations that record one polarisation after the other, so that the two bands of
a subband lie apart, against the FP64 oracle's Mode FFT output: in one 32-bit word
of a sample time and in words of their own, 2 and 8 bits, real and complex samples;
whole windows, windows with invalid frames, frames shorter than an eighth of the
window.  Interleaved complex bands (side by side) too.

Tolerances, per spectrum in the 2-norm, as of the two-band F stage (15 operations
within 2^-24 and the fast sine's 2^-21: 2e-6; FP16 spectra round once to 11 bits:
6e-4)."""
import numpy as np
import pytest

from fxb200 import synth
from fxb200.job import Freq, full_job
from fxb200.native import Correlator
from helpers import rel_err

import fxoracle

pytestmark = pytest.mark.gpu
TOL = {"fp32": 2e-6, "fp16": 6e-4}


def band_order_job(nchan, nfreq, nbits=2, apart=True, cplx=False, payload=8000, nfft=5, **kw):
    job = full_job(2, [Freq(8400.0 + 16 * k, 16.0, nchan, kw.get("sideband", "U")) for k in range(nfreq)],
                   full_pol=True, subint_ns=nfft * nchan * 1000 // 16, nbits=nbits,
                   fringe_rot_order=kw.get("order", 1))
    if apart:
        for st in job.stations:
            st.bands = [(f, p) for p in "RL" for f in range(nfreq)]
        for b in job.baselines:
            b.products = [(f, [((x % 2) * nfreq + f, (y % 2) * nfreq + f) for x, y in pp]) for f, pp in b.products]
    for st in job.stations:
        st.payload_bytes = payload
        st.complex_sampling = cplx
    synth.make_delay_polys(job, seed=6)
    job.validate()
    return job


CASES = [dict(nchan=16, nfreq=2), dict(nchan=128, nfreq=8), dict(nchan=1024, nfreq=8), dict(nchan=1024, nfreq=16),
         dict(nchan=2048, nfreq=2, order=2), dict(nchan=4096, nfreq=4, sideband="L"), dict(nchan=256, nfreq=2, nbits=8),
         dict(nchan=512, nfreq=2, nbits=8, sideband="L", order=0), dict(nchan=4096, nfreq=2, nbits=8),
         dict(nchan=1024, nfreq=4, payload=400), dict(nchan=1024, nfreq=16, payload=400), dict(nchan=2048, nfreq=2, payload=80),
         dict(nchan=32, nfreq=2, cplx=True), dict(nchan=512, nfreq=8, cplx=True), dict(nchan=2048, nfreq=16, cplx=True),
         dict(nchan=1024, nfreq=2, cplx=True, nbits=8, sideband="L"), dict(nchan=4096, nfreq=4, cplx=True, order=2),
         dict(nchan=256, nfreq=4, cplx=True, apart=False), dict(nchan=1024, nfreq=2, cplx=True, apart=False, nbits=8),
         dict(nchan=4096, nfreq=16, cplx=True, apart=False, sideband="L")]


@pytest.mark.parametrize("xmac", ["fp32", "fp16"])
@pytest.mark.parametrize("invalid", [False, True])
@pytest.mark.parametrize("kw", CASES, ids=lambda kw: "-".join("%s%s" % x for x in kw.items()))
def test_spectra_match_oracle(kw, invalid, xmac):
    job = band_order_job(**kw)
    sec, ns = 0, 4_000_000
    f0, nf = synth.subint_window(job, 0, sec, ns)[:2]
    bad = {0: list(range(f0 + nf // 3, f0 + nf, 4))} if invalid else None
    inputs = synth.subint_inputs(job, sec, ns, rho=0.05, seed=7, invalid=bad)
    corr = Correlator(job, xmac=xmac)
    corr.submit(inputs, sec, ns)
    freq = len(job.freqs) - 1
    spec = corr.spectra(freq)
    corr.close()
    orc = fxoracle.OracleCorrelator(job)
    seen = 0
    for s in range(2):
        buf, dsec, dns = inputs[s]
        for t in range(5):
            ref, w, _ = orc.mode_fft(s, buf, dsec, dns, sec, ns, t)
            for p, pol in enumerate("RL"):
                g, r = spec[t, 2 * s + p], ref[job.stations[s].bands.index((freq, pol))]
                if not np.any(r):
                    assert not np.any(g), (s, t, p)
                    continue
                seen += 1
                assert rel_err(g, r) < TOL[xmac], (s, t, p, w)
    assert seen >= 4
