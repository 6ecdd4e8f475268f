"""The two-band F stage (csrc/fxb_fstage_pair.cuh) against the FP64 oracle's
Mode FFT output, at every length and along each of its branches: the passes'
schedules (last radix 2, 4 and 8; FFTs inside a warp, in part of a CTA, in CTAs
of 256, 512 and 1024 threads), both sidebands and all fringe-rotation orders,
frames longer and shorter than an eighth of the window (fast and general
reads), 2- and 8-bit fields of every position, and windows with invalid frames.

Tolerances, per spectrum in the 2-norm: FP32 spectra 2e-6 (FP32 arithmetic of
about 15 additions and products per value, each within 2^-24, and the fast
sine's 2^-21 absolute error on the rotators); FP16 spectra 6e-4 (one rounding
to 11 bits: 2^-12 of each value at most, 2.8e-4 in the norm)."""
import numpy as np
import pytest

from fxb200 import synth
from fxb200.native import Correlator
from helpers import corr_job, rel_err, small_job

import fxoracle

pytestmark = pytest.mark.gpu
TOL = {"fp32": 2e-6, "fp16": 6e-4}

# (channels, keywords): 2 nchan points
CASES = [(16, dict()), (32, dict(lsb=True)), (64, dict(order=2)), (128, dict(nbits=8)), (256, dict(order=0, lsb=True)),
         (512, dict(order=0)), (512, dict(lsb=True, nbits=8, nfreq=2)), (1024, dict(order=2, lsb=True)),
         (2048, dict()), (2048, dict(lsb=True, nbits=8)), (4096, dict(nbits=8, nfreq=2)), (4096, dict(order=0, lsb=True)),
         (256, dict(payload=40)), (2048, dict(payload=1000, nfreq=2)),
         (2048, dict(payload=200, nfreq=2)), (2048, dict(payload=80, nfreq=2, lsb=True)), (128, dict(invalid=True)),
         (1024, dict(invalid=True, nbits=8, nfreq=2)), (4096, dict(invalid=True)), (64, dict(nfreq=16))]


@pytest.mark.parametrize("xmac", ["fp32", "fp16"])
@pytest.mark.parametrize("nchan,kw", CASES)
def test_spectra_match_oracle(nchan, kw, xmac, monkeypatch):
    monkeypatch.setenv("FXB_TC_FFT", "0")       # 2048 points: this F stage, not the tensor-core FFT
    kw = dict(kw)
    payload, invalid = kw.pop("payload", 8000), kw.pop("invalid", False)
    nfft = max(3, 600 // nchan) | 1             # an odd count: a partly filled last unit
    job = small_job(nstation=2, nchan=nchan, bw=16.0, full_pol=True, subint_ns=nfft * nchan * 1000 // 16, seed=6, **kw)
    for st in job.stations:
        st.payload_bytes = payload
    job.validate()
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
        for t in sorted({0, 1, nfft // 2, nfft - 1}):
            ref, w, _ = orc.mode_fft(s, buf, dsec, dns, sec, ns, t)
            for p in range(2):
                g, r = spec[t, 2 * s + p], ref[2 * freq + p]
                if not np.any(r):
                    assert not np.any(g), (s, t, p)
                    continue
                seen += 1
                assert rel_err(g, r) < TOL[xmac], (s, t, p, w)
    assert seen >= 4


@pytest.mark.parametrize("nchan", [64, 2048])
def test_bands_with_their_own_rotations(nchan):
    """R/L clock deltas and phase offsets: the two bands' output rotators differ."""
    job = corr_job(nchan=nchan, nstation=2, subint_ns=4_096_000)
    sec, ns = 1, 500_000_000
    inputs = synth.subint_inputs(job, sec, ns, rho=0.05, seed=3)
    corr = Correlator(job)
    corr.submit(inputs, sec, ns)
    spec = corr.spectra(1)
    corr.close()
    orc = fxoracle.OracleCorrelator(job)
    for s in range(2):
        buf, dsec, dns = inputs[s]
        ref, _, _ = orc.mode_fft(s, buf, dsec, dns, sec, ns, 3)
        for p in range(2):
            assert rel_err(spec[3, 2 * s + p], ref[2 + p]) < TOL["fp32"], (s, p)


@pytest.mark.parametrize("xmac", ["fp32", "fp16"])
@pytest.mark.parametrize("nchan,nfreq,kw", [(16, 2, dict()), (128, 4, dict(fringe_rot_order=2)), (256, 1, dict()),
                                            (512, 2, dict(sideband="L")), (1024, 4, dict(sideband="L", nbits=8)),
                                            (1024, 2, dict(fringe_rot_order=0)), (2048, 2, dict(nbits=8)),
                                            (4096, 4, dict(sideband="L", fringe_rot_order=0))])
def test_single_bands_of_two_subbands(nchan, nfreq, kw, xmac):
    """Stations of one polarisation: two subbands of equal sideband make one item,
    whose bands have fringe rotations of their own (a subband alone and mixed
    sidebands stay single)."""
    from fxb200.job import Freq, full_job
    kw = dict(kw)
    side = kw.pop("sideband", "U")
    freqs = [Freq(8400.25 + 16 * k, 16.0, nchan, "U" if k == 3 and nchan == 128 else side) for k in range(nfreq)]
    job = full_job(2, freqs, pols="R", full_pol=False, subint_ns=3 * nchan * 1000 // 16, **kw)
    synth.make_delay_polys(job, seed=4)
    job.validate()
    sec, ns = 0, 4_000_000
    inputs = synth.subint_inputs(job, sec, ns, rho=0.05, seed=7)
    corr = Correlator(job, xmac=xmac)
    corr.submit(inputs, sec, ns)
    spec = [corr.spectra(f) for f in range(nfreq)]
    corr.close()
    orc = fxoracle.OracleCorrelator(job)
    for s in range(2):
        buf, dsec, dns = inputs[s]
        for t in range(3):
            ref, _, _ = orc.mode_fft(s, buf, dsec, dns, sec, ns, t)
            for f in range(nfreq):
                assert rel_err(spec[f][t, s], ref[f]) < TOL[xmac], (s, t, f)
