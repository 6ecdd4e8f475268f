"""Where the F stage puts its values in the tensor-core spectra: blocks of 2 to 32
channels, rows of 1 to 50 inputs, four channels stored at once.  Items of one band
(one polarisation, one subband) and of two at every length, both sidebands, mirrored
(order-0 lower) bands, complex sampling, the tensor-core FFT, zoom windows.

Against the FP32 form's spectra of the same job, value by value: the same FP32
arithmetic in both but for contractions (1e-5 of the rms: five times 2e-6, the FP32
form's own tolerance), and one rounding to 11 bits (half a unit, 2^-12 of each
component, 2^-11 with the scale's margin)."""
import numpy as np
import pytest

from fxb200 import synth
from fxb200.job import Freq, full_job
from fxb200.native import Correlator
from helpers import ZOOMS, zoom_job

pytestmark = pytest.mark.gpu


def spectra(nstation, nchan, xmac, pols="R", nfreq=1, nbits=8, sideband="U", cplx=False, **kw):
    nfft = 3 if nchan > 64 else 67               # an odd count: a partly filled last unit
    freqs = [Freq(8400.25 + 16 * k, 16.0, nchan, sideband) for k in range(nfreq)]
    job = full_job(nstation, freqs, pols=pols, full_pol=False, subint_ns=nfft * nchan * 1000 // 16, nbits=nbits, **kw)
    for st in job.stations:
        st.complex_sampling = cplx
    synth.make_delay_polys(job, seed=4)
    job.validate()
    inputs = synth.subint_inputs(job, 0, 4_000_000, rho=0.05, seed=7)
    out = []
    for form in ("fp32", xmac):
        corr = Correlator(job, xmac=form)
        corr.submit(inputs, 0, 4_000_000)
        out.append([corr.spectra(f) for f in range(nfreq)])
        corr.close()
    return out


def compare(ref, got):
    for r, g in zip(ref, got):
        rms = np.sqrt(np.mean(np.abs(r) ** 2))
        assert rms > 0
        for x, y in ((r.real, g.real), (r.imag, g.imag)):
            assert np.all(np.abs(x - y) <= 2.0 ** -11 * np.abs(x) + 1e-5 * rms)


@pytest.mark.parametrize("nchan", [16, 32, 64, 128, 256, 512, 1024, 2048, 4096, 8192])
@pytest.mark.parametrize("kw", [dict(), dict(sideband="L"), dict(sideband="L", fringe_rot_order=0)])
def test_one_band(nchan, kw, monkeypatch):
    monkeypatch.setenv("FXB_TC_FFT", "0")
    compare(*spectra(3, nchan, "fp16", **kw))


@pytest.mark.parametrize("nstation,xmac", [(2, "fp16"), (13, "fp16"), (25, "bf16"), (50, "fp16"), (2, "fp8"), (5, "fp8"),
                                           (7, "fp8"), (9, "fp8"), (17, "fp8"), (25, "fp8"), (33, "fp8")])
@pytest.mark.parametrize("nchan", [16, 256])
def test_blocks(nstation, xmac, nchan):
    ref, got = spectra(nstation, nchan, xmac)
    if xmac != "bf16":
        compare(ref, got)
    else:                                        # 8 bits: 2^-9 of each component, 2^-8 with margin
        rms = np.sqrt(np.mean(np.abs(ref[0]) ** 2))
        for x, y in ((ref[0].real, got[0].real), (ref[0].imag, got[0].imag)):
            assert np.all(np.abs(x - y) <= 2.0 ** -8 * np.abs(x) + 1e-5 * rms)


@pytest.mark.parametrize("nstation", [3, 7, 13])
@pytest.mark.parametrize("nchan", [16, 32, 64, 128, 256, 512, 1024, 2048, 4096])
@pytest.mark.parametrize("kw", [dict(), dict(sideband="L"), dict(sideband="L", fringe_rot_order=0)])
def test_two_bands(nstation, nchan, kw, monkeypatch):
    monkeypatch.setenv("FXB_TC_FFT", "0")
    compare(*spectra(nstation, nchan, "fp16", pols="RL", **kw))


@pytest.mark.parametrize("nstation", [2, 3, 5, 8, 9, 13, 17])
@pytest.mark.parametrize("kw", [dict(), dict(sideband="L", fringe_rot_order=0), dict(cplx=True)])
def test_two_bands_of_fp8_blocks(nstation, kw):
    compare(*spectra(nstation, 64, "fp8", pols="RL", **kw))


@pytest.mark.parametrize("nchan", [32, 64, 128, 256, 512, 1024, 2048, 4096, 8192])
@pytest.mark.parametrize("sideband", ["U", "L"])
@pytest.mark.parametrize("nstation,pols", [(3, "R"), (7, "RL"), (13, "RL")])
def test_complex(nchan, sideband, nstation, pols):
    compare(*spectra(nstation, nchan, "fp16", pols=pols, sideband=sideband, cplx=True))


@pytest.mark.parametrize("nstation,pols,nfreq,xmac", [(2, "RL", 1, "fp16"), (6, "RL", 4, "fp16"), (7, "RL", 8, "fp16"),
                                                      (13, "RL", 2, "bf16"), (25, "RL", 2, "fp16"), (31, "RL", 1, "fp16"),
                                                      (32, "RL", 2, "fp16"), (3, "RL", 2, "fp8"), (5, "RL", 2, "fp8"),
                                                      (9, "RL", 2, "fp8"), (13, "RL", 2, "fp8"), (3, "R", 1, "fp16"),
                                                      (13, "R", 1, "fp16"), (9, "R", 1, "fp8")])
def test_tensor_core_fft(nstation, pols, nfreq, xmac):
    """The tensor-core FFT's stores.  In the 2-norm of each spectrum: FP16 samples,
    tables (twice), intermediate and output, each within 2^-12 (BF16 output: 2^-9)."""
    ref, got = spectra(nstation, 1024, xmac, pols=pols, nfreq=nfreq, nbits=2)
    tol = 5 * 2.0 ** -12 + (2.0 ** -9 if xmac == "bf16" else 0)
    for r, g in zip(ref, got):
        err = np.linalg.norm(g - r, axis=2) / np.linalg.norm(r, axis=2)
        assert err.shape == (3, nstation * len(pols)) and np.all(err <= tol), err.max()


@pytest.mark.parametrize("nstation,xmac", [(2, "fp16"), (3, "fp16"), (7, "fp16"), (13, "fp16"), (31, "fp16"), (2, "fp8"),
                                           (5, "fp8"), (9, "fp8"), (13, "fp8")])
def test_zoom_windows(nstation, xmac):
    """Zoom windows (at the start, inside and at the end of their subband) are copies
    of their parents' channels, in their own blocks."""
    job = zoom_job(nstation=nstation, subint_ns=16_000 * 11)
    inputs = synth.subint_inputs(job, 0, 4_000_000, rho=0.05, seed=7)
    out = []
    for form in ("fp32", xmac):
        corr = Correlator(job, xmac=form)
        corr.submit(inputs, 0, 4_000_000)
        out.append([corr.spectra(f) for f in range(len(job.freqs))])
        corr.close()
    compare(*out)
    for ref, got in zip(*out):
        assert ref.shape == got.shape
    for (parent, off, bw), z in zip(ZOOMS, range(2, 5)):
        c0, n = int(off * 16), int(bw * 16)
        for o in out:
            assert np.array_equal(o[z], o[parent][:, :, c0:c0 + n])
