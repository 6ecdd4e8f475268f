"""The FP16 tensor-core XMAC (csrc/fxb_xmac_h.cu) against the FP64 oracle where
its shapes change: inputs around 12, 24 and 48 (blocks of 8, 4 and 2 channels, one
or two operand tiles, a tile per unit), odd inputs (padded rows), few channels with
many FFTs (time slices) and fewer FFTs than one K tile, FFT counts around 32.

Tolerance: TC_REL_TOL (1e-3, the tensor-core forms' gate on cross and auto norms
and on the rms amplitude and phase; the FP16 rounding of the spectra gives 5.5e-4).
A second run gives the same bits when every output is summed once per subint."""
import numpy as np
import pytest

from fxb200 import synth
from fxb200.native import Correlator
from helpers import assert_tc_gate, small_job, vis_errors

import fxoracle

pytestmark = pytest.mark.gpu

# stations, polarisations, channels, subbands, FFTs
CASES = [(2, 2, 16, 1, 2000), (3, 1, 32, 2, 33), (6, 2, 64, 1, 64), (7, 1, 64, 2, 31), (7, 2, 16, 1, 200),
         (12, 2, 32, 1, 96), (13, 2, 32, 1, 65), (24, 2, 16, 1, 70), (25, 2, 16, 1, 70), (32, 2, 16, 1, 64),
         (5, 2, 128, 1, 3)]


@pytest.mark.parametrize("nstation,npol,nchan,nfreq,nfft", CASES)
def test_shapes_match_oracle(nstation, npol, nchan, nfreq, nfft):
    from fxb200.job import Freq, full_job
    job = full_job(nstation, [Freq(8400.0 + 16 * k, 16.0, nchan) for k in range(nfreq)], pols="RL"[:npol],
                   full_pol=npol == 2, subint_ns=nfft * nchan * 1000 // 16)
    synth.make_delay_polys(job, seed=nstation)
    job.validate()
    when = (0, 4_000_000)
    inputs = synth.subint_inputs(job, *when, rho=0.3, seed=8)
    corr = Correlator(job, xmac="fp16")
    corr.submit(inputs, *when)
    got = corr.results()
    corr.reset()
    corr.submit(inputs, *when)
    again = corr.results()
    layout, n = corr.layout(), corr.corelen
    corr.close()
    ref = fxoracle.OracleCorrelator(job).process_subint(inputs, *when)
    e = vis_errors(job, layout, n, got, ref)
    print(e)
    assert_tc_gate(e)
    assert np.array_equal(got, again)
