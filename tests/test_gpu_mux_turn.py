"""The corner turn of fxb_vdif_mux against numpy, byte for byte: the index
permutation (2, 4, 8, 16 threads of 1, 2, 4, 8-bit fields) and the general form
(other thread counts and widths), output buffers of 32-, 16- and 4-byte
alignment, and word counts that leave a CTA partly filled."""
import numpy as np
import pytest
import torch

from fxb200 import synth
from fxb200.native import vdif_mux_device

pytestmark = pytest.mark.gpu

CASES = [(nt, nb, 1000, 0) for nt in (2, 4, 8, 16) for nb in (1, 2, 4, 8) if nt * nb <= 32] + \
        [(1, 2, 1000, 0), (3, 2, 1000, 0), (5, 4, 1000, 0), (32, 1, 1000, 0), (16, 2, 8, 0), (16, 2, 520, 16),
         (16, 2, 24, 4), (8, 2, 40, 16), (4, 2, 5000, 4)] + \
        [(1, 1, 1000, 0), (1, 3, 1000, 4), (1, 16, 40, 0), (2, 16, 1000, 0), (2, 3, 1000, 4), (4, 6, 1008, 0),
         (4, 7, 1000, 4), (8, 3, 992, 0), (8, 3, 1000, 16)]


@pytest.mark.parametrize("nthreads,nbits,payload,off", CASES)
def test_corner_turn(nthreads, nbits, payload, off):
    nframes, fps = 5, 1000
    data = synth.interlaced_vdif(nthreads=nthreads, nframes=nframes, payload=payload, nbits=nbits, fps=fps, seed=payload + nthreads)
    fb = payload + 32
    din = torch.from_numpy(data).cuda()
    ofb = payload * nthreads + 32
    dout = torch.full((nframes * ofb + off,), 0xAB, dtype=torch.uint8, device="cuda")[off:]
    n = vdif_mux_device(din.data_ptr(), data.size, list(range(nthreads)), fb, fps, nbits, dout.data_ptr(), dout.numel())
    assert n == nframes * ofb
    got = dout.cpu().numpy().reshape(nframes, ofb)
    frames = data.reshape(-1, fb)
    heads = frames[:, :32].copy().view(np.uint32)
    ids, times = (heads[:, 3] >> 16) & 0x3FF, heads[:, 1] & 0xFFFFFF
    spow = 32 // nbits // nthreads                    # steps of a thread per output word
    shifts = np.arange(32 // nbits, dtype=np.uint64) * nbits
    for k in range(nframes):
        words = np.stack([frames[(ids == t) & (times == times.min() + k)][0, 32:].copy().view(np.uint32)
                          for t in range(nthreads)])
        codes = (words[:, :, None].astype(np.uint64) >> shifts) & ((1 << nbits) - 1)      # thread, word, step
        codes = codes[:, :, :spow * nthreads].reshape(nthreads, -1, nthreads, spow)       # thread, word, j, step
        out = np.zeros((words.shape[1], nthreads), dtype=np.uint64)
        for kk in range(spow):
            for t in range(nthreads):
                out |= codes[t, :, :, kk] << np.uint64((kk * nthreads + t) * nbits)
        assert np.array_equal(got[k, 32:].copy().view(np.uint32), out.reshape(-1).astype(np.uint32)), k
