"""The work that users of fxb200 have it do, as cases to be timed.

Every case goes through the package's public entry points on seeded synthetic
recordings: a sky signal common to all stations, delayed by each station's own
delay polynomial, plus station noise, quantised to 2 or 8 bits and framed as
VDIF the way a DataStream's receive ring holds it (the subints of a pass are
windows of one run of frames per station).  A pass is one integration: zero the
accumulators, submit its subints, read the core result.

Kinds: "corr" (recordings in device memory, result left in device memory),
"host" (page-locked host memory in, host memory out), "batch" (one context per
subband shape, submitted together) and "mux" (multi-thread VDIF to
single-thread frames).
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "difx-svn2git-try3_b200"))

from fxb200 import configs  # noqa: E402
from fxb200.job import DelayPoly, Freq, add_zoom_bands, full_job  # noqa: E402
from fxb200.native import Batch, Correlator, pinned_empty, vdif_mux_device  # noqa: E402

CORR = dict(kind="corr", nstation=10, nfreq=8, bw=32.0, nchan=1024, npol=2, full_pol=True, nbits=2, lsb=False,
            order=1, avg=1, subint_ns=8_000_000, nsub=1, xmac="fp16", payload=8000, invalid=0.0, pcal=0.0,
            zoom=False, raw=False, cplx=False)


def _corr(name, **kw):
    return dict(CORR, name=name, **kw)


def listed():
    return [
        # the smallest job the tests and the smoke run use as a unit: four stations, one band pair, a
        # single subint in the default arithmetic, as a fringe check during an observation asks for
        _corr("fringe_check_4st", nstation=4, nfreq=1, bw=16.0, nchan=256, full_pol=False, xmac="fp32"),
        # the 10-station production workload of the benchmark in its headline arithmetic (0.128 s)
        _corr("production_10st_fp16", nsub=16),
        # the same workload in the default arithmetic
        _corr("production_10st_fp32", nsub=4, xmac="fp32"),
        # the same workload end to end: host memory in, core result in host memory
        _corr("production_10st_host", kind="host", nsub=8),
        # spectral-line shape of the uneven observation: wide 8-bit subband, 15.6 kHz channels
        _corr("line_4096ch_8bit", nstation=20, nfreq=1, bw=64.0, nchan=4096, nbits=8, subint_ns=8_192_000, nsub=4),
        # continuum shape of the uneven observation: wide subbands, coarse channels
        _corr("continuum_128ch", nstation=20, nfreq=4, bw=64.0, nchan=128, subint_ns=8_192_000, nsub=2),
        # the uneven observation as a whole: 20 stations, 16 subbands of mixed width, channels and bits
        dict(kind="batch", name="uneven_20st_batch", nstation=20, nsubband=16, plan=3, nsub=4, xmac="fp16"),
        # the largest array the serving workload takes: 32 dual-polarisation stations, full cross hands
        _corr("array_32st", nstation=32, nfreq=4, nsub=4),
        # geodesy: an odd number of stations, narrow lower-sideband bands of one polarisation, phase-cal
        # tones, 5000-byte frames, some of them invalid, default arithmetic, channels averaged on output
        _corr("geodesy_7st", nstation=7, nfreq=16, bw=8.0, nchan=64, npol=1, full_pol=False, lsb=True, avg=2,
              subint_ns=16_040_000, nsub=3, xmac="fp32", payload=5000, invalid=0.01, pcal=1.0),
        # spectral line with zoom windows beside the parent bands, quadratic fringe rotation
        _corr("zoom_5st", nstation=5, nfreq=2, bw=16.0, nchan=2048, order=2, subint_ns=10_240_000, nsub=4, zoom=True),
        # the production workload recorded as 16 threads of one channel, read raw
        _corr("threads_10st_raw", nsub=4, payload=128000, raw=True),
        # one read of the same recording muxed to single-thread frames
        dict(kind="mux", name="mux_16_threads", nthread=16, nframe=1000, payload=8000, nbits=2),
    ]


def draw(rng):
    u = rng.random()
    if u < 0.08:
        nthread = rng.choice([2, 4, 8, 16])
        return dict(kind="mux", nthread=nthread, payload=rng.choice([5000, 8000]), nbits=2,
                    nframe=int(math.exp(rng.uniform(math.log(20), math.log(16000 // nthread)))))
    if u < 0.16:
        return dict(kind="batch", nstation=rng.randint(2, 20), nsubband=rng.randint(2, 16), plan=rng.randint(4, 999),
                    nsub=rng.randint(1, 3), xmac="fp16")
    while True:
        c = dict(CORR)
        c["kind"] = "host" if rng.random() < 0.1 else "corr"
        c["nbits"] = rng.choice([2, 2, 2, 8])
        c["npol"] = rng.choice([1, 2, 2, 2])
        c["nfreq"] = rng.choice([1, 2, 4, 8, 16] if c["nbits"] == 2 else [1, 2])
        c["full_pol"] = c["npol"] == 2 and rng.random() < 0.8
        c["nstation"] = int(round(math.exp(rng.uniform(math.log(2), math.log(32)))))
        c["bw"] = rng.choice([4.0, 8.0, 16.0, 32.0, 64.0])
        c["nchan"] = rng.choice([32, 64, 128, 256, 512, 1024, 1024, 1024, 2048, 4096, 8192])
        c["lsb"] = rng.random() < 0.25
        c["order"] = rng.choice([0, 1, 1, 1, 1, 1, 1, 2])
        c["avg"] = rng.choice([1, 1, 1, 2, 8])
        c["xmac"] = rng.choice(["fp16", "fp16", "fp16", "fp32", "fp32", "bf16"])
        c["nsub"] = rng.randint(1, 8)
        c["payload"] = rng.choice([8000, 8000, 5000])
        extra = rng.choice(["", "", "", "", "", "pcal", "zoom", "raw", "cplx"])
        if extra == "pcal":
            c["pcal"] = 1.0
        elif extra == "zoom":
            c["zoom"], c["lsb"] = True, False
            c["avg"] = 1
            if c["nchan"] < 64:
                continue
        elif extra == "raw":
            c["raw"] = True
            c["nbits"], c["kind"] = 2, "corr"
            c["payload"] *= c["nfreq"] * c["npol"]
            if c["nfreq"] * c["npol"] not in (2, 4, 8, 16):
                continue
        elif extra == "cplx":
            c["cplx"] = True
            c["order"] = rng.choice([1, 2])
            if c["nfreq"] * c["npol"] * c["nbits"] < 4 or c["nchan"] > 4096:
                continue
        if c["nbits"] == 2 and not extra and rng.random() < 0.3:
            c["invalid"] = 0.01
        # samples of a pass over all stations and bands, then FFTs per subint to match
        total = math.exp(rng.uniform(math.log(2e6), math.log(3e8)))
        nband = c["nfreq"] * c["npol"]
        T = int(total / (c["nstation"] * nband * 2 * c["nchan"] * c["nsub"]))
        fsamp = c["payload"] * 8 / (c["nbits"] * nband * (2 if c["cplx"] else 1))
        rate = (1 if c["cplx"] else 2) * c["bw"] * 1e6
        if nband * c["nbits"] > 128 or T < 3 or fsamp != int(fsamp) or rate % fsamp or 2 * c["nchan"] / fsamp > 28:
            continue
        c["subint_ns"] = int(T * c["nchan"] * 1000 / c["bw"])
        if 100_000 <= c["subint_ns"] <= 100_000_000:
            return c


# ---------------------------------------------------------------- recordings

THRESH, HIMAG, BLOCK, MARGIN_US = 0.98, 3.3359, 1 << 14, 20.0


def _polys(seed, nstation):
    """Per station a delay polynomial (us, us/s, us/s^2)."""
    r = np.random.default_rng([seed, 11])
    return [(float(r.uniform(-5, 5)), float(r.uniform(-1, 1)), float(r.uniform(-1e-4, 1e-4))) for _ in range(nstation)]


class _Geometry:
    """Frames and windows of one job's recordings (every station alike)."""

    def __init__(self, c):
        self.nband = c["nfreq"] * c["npol"]
        self.parts = 2 if c["cplx"] else 1
        self.rate = int((1 if c["cplx"] else 2) * c["bw"] * 1e6)
        self.fsamp = c["payload"] * 8 // (c["nbits"] * self.nband * self.parts)
        self.fps = self.rate // self.fsamp
        self.N = c["nchan"] * (1 if c["cplx"] else 2)
        self.T = int(round(c["subint_ns"] * c["bw"] / (c["nchan"] * 1000)))
        self.windows = []        # per subint: sec, ns, first frame, frames
        for k in range(1, c["nsub"] + 1):
            sec, ns = divmod(k * c["subint_ns"], 1_000_000_000)
            t = sec + ns * 1e-9
            f0 = max(0, int(math.floor((t - MARGIN_US * 1e-6) * self.fps)))
            f1 = int(math.floor((t + c["subint_ns"] * 1e-9 + MARGIN_US * 1e-6) * self.fps)) + 1
            self.windows.append((sec, ns, f0, f1 - f0))
        self.frame0 = self.windows[0][2]
        self.nframe = self.windows[-1][2] + self.windows[-1][3] - self.frame0

    def data_time(self, frame):
        return frame // self.fps, int(round((frame % self.fps) * 1e9 / self.fps))


def _codes(c, seed):
    """Yields per station the quantised samples [band * part][sample] (uint8
    codes) of its run of frames and a flag per frame (True: valid)."""
    g = _Geometry(c)
    gen = torch.Generator(device="cuda").manual_seed(1_000_003 * seed + 17)
    n = g.nframe * g.fsamp
    nblk = -(-n // BLOCK)
    dt = torch.complex64 if c["cplx"] else torch.float32
    rho = 0.05
    fwd, back = (torch.fft.fft, torch.fft.ifft) if c["cplx"] else (torch.fft.rfft, torch.fft.irfft)
    sky = [fwd(torch.randn(nblk, BLOCK, device="cuda", generator=gen, dtype=dt)) for _ in range(g.nband)]
    fs = g.rate * 1e-6
    fb = torch.arange(sky[0].shape[1], device="cuda", dtype=torch.float64) * (fs / BLOCK)
    tmid = (torch.arange(nblk, device="cuda", dtype=torch.float64) + 0.5) * (BLOCK / g.rate) + g.frame0 / g.fps
    for c0, c1, c2 in _polys(seed, c["nstation"]):
        tau = c0 + c1 * tmid + c2 * tmid * tmid
        out = torch.empty(g.nband * g.parts, n, device="cuda", dtype=torch.uint8)
        for b in range(g.nband):
            lo = 8400.0 + c["bw"] * (b // c["npol"])
            turns = (fb - lo if c["lsb"] and not c["cplx"] else -(lo + fb))[None, :] * tau[:, None]
            ph = (turns - torch.round(turns)).float() * (2 * math.pi)
            x = back(sky[b] * torch.polar(torch.ones_like(ph), ph), n=BLOCK).reshape(-1)[:n] * math.sqrt(rho)
            x = x + torch.randn(n, device="cuda", generator=gen, dtype=dt) * math.sqrt(1 - rho)
            for p, v in enumerate((x.real, x.imag) if c["cplx"] else (x,)):
                if c["nbits"] == 2:
                    q = (v >= -THRESH).to(torch.uint8) + (v >= 0).to(torch.uint8) + (v >= THRESH).to(torch.uint8)
                else:
                    q = torch.clamp(torch.round(v * 10) + 128, 0, 255).to(torch.uint8)
                out[b * g.parts + p] = q
        valid = torch.rand(g.nframe, device="cuda", generator=gen) >= c["invalid"]
        yield out, valid


def _headers(frames, fps, frame_bytes, log2ch, bits_word):
    h = torch.zeros(frames.numel(), 8, device="cuda", dtype=torch.int64)
    h[:, 0] = frames // fps
    h[:, 1] = frames % fps
    h[:, 2] = (1 << 29) | (log2ch << 24) | (frame_bytes // 8)
    h[:, 3] = bits_word
    return h


def _bytes(words):
    """int64 words [...] below 2^32 as little-endian bytes [..., 4]."""
    return torch.stack([(words >> s) & 255 for s in (0, 8, 16, 24)], dim=-1).to(torch.uint8)


def _pack(q, nbits):
    """codes [..., fields] -> payload bytes, fields from the lowest bit up."""
    if nbits == 8:
        return q
    q = q.reshape(*q.shape[:-1], -1, 4)
    return q[..., 0] | (q[..., 1] << 2) | (q[..., 2] << 4) | (q[..., 3] << 6)


def _recording(c, seed):
    """Per station the frames [frame, bytes] of its run (raw reads: the
    threads' frames, each frame time's in random order)."""
    g = _Geometry(c)
    frames = g.frame0 + torch.arange(g.nframe, device="cuda")
    out = []
    order = torch.Generator(device="cuda").manual_seed(seed + 5)
    for s, (q, valid) in enumerate(_codes(c, seed)):
        bits = ((c["nbits"] - 1) << 26) | s | ((1 << 31) if c["cplx"] else 0)
        if c["raw"]:
            tb = c["payload"] // g.nband
            body = _pack(q.reshape(g.nband, g.nframe, g.fsamp), c["nbits"]).permute(1, 0, 2)     # frame, thread, bytes
            head = _headers(frames, g.fps, tb + 32, 0, bits)[:, None, :].repeat(1, g.nband, 1)
            head[:, :, 3] |= torch.arange(g.nband, device="cuda")[None, :] << 16
            f = torch.cat([_bytes(head).reshape(g.nframe, g.nband, 32), body], dim=2)
            perm = torch.argsort(torch.rand(g.nframe, g.nband, device="cuda", generator=order), dim=1)
            f = torch.gather(f, 1, perm[:, :, None].expand(-1, -1, f.shape[2])).reshape(g.nframe, -1)
        else:
            body = _pack(q.reshape(-1, g.nframe, g.fsamp).permute(1, 2, 0).reshape(g.nframe, -1), c["nbits"])
            log2ch = int(math.log2(g.nband))
            head = _headers(frames, g.fps, c["payload"] + 32, log2ch, bits)
            head[:, 0] |= (~valid).to(torch.int64) << 31
            f = torch.cat([_bytes(head).reshape(g.nframe, 32), body], dim=1)
        out.append(f.contiguous())
        del q, body, head
    return out


# ---------------------------------------------------------------- prepare / run

ZOOMS = ((0, 0.25, 0.25), (1, 0.5, 0.5))      # parent subband, offset and width as fractions of its bandwidth


def _zooms(c):
    return [(p, o, w) for p, o, w in ZOOMS if p < c["nfreq"]] if c["zoom"] else []


def _job(c, seed):
    freqs = [Freq(8400.0 + c["bw"] * k, c["bw"], c["nchan"], "L" if c["lsb"] else "U", c["avg"])
             for k in range(c["nfreq"])]
    job = full_job(c["nstation"], freqs, pols="RL"[:c["npol"]], full_pol=c["full_pol"], subint_ns=c["subint_ns"],
                   nbits=c["nbits"], fringe_rot_order=c["order"])
    for st, p in zip(job.stations, _polys(seed, c["nstation"])):
        st.payload_bytes = c["payload"]
        st.pcal_interval_mhz = c["pcal"]
        st.complex_sampling = c["cplx"]
        if c["raw"]:
            st.mux_threads, st.mux_raw = st.nband, True
        st.polys = [DelayPoly(0.0, 120, p)]
    if c["zoom"]:
        add_zoom_bands(job, [(p, o * c["bw"], w * c["bw"]) for p, o, w in _zooms(c)])
    return job


def _members(c):
    """A batch's members as "corr" cases."""
    out = []
    for job in configs.c3(seed=c["plan"], nstation=c["nstation"], nsub=c["nsubband"]):
        f = job.freqs[0]
        out.append(dict(CORR, nstation=c["nstation"], nfreq=len(job.freqs), bw=f.bw_mhz, nchan=f.nchan,
                        nbits=job.stations[0].nbits, subint_ns=job.subint_ns, nsub=c["nsub"], xmac=c["xmac"]))
    return out


def _regions(corr):
    """The core result's parts: cross-correlations, baseline weights,
    autocorrelations, autocorrelation weights, phase-cal tones."""
    job, n = corr.job, 2 * corr.corelen
    lay = corr.layout()
    nfb, ns = len(job.freqs) * len(job.baselines), len(job.stations)
    bw = 2 * int(lay[nfb:2 * nfb][lay[nfb:2 * nfb] >= 0].min())
    ac, acw, pc = (lay[2 * nfb + i * ns:2 * nfb + (i + 1) * ns] for i in range(3))
    a, aw = 2 * int(ac.min()), 2 * int(acw.min())
    end = 2 * int(pc.min()) if pc.min() >= 0 else n
    return {"cross": slice(0, bw), "cross_weights": slice(bw, a), "auto": slice(a, aw), "auto_weights": slice(aw, end),
            "tones": slice(end, n)}


def _windows(c, frames):
    """Per subint: buffers, sizes and start times of every station's window, and the subint's time."""
    g = _Geometry(c)
    subs = []
    for sec, ns, f0, nf in g.windows:
        at = [f[f0 - g.frame0:f0 - g.frame0 + nf] for f in frames]
        dsec, dns = g.data_time(f0)
        n = len(at)
        subs.append(([a.data_ptr() for a in at], [a.numel() for a in at], [dsec] * n, [dns] * n, sec, ns))
    return subs


def prepare(case, seed):
    s = {"case": case}
    if case["kind"] == "mux":
        n, nt, fb = case["nframe"], case["nthread"], case["payload"] + 32
        gen = torch.Generator(device="cuda").manual_seed(seed + 3)
        s["fps"] = 4000
        head = _headers(torch.arange(n, device="cuda") + 7, s["fps"], fb, 0, (case["nbits"] - 1) << 26)
        head = head[:, None, :].repeat(1, nt, 1)
        head[:, :, 3] |= torch.arange(nt, device="cuda")[None, :] << 16
        body = torch.randint(0, 256, (n, nt, case["payload"]), device="cuda", generator=gen, dtype=torch.uint8)
        f = torch.cat([_bytes(head).reshape(n, nt, 32), body], dim=2)
        perm = torch.argsort(torch.rand(n, nt, device="cuda", generator=gen), dim=1)
        s["in"] = torch.gather(f, 1, perm[:, :, None].expand(-1, -1, fb)).reshape(-1)
        s["out"] = torch.empty(n * (case["payload"] * nt + 32), device="cuda", dtype=torch.uint8)
    else:
        batch = case["kind"] == "batch"
        cases = _members(case) if batch else [case]
        s["corr"], s["frames"], s["subs"], s["result"], s["regions"] = [], [], [], [], []
        for m, c in enumerate(cases):
            corr = Correlator(_job(c, seed + 1000 * m), xmac=c["xmac"], inflight=3)
            frames = _recording(c, seed + 1000 * m)
            n = 2 * corr.corelen
            if case["kind"] == "host":
                pinned = pinned_empty(sum(f.numel() for f in frames))
                held, at = [], 0
                for f in frames:
                    t = torch.from_numpy(pinned[at:at + f.numel()]).view(f.shape)
                    t.copy_(f)
                    held.append(t)
                    at += f.numel()
                frames = held
                s["pinned"] = pinned
                s["result"].append(np.zeros(n, dtype=np.float32))
            else:
                s["result"].append(torch.zeros(n, device="cuda", dtype=torch.float32))
            s["corr"].append(corr)
            s["frames"].append(frames)
            s["subs"].append(_windows(c, frames))
            s["regions"].append(_regions(corr))
        if batch:
            s["batch"] = Batch(s["corr"])
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return s


def _parts(result, regions):
    return {k: result[sl] for k, sl in regions.items() if sl.stop > sl.start}


def run(state):
    kind = state["case"]["kind"]
    if kind == "mux":
        case = state["case"]
        n = vdif_mux_device(state["in"].data_ptr(), state["in"].numel(), range(case["nthread"]), case["payload"] + 32,
                            state["fps"], case["nbits"], state["out"].data_ptr(), state["out"].numel())
        return state["out"][:n]
    if kind == "batch":
        for corr in state["corr"]:
            corr.reset()
        for k in range(state["case"]["nsub"]):
            sec, ns = state["subs"][0][k][4:]
            state["batch"].submit_device([subs[k][:4] for subs in state["subs"]], sec, ns)
        out = []
        for corr, result, regions in zip(state["corr"], state["result"], state["regions"]):
            corr.results_device(result.data_ptr(), result.numel())
            out.append(_parts(result, regions))
        return out
    corr, result = state["corr"][0], state["result"][0]
    corr.reset()
    submit = corr.submit_ptrs if kind == "host" else corr.submit_device
    for sub in state["subs"][0]:
        submit(*sub)
    if kind == "host":
        corr.results_into(result)
    else:
        corr.results_device(result.data_ptr(), result.numel())
    return _parts(result, state["regions"][0])


# ---------------------------------------------------------------- what a pass cannot do without

def _outputs(c):
    """(frequencies as (parent subband, first channel, channels), baseline products, autocorrelation passes)."""
    freqs = [(f, 0, c["nchan"]) for f in range(c["nfreq"])]
    freqs += [(p, int(o * c["nchan"] + 0.5), int(round(w * c["nchan"]))) for p, o, w in _zooms(c)]
    if c["npol"] == 1:
        prods = [(0, 0)]
    else:
        prods = [(0, 0), (0, 1), (1, 0), (1, 1)] if c["full_pol"] else [(0, 0), (1, 1)]
    return freqs, prods, 2 if len(prods) > 2 else 1


def _work(c):
    if c["kind"] == "mux":
        fb = c["payload"] + 32
        return c["nframe"] * c["nthread"] * fb + c["nframe"] * (c["payload"] * c["nthread"] + 32), 0
    if c["kind"] == "batch":
        w = [_work(m) for m in _members(c)]
        return sum(x for x, _ in w), sum(x for _, x in w)
    g = _Geometry(c)
    freqs, prods, passes = _outputs(c)
    S, nbl = c["nstation"], c["nstation"] * (c["nstation"] - 1) // 2
    frame = (c["payload"] + 32 * g.nband) if c["raw"] else c["payload"] + 32
    chans = sum(n for _, _, n in freqs)
    nout = (nbl * len(prods) + S * c["npol"] * passes) * chans
    nbytes = S * g.nframe * frame + 8 * nout // c["avg"]
    ffts = S * g.nband * g.T * c["nsub"]
    # decode and fringe rotation 2 per sample, one-sided FFT 2.5 N log2 N, fractional-sample rotation 6 per channel
    flops = ffts * (2 * g.N + 2.5 * g.N * math.log2(g.N) + 6 * c["nchan"]) + 8 * nout * g.T * c["nsub"]
    return nbytes, flops


def work(case):
    b, f = _work(case)
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------- the same in 64 bits

def _stride(n):
    if n <= 16:
        return n
    d = int(math.sqrt(n + 0.1))
    while n % d:
        d -= 1
    return n // d


def _interpolator(poly, t, span, T):
    d = [poly[0] + poly[1] * x + poly[2] * x * x for x in (t, t + span / 2, t + span)]
    return ((2 * d[0] - 4 * d[1] + 2 * d[2]) / (T * T), (-3 * d[0] + 4 * d[1] - d[2]) / T, d[0])


def _levels(codes, c):
    if c["nbits"] == 2:
        lut = torch.tensor([-HIMAG, -1.0, 1.0, HIMAG], device="cuda", dtype=torch.float32).double()
    else:
        lut = ((torch.arange(256, device="cuda", dtype=torch.float64) - 128) / 3.3).float().double()
    return lut[codes.long()]


def _station_spectra(c, g, poly, codes, valid, window):
    """Spectra [band, T, channel] of one station and subint, and its data weight per FFT."""
    sec, ns, f0, nf = window
    T, N, nchan = g.T, g.N, c["nchan"]
    dsec, dns = g.data_time(f0)
    sampletime = 1.0 / c["bw"] if c["cplx"] else 1.0 / (2 * c["bw"])
    span = T * 2 * nchan * (1.0 / (2 * c["bw"])) / 1e6
    c0, c1, c2 = _interpolator(poly, sec + ns / 1e9, span, T)
    i = np.arange(T, dtype=np.float64)
    mean = c0 * (i + 0.5) * (i + 0.5) + c1 * (i + 0.5) + c2
    start = (sec - dsec) * 1e6 + (ns - dns) / 1000.0 + i * N * sampletime - mean
    near = np.trunc(start / sampletime + 0.5)
    fse = torch.from_numpy(start - near * sampletime).cuda()
    n = torch.arange(N, device="cuda")
    at = torch.from_numpy(near.astype(np.int64)).cuda()[:, None] + n[None, :] + (f0 - g.frame0) * g.fsamp
    good = valid[at // g.fsamp]
    weight = good.double().mean(dim=1)
    asl = _stride(nchan)
    xj, kk = (n % asl).double() / N, (n // asl).double()
    Xk, X1 = kk * (asl / N), asl / N
    if c["order"] == 1:
        d0, d1, d2 = (c0 * x * x + c1 * x + c2 for x in (i, i + 0.5, i + 1))
        a = d2 - d0
        b = d0 + (d1 - (a * 0.5 + d0)) / 3.0
        whole = np.trunc(b)
        col = [torch.from_numpy(v).cuda()[:, None] for v in (a, b - whole)]
        delay = xj * col[0] + col[1] + Xk * col[0]
    elif c["order"] == 2:
        b, cc = c1 + i * c0 * 2, c2 + i * c1 + i * i * c0
        whole = np.trunc(cc)
        col = [torch.from_numpy(v).cuda()[:, None] for v in (b, cc - whole)]
        delay = xj * (col[0] + c0 * X1) + col[1] + kk * (xj * (2 * c0 * X1)) + Xk * col[0] + Xk * Xk * c0
    else:
        whole = np.trunc(mean)
        delay = torch.from_numpy(mean - whole).cuda()[:, None]
    whole = torch.from_numpy(whole).cuda()[:, None]
    chan = torch.arange(nchan, device="cuda", dtype=torch.float64) - (nchan if c["lsb"] else 0)
    frac = chan[None, :] * (c["bw"] / nchan) * fse[:, None]
    keep = (weight > 0)[:, None]
    out = []
    for band in range(g.nband):
        lo = 8400.0 + c["bw"] * (band // c["npol"])
        if c["cplx"]:
            x = torch.complex(_levels(codes[2 * band], c)[at], _levels(codes[2 * band + 1], c)[at])
            lo = -lo if c["lsb"] else lo
        else:
            x = _levels(codes[band], c)[at]
        x = x * good
        ph = delay * lo + (lo - int(lo)) * whole
        rot = torch.polar(torch.ones_like(ph), -2 * math.pi * (ph - torch.floor(ph)))
        X = torch.fft.fft(x * rot if c["order"] else x.to(torch.complex128))
        if not c["lsb"]:
            X = X[:, :nchan]
        elif c["cplx"]:
            X = torch.cat([X[:, :1], X[:, 1:].flip(1).conj()], dim=1)
        elif c["order"]:
            X = X[:, nchan:]
        else:
            X = X[:, 1:nchan + 1].flip(1).conj()
        X = X * torch.polar(torch.ones_like(frac), 2 * math.pi * (frac - torch.round(frac)))
        if not c["order"]:
            X = X * rot
        out.append(X * keep)
    return torch.stack(out), weight


def _exact_corr(c, seed):
    g = _Geometry(c)
    freqs, prods, passes = _outputs(c)
    S, npol = c["nstation"], c["npol"]
    polys = _polys(seed, S)
    data = list(_codes(c, seed))
    acc = [0] * c["nfreq"]
    wsum, wbase = 0, 0
    for w in g.windows:
        spec, weights = [], []
        for s in range(S):
            X, wt = _station_spectra(c, g, polys[s], *data[s], w)
            spec.append(X)
            weights.append(wt)
        wt = torch.stack(weights)
        wsum = wsum + wt.sum(dim=1)
        wbase = wbase + wt @ wt.T
        for f in range(c["nfreq"]):
            X = torch.cat([x[f * npol:(f + 1) * npol] for x in spec]).permute(2, 0, 1)     # channel, input, T
            acc[f] = acc[f] + X @ X.mH
        del spec
    avg = c["avg"]

    def mean(v):
        return torch.view_as_real(v.reshape(-1, avg).mean(dim=1)).reshape(-1)

    cross, cross_w, auto, auto_w = [], [], [], []
    for f, first, n in freqs:
        V = acc[f][first:first + n]
        for s1 in range(S):
            for s2 in range(s1 + 1, S):
                for p1, p2 in prods:
                    cross.append(mean(V[:, s1 * npol + p1, s2 * npol + p2]))
                cross_w += [wbase[s1, s2]] * len(prods) + [wbase[0, 0] * 0] * (len(prods) % 2)
    for s in range(S):
        for hand in range(passes):
            for f, first, n in freqs:
                for p in range(npol):
                    auto.append(mean(acc[f][first:first + n, s * npol + p, s * npol + (p ^ hand)]))
        nw = passes * len(freqs) * npol
        auto_w += [wsum[s]] * nw + [wsum[s] * 0] * (nw % 2)
    out = {"cross": torch.cat(cross), "cross_weights": torch.stack(cross_w), "auto": torch.cat(auto),
           "auto_weights": torch.stack(auto_w)}
    if c["pcal"]:
        out["tones"] = None
    return out


def exact(case, seed):
    if case["kind"] == "mux":
        return None
    if case["kind"] == "batch":
        return [_exact_corr(c, seed + 1000 * m) for m, c in enumerate(_members(case))]
    return _exact_corr(case, seed)
