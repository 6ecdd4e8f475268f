// F stage (Mode::process, mpifxcorr/src/mode.cpp:845-1308) for sm_100a.
//
// One CTA per (station, subband, chunk of FFTs).  This file has the form of a
// subband with one band; two polarisations are transformed together by the
// form of fxb_fstage_pair.cuh, which runs the same steps.  The FFT length is a template
// parameter, so the pass schedule and every shared-memory index fold to
// constants.  Each thread owns KB radix-8 butterflies of every pass of one
// FFT ("slot"): an FFT of N points takes N / (8 KB) threads, and a CTA runs
// several slots side by side when N is small.  Per FFT a thread
//   1. decodes its 8 KB samples x[b + r N/8] straight from the VDIF words in
//      global memory (2-bit / 8-bit levels of format_vdif.c:74-149; samples of
//      invalid frames and, for 8-bit 2/4-channel streams, every sample after
//      the first blanked one, read as zero: format_vdif.c:1879-1922),
//   2. multiplies them by the fringe rotator exp(-2 pi i phi(n)) of the order
//      in use (mode.cpp:906-1051; phi reduced to [-1/2, 1/2) turns in FP64 at
//      the FFT start, per sample in FP32),
//   3. runs the first radix-8 pass of a Stockham autosort FFT in registers
//      and exchanges through padded shared memory for the remaining passes
//      (two buffers used alternately: one barrier per exchange),
//   4. in the last pass selects the sideband (USB bins 0..nchan-1, LSB
//      nchan..2nchan-1, order-0 LSB the conjugate mirror), applies the
//      fractional-sample rotator exp(+2 pi i f_c fse) (mode.cpp:1053-1097,
//      1279-1286) and the post-F fringe phase of order 0 (mode.cpp:1061-1070),
//      and stores its channels to the spectra [t][row][chan].
//
// The FFT is FP32.  Two output forms:
//   out 0: spectra as float2 [t][row][chan] (the plain FP32 form);
//   out 1: spectra of the tensor-core forms, half2 or bf16x2 (re, im) of
//          X 2^-kTcSpecExp in the blocked layout the tensor-core XMAC reads
//          (one rounding per value, for the kinds the tensor-core FFT of
//          fxb_fstage_tc.cu does not cover).
//
// Twiddles come from a per-length table laid out [pass][r - 1][p] (entry
// w_N^(r p s) for pass stride s), so that the twiddle loads of a warp are
// coalesced (first pass) or broadcasts (later passes).

#pragma once

#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cstdint>
#include <type_traits>

#include "fxb_internal.h"
#include "fxb_kernels.h"
#include "fxb_ptx.cuh"

namespace fxb {

namespace {

// padded index of 8-byte element i: every exchange of the pass schedule
// below is free of bank conflicts, and runs of 8 starting at multiples of 8
// stay contiguous and 16-byte aligned (the first pass stores them as pairs)
__host__ __device__ constexpr int xpad(int i) { return i + 2 * (i >> 4); }

// Compile-time shape of the F stage for FFT length 2^LOGN.
template <int LOGN>
struct FShape {
	static constexpr int N = 1 << LOGN;
	static constexpr int KB = N <= 2048 ? 1 : (N <= 8192 ? 2 : 4);
	static constexpr int TPF = N / (8 * KB);                 // threads per FFT
	static constexpr int NT = TPF >= 256 ? TPF : 256;        // threads per CTA
	static constexpr int FPC = NT / TPF;                     // FFTs side by side
	static constexpr int PADN = xpad(N);
	static constexpr int NMID = (LOGN % 3 == 0) ? LOGN / 3 - 2 : LOGN / 3 - 1;
	static constexpr int RL = (LOGN % 3 == 0) ? 8 : (1 << (LOGN % 3));
	// 8192 points: two butterflies per thread in 512-thread CTAs at 64 registers
	// (two CTAs per SM) run 37 % faster than four per thread at 128 registers
	static constexpr int MINB = KB == 1 ? 3 : (NT == 256 || KB == 2 ? 2 : 1);
};

// offset of the twiddles of radix-8 pass `pass` (stride 8^pass) in the table
__host__ __device__ constexpr int tw_offset(int N, int pass)
{
	int o = 0, n8 = N / 8;
	for(int i = 0; i < pass; i++)
	{
		o += 7 * n8;
		n8 /= 8;
	}
	return o;
}

// padded index of element i + S r (i >= 0): for S a multiple of 16 the
// padding of i + S r is that of i plus r S / 8, a constant offset per r.
// Used for FFTs of 8192 points and more (FAST); shorter lengths keep the
// plain form, whose register allocation measured better.
template <int S, bool FAST>
__device__ __forceinline__ int st_index(int i, int r)
{
	if constexpr(FAST && S % 16 == 0)
		return xpad(i) + r * xpad(S);
	else
		return xpad(i + S * r);
}

// ---- lane values: FP32 complex
struct cf { float x, y; };

__device__ __forceinline__ cf add(cf a, cf b) { return {a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ cf sub(cf a, cf b) { return {a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ cf add_mi(cf a, cf b) { return {a.x + b.y, a.y - b.x}; }   // a - i b
__device__ __forceinline__ cf add_pi(cf a, cf b) { return {a.x - b.y, a.y + b.x}; }   // a + i b
__device__ __forceinline__ cf rot45(cf a)                                               // a (1 - i) / sqrt2
{
	const float r = 0.70710678118654752440f;
	return {(a.x + a.y) * r, (a.y - a.x) * r};
}
__device__ __forceinline__ cf twid(cf a, float2 w) { return {a.x * w.x - a.y * w.y, a.x * w.y + a.y * w.x}; }

__device__ __forceinline__ float2 ldtw(const float2 *t, int i) { return __ldg(t + i); }
// 8-byte shared-memory element <-> lane value
__device__ __forceinline__ cf lds(const uint2 *p)
{
	const float2 v = *(const float2 *)p;
	return {v.x, v.y};
}
__device__ __forceinline__ uint2 bits(cf v) { return make_uint2(__float_as_uint(v.x), __float_as_uint(v.y)); }
__device__ __forceinline__ void sts(uint2 *p, cf v) { *p = bits(v); }
__device__ __forceinline__ void sts2(uint2 *p, cf a, cf b)
{
	const uint2 u = bits(a), w = bits(b);
	*(uint4 *)p = make_uint4(u.x, u.y, w.x, w.y);
}

// forward DFTs in place (w = exp(-2 pi i / R))
template <typename C>
__device__ __forceinline__ void dft8(C *x)
{
	const C a0 = add(x[0], x[4]), d0 = sub(x[0], x[4]);
	const C a1 = add(x[1], x[5]), d1 = sub(x[1], x[5]);
	const C a2 = add(x[2], x[6]), d2 = sub(x[2], x[6]);
	const C a3 = add(x[3], x[7]), d3 = sub(x[3], x[7]);
	const C b0 = add(a0, a2), b2 = sub(a0, a2), b1 = add(a1, a3), b3 = sub(a1, a3);
	x[0] = add(b0, b1);
	x[4] = sub(b0, b1);
	x[2] = add_mi(b2, b3);
	x[6] = add_pi(b2, b3);
	// odd bins: DFT4 of d_k w^k, with d1 w + d3 w^3 = (d1 - i d3) w and d1 w - d3 w^3 = (d1 + i d3) w
	const C f0 = add_mi(d0, d2), f2 = add_pi(d0, d2);
	const C f1 = rot45(add_mi(d1, d3)), f3 = rot45(add_pi(d1, d3));
	x[1] = add(f0, f1);
	x[5] = sub(f0, f1);
	x[3] = add_mi(f2, f3);
	x[7] = add_pi(f2, f3);
}

template <typename C>
__device__ __forceinline__ void dft4(C *x)
{
	const C b0 = add(x[0], x[2]), b2 = sub(x[0], x[2]), b1 = add(x[1], x[3]), b3 = sub(x[1], x[3]);
	x[0] = add(b0, b1);
	x[2] = sub(b0, b1);
	x[1] = add_mi(b2, b3);
	x[3] = add_pi(b2, b3);
}

template <typename C>
__device__ __forceinline__ void dft2(C *x)
{
	const C a = x[0], b = x[1];
	x[0] = add(a, b);
	x[1] = sub(a, b);
}

template <int R, typename C>
__device__ __forceinline__ void dftR(C *x)
{
	if constexpr(R == 8)
		dft8(x);
	else if constexpr(R == 4)
		dft4(x);
	else
		dft2(x);
}

// 2-bit code -> {-HiMag, -1, +1, +HiMag} (format_vdif.c:78): sign from bit 1,
// magnitude HiMag for codes 0 and 3
__host__ __device__ inline float level2(uint32_t code)
{
	const float mag = ((code ^ (code >> 1)) & 1u) ? 1.0f : 3.3359f;
	return (code & 2u) ? mag : -mag;
}

__device__ __forceinline__ float frac_centered(double x) { return (float)(x - rint(x)); }

// A row of the tensor-core spectra: its first value of time 0 and the step of a time
struct OutRow {
	int64_t first;
	int32_t tstride;
	uint32_t tcb, magic, bextra;
};
__device__ __forceinline__ OutRow out_row(const DevFreqPlan &P, int row)
{
	return {P.spec_off + (int64_t)max(row, 0) * P.tcb, P.tnblk * P.trow * P.tcb, (uint32_t)P.tcb, P.magic,
	        (uint32_t)(P.trow - 1) * (uint32_t)P.tcb};
}

// CTAs per SM the register budget is sized for
template <int LOGN>
constexpr int fstage_minb()
{
	return FShape<LOGN>::MINB;
}

constexpr int kMaxTQ = 4;         // FFT iterations per CTA at most

// Constants of one FFT, computed once per CTA (one warp per FFT).
struct FftConst {
	float P0, alpha, beta, gamma, eps;   // fringe phase (turns): start and per-sample terms
	float stc, sts;                      // order 1: rotator step over N/8 samples, exp(-2 pi i alpha N/8)
	float dhi, dlo;                      // fractional-sample turns per channel (split_turns)
	float postf;                         // order-0 post-F turns
	uint32_t fa, so;                     // first frame of the window, window start within it
	uint32_t fmask;                      // validity of the window's frames (bit k: frame fa + k)
	int32_t stuck;                       // samples [stuck, N) read as zero
	int32_t flags;                       // 1: valid FFT, 2: fmask covers the window,
	                                     // 4: a valid frame of the window blanks the item's band
};

// One middle radix-8 pass (stride s = 2^LOGS, m = N / (8 s)) over the
// thread's KB butterflies: x_r = X[q + s (p + r m)], y = DFT8(x),
// Y[q + s (8 p + r)] = y_r w_N^(r p s).  With two buffers each butterfly
// reads, transforms and writes on its own; with one buffer all reads of the
// pass come before any write.
template <int LOGN, int LOGS>
__device__ __forceinline__ void mid_pass(int &wb, uint2 *side0, uint2 *side1, int pp, int bt, const float2 *twp)
{
	using SH = FShape<LOGN>;
	constexpr int N = SH::N, KB = SH::KB, TPF = SH::TPF;
	constexpr int s = 1 << LOGS;
	constexpr int m = N >> (LOGS + 3);
	constexpr int np = N / (8 * s);
	const uint2 *src = wb ? side1 : side0;
	wb ^= 1;
	uint2 *dst = wb ? side1 : side0;
	cf x[KB][8];
#pragma unroll
	for(int k = 0; k < KB; k++)
	{
		const int b = bt + k * TPF;
		const int q = b & (s - 1), p8 = b >> LOGS;
#pragma unroll
		for(int r = 0; r < 8; r++)
		{
			// for N >= 128 the stride s m = N/8 is a multiple of 16, so the
			// padding of point r is a constant offset from that of point 0
			if constexpr(N >= 128)
				x[k][r] = lds(src + xpad(q + s * p8) + r * xpad(s * m));
			else
				x[k][r] = lds(src + xpad(q + s * (p8 + r * m)));
		}
		dft8(x[k]);
#pragma unroll
		for(int r = 1; r < 8; r++)
			x[k][r] = twid(x[k][r], ldtw(twp, (r - 1) * np + p8));
		if(pp)
		{
#pragma unroll
			for(int r = 0; r < 8; r++)
				sts(dst + st_index<s, (N >= 8192)>(q + s * 8 * p8, r), x[k][r]);
		}
	}
	if(!pp)
	{
		__syncthreads();
#pragma unroll
		for(int k = 0; k < KB; k++)
		{
			const int b = bt + k * TPF;
			const int q = b & (s - 1), p8 = b >> LOGS;
#pragma unroll
			for(int r = 0; r < 8; r++)
				sts(dst + st_index<s, (N >= 8192)>(q + s * 8 * p8, r), x[k][r]);
		}
	}
	__syncthreads();
}

template <int LOGN, int PS>
__device__ __forceinline__ void mid_passes(int &wb, uint2 *side0, uint2 *side1, int pp, int bt, const float2 *tw)
{
	if constexpr(PS < FShape<LOGN>::NMID)
	{
		mid_pass<LOGN, 3 * (PS + 1)>(wb, side0, side1, pp, bt, tw + tw_offset(1 << LOGN, PS + 1));
		mid_passes<LOGN, PS + 1>(wb, side0, side1, pp, bt, tw);
	}
}

}  // namespace

// Level tables of the decode: 8-bit levels (b - 128) / 3.3 computed in double
// and rounded to float (format_vdif.c:122).
__device__ __forceinline__ void fstage_luts(float *lut8)
{
	for(int i = threadIdx.x; i < 256; i += blockDim.x)
		lut8[i] = (float)((i - 128) / 3.3);
}

// One work unit of the F stage: FFT times [tchunk tq FPC, +tq FPC) of work
// item gidx (an FGroup of one band), run by the CTA's FShape<LOGN>::NT threads
// with the level table already in shared memory, fsm the unit's exchange buffers
// (two when pp) and fcs room for tq FPC FFT constants.
// TCO: tensor-core spectra out;
// VAR 1: raw INTERLACEDVDIF reads (each band read from its thread's frame);
// VAR 2: complex sampling (nchan-point complex FFT: every bin a channel of
// the upper sideband, or bin 0 and the conjugated mirror of the rest for the
// lower sideband, mode.cpp:1182-1234).
template <int LOGN, bool TCO, int VAR>
__device__ __forceinline__ void fstage_unit(const FsArgs &a, const int gidx, const int tchunk, const int tq, const int pp,
                                            const float2 *tw, uint2 *fsm, const float *lut8, FftConst *fcs)
{
	using SH = FShape<LOGN>;
	constexpr int N = SH::N, KB = SH::KB, TPF = SH::TPF, FPC = SH::FPC, PADN = SH::PADN, RL = SH::RL;
	const FGroup g = a.groups[gidx];
	const DevStation *Sp = a.st + g.station;
	constexpr bool MUX = VAR == 1, CPLX = VAR == 2;
	constexpr int nchan = CPLX ? N : N / 2;
	const uint32_t fs = (uint32_t)Sp->framesamples;
	const int nbits = Sp->nbits;
	// raw INTERLACEDVDIF reads: band b's samples are those of its thread's
	// frame, found through the frame-slot table (one band per frame)
	constexpr bool muxraw = MUX;
	const int32_t *mslot = muxraw ? a.sub[g.station].mux_slot : nullptr;
	const int64_t mk0 = muxraw ? a.sub[g.station].mux_k0 : 0;
	const int mnthr = Sp->nthr, minfb = Sp->inframebytes;
	// complex samples: real then imaginary field of nbits per band and time
	constexpr uint32_t cpl = CPLX ? 2u : 1u;
	const uint32_t bpt = muxraw ? (uint32_t)nbits : (uint32_t)(Sp->nband * nbits) * cpl;
	const int header = Sp->header, framebytes = Sp->framebytes, asl = Sp->asl;
	const double bw = Sp->bw;
	const uint8_t *buf = a.sub[g.station].buf;
	const int slot = (int)threadIdx.x / TPF, bt = (int)threadIdx.x - slot * TPF;
	uint2 *const side0 = fsm + (size_t)slot * PADN;
	uint2 *const side1 = pp ? side0 + (size_t)FPC * PADN : side0;
	const uint8_t *vrow = a.valid + (int64_t)g.station * a.valid_stride;
	const bool lsb = g.lsb != 0;
	const double lo = g.lofreq;
	const float ph0 = g.phase[0];                      // phase-offset rotation (turns)
	const int row0 = g.row[0];
	const uint32_t boff0 = muxraw ? 0u : (uint32_t)(g.band[0] * nbits) * cpl;
	const int order = a.order;
	constexpr float osc = 1.0f / (float)(1 << kTcSpecExp);
	const bool h16 = a.h16 != 0;

	// (tensor-core form up to 8192 points, where registers are short: read at each
	// FFT's output)
	OutRow out = {};
	if constexpr(TCO && N > 8192)
		out = out_row(a.plans[g.freq], row0);
	const int64_t spec_off = TCO ? 0 : a.plans[g.freq].spec_off;
	const int prow = TCO ? 0 : a.plans[g.freq].nrow;

	const int t0 = tchunk * tq * FPC;
	const int nit = min(tq, (a.T - t0 + FPC - 1) / FPC);
	// ---- constants of the unit's FFTs (FFT f is time t0 + f), one thread per FFT
	{
		const int nfc = nit * FPC;
		for(int f = (int)threadIdx.x; f < nfc; f += (int)blockDim.x)
		{
			const int t = t0 + f;
			FftConst c;
			c.P0 = c.alpha = c.beta = c.gamma = c.eps = c.postf = 0.0f;
			c.dhi = c.dlo = 0.0f;
			c.stc = 1.0f;
			c.sts = 0.0f;
			c.fa = c.so = c.fmask = 0u;
			c.stuck = 0;
			c.flags = 0;
			if(t < a.T)
			{
				const FftParam *pq = a.params + (int64_t)g.station * a.T + t;
				if(pq->status == kFftOk)
				{
					c.flags = 1;
					const uint32_t g0 = (uint32_t)pq->nearest;
					c.fa = g0 / fs;
					c.so = g0 - c.fa * fs;
					c.stuck = pq->stuck;
					const double invN = 1.0 / N;
					const int idl = pq->integerdelay;
					const double fraclo = a.fraclo ? (lo - (int)lo) * (double)idl : 0.0;
					// LO offset: seconds since the job start of the FFT's first
					// sample (mode.cpp:686-694; the scan starts with the job) and
					// the offset's turns per sample
					const double walls = (double)a.sub[g.station].subsec + a.sub[g.station].subns / 1.0e9 +
					                     (double)t * N * Sp->sampletime / 1.0e6;
					const double low = g.corr ? looff_wall_turns(g.looff, walls) : 0.0;
					const double los = -g.looff * Sp->sampletime / 1.0e6;
					if(order == 1)
					{
						c.P0 = frac_centered(lo * pq->b + fraclo + low);
						c.alpha = (float)(lo * pq->a * invN + los);
						// each thread's samples are N/8 apart: one step phasor per FFT
						const double st = (double)c.alpha * (double)(N / 8);
						double ss, sc;
						sincospi(-2.0 * (st - rint(st)), &ss, &sc);
						c.stc = (float)sc;
						c.sts = (float)ss;
					}
					else if(order == 2)
					{
						const double pa = pq->a, pb = pq->b;
						const double X1 = (double)asl * invN;
						c.P0 = frac_centered(lo * pq->c + fraclo + low);
						c.alpha = (float)(lo * (pb + pa * X1) * invN + los);
						c.beta = (float)(lo * 2.0 * pa * X1 * invN);
						c.gamma = (float)(lo * pb * asl * invN + los * asl);
						c.eps = (float)(lo * pa * X1 * X1);
					}
					// fse - clock offset (mode.cpp:1053-1059, 1099-1106)
					split_turns(bw * (1.0 / nchan) * ((double)pq->fse - g.clk[0]), c.dhi, c.dlo);
					if(order == 0)
					{
						double pr = (pq->averagedelay - idl) * lo;
						if(a.fraclo)
							pr += idl * (lo - (int)lo);
						pr -= walls * g.looff;
						c.postf = -(float)(pr - (int)pr);
					}
				}
			}
			// validity of the window's frames, one bit per frame relative to fa
			const uint32_t nwf = (c.so + (uint32_t)N - 1) / fs + 1;
			if(c.flags & 1)
			{
				const uint32_t nm = nwf < 32u ? nwf : 32u;
				for(uint32_t k = 0; k < nm; k++)
				{
					const int64_t fr = (int64_t)c.fa + k;
					// complex data: the unpack's first frame is checked for fill
					// pattern only (mark5_stream_unpacker.c:189)
					const uint8_t *vsrc =
					    (CPLX && k == 0 && a.fillok) ? a.fillok + (int64_t)g.station * a.valid_stride : vrow;
					if(fr < a.valid_stride && vsrc[fr] != 0)
						c.fmask |= 1u << k;
				}
			}
			if(nwf <= 32)
				c.flags |= 2;
			if(a.bandok)
			{
				// EDV4-blanked bands (INTERLACEDVDIF): the slow decode path below
				const uint32_t need = 1u << g.band[0];
				bool part = false;
				for(uint32_t k = 0; (c.flags & 1) && k < nwf && !part; k++)
				{
					const int64_t fk = (int64_t)c.fa + k;
					part = fk < a.valid_stride && vrow[fk] != 0 &&
					       (a.bandok[(int64_t)g.station * a.valid_stride + fk] & need) != need;
				}
				if(part)
					c.flags |= 4;
			}
			fcs[f] = c;
		}
		__syncthreads();
	}
	int wb = 0;
	for(int it = 0; it < nit; it++)
	{
		const int t = t0 + it * FPC + slot;
		const bool tok = t < a.T;
		// ---- per-FFT constants
		const FftConst &fc = fcs[it * FPC + slot];
		const bool active = (fc.flags & 1) != 0;
		const uint32_t fa = fc.fa, so = fc.so, fmask = fc.fmask;
		const int stuck = fc.stuck;
		const float P0 = fc.P0, alpha = fc.alpha, beta = fc.beta, gamma = fc.gamma, eps = fc.eps;
		const float stc = fc.stc, sts = fc.sts;
		const float dhi = fc.dhi, dlo = fc.dlo, postf = fc.postf;
		const bool narrow = (fc.flags & 2) != 0;
		const bool blank = (fc.flags & 4) != 0;
		// ---- 1-3. decode, fringe-rotate and run the first radix-8 pass (s = 1:
		// butterfly b, twiddle w_N^(r b)), one butterfly at a time
		{
			uint2 *dst = wb ? side1 : side0;
			if(!pp)
				__syncthreads();                    // the single buffer has been read by the last FFT
#pragma unroll
			for(int k = 0; k < KB; k++)
			{
				const int b = bt + k * TPF;
				const uint32_t xs = so + (uint32_t)b;
				uint32_t kf = xs / fs, tin = xs - kf * fs;
				const uint8_t *fp = buf + ((int64_t)fa + kf) * framebytes + header;
				// phase A: frame tracking and every word load of the 8 samples
				// (nothing waits on a load before all are issued)
				uint32_t raw0[8], pk[8];
#pragma unroll
				for(int r = 0; r < 8; r++)
				{
					const int n = b + r * (N / 8);
					bool ok;
					if(narrow)
						ok = (fmask >> kf) & 1u;
					else
					{
						const int64_t fr = (int64_t)fa + kf;
						ok = active && fr < a.valid_stride && vrow[fr] != 0;
					}
					ok = ok && n < stuck;
					const uint32_t bit0 = tin * bpt + boff0;
					if(muxraw)
					{
						// valid frames of raw reads are complete slots: every thread is there
						const int32_t *slr = mslot + (mk0 + (int64_t)fa + kf) * mnthr;
						const int i0 = ok ? __ldg(slr + g.band[0]) : -1;
						raw0[r] = i0 >= 0 ? __ldg((const uint32_t *)(buf + (int64_t)i0 * minfb + 32) + (bit0 >> 5)) : 0u;
					}
					else
					{
						const uint32_t *wp = (const uint32_t *)fp;
						raw0[r] = ok ? __ldg(wp + (bit0 >> 5)) : 0u;
					}
					pk[r] = (bit0 & 31u) | ((uint32_t)ok << 16);
					if(r < 7)
					{
						tin += (uint32_t)(N / 8);
						while(tin >= fs)
						{
							tin -= fs;
							kf++;
							fp += framebytes;
						}
					}
				}
				// phase B: levels, fringe rotation (order 1: the rotator of sample b,
				// then one complex step per N/8 samples)
				float rc = 1.0f, rs = 0.0f;
				if(order == 1)
				{
					float ph0 = P0 + (float)b * alpha;
					ph0 -= rintf(ph0);
					__sincosf(-6.283185307179586f * ph0, &rs, &rc);
				}
				cf x[8];
#pragma unroll
				for(int r = 0; r < 8; r++)
				{
					const int n = b + r * (N / 8);
					float v0 = 0.0f, u0 = 0.0f;       // u: imaginary part (complex sampling)
					if((pk[r] >> 16) & 1u)
					{
						const uint32_t w0 = raw0[r] >> (pk[r] & 31u);
						v0 = nbits == 2 ? level2(w0 & 3u) : lut8[w0 & 255u];
						if constexpr(CPLX)
							u0 = nbits == 2 ? level2((w0 >> 2) & 3u) : lut8[(w0 >> 8) & 255u];
						if(blank)
						{
							// band of this sample's frame blanked by its EDV4 validity mask
							// (blank_vdif_EDV4, format_vdif.c:4699-4780)
							const uint32_t bo = a.bandok[(int64_t)g.station * a.valid_stride + fa + (so + (uint32_t)n) / fs];
							if(!((bo >> g.band[0]) & 1u))
								v0 = u0 = 0.0f;
						}
					}
					float sn = 0.0f, cs = 1.0f;
					if(order == 1)
					{
						cs = rc;
						sn = rs;
						const float nc = rc * stc - rs * sts;
						rs = rc * sts + rs * stc;
						rc = nc;
					}
					else if(order == 2)
					{
						const int kk = n / asl, jj = n - kk * asl;
						float ph = P0 + (float)jj * alpha + (float)(kk * jj) * beta + (float)kk * gamma +
						           (float)(kk * kk) * eps;
						ph -= rintf(ph);
						__sincosf(-6.283185307179586f * ph, &sn, &cs);
					}
					if constexpr(CPLX)
						x[r] = cf{v0 * cs - u0 * sn, v0 * sn + u0 * cs};
					else
						x[r] = cf{v0 * cs, v0 * sn};
				}
				dft8(x);
#pragma unroll
				for(int r = 1; r < 8; r++)
					x[r] = twid(x[r], ldtw(tw, (r - 1) * (N / 8) + b));
				uint2 *q = dst + xpad(8 * b);
				sts2(q, x[0], x[1]);
				sts2(q + 2, x[2], x[3]);
				sts2(q + 4, x[4], x[5]);
				sts2(q + 6, x[6], x[7]);
			}
			__syncthreads();
		}
		// ---- middle radix-8 passes through shared memory
		mid_passes<LOGN, 0>(wb, side0, side1, pp, bt, tw);
		// ---- 4. last pass, sideband selection, fractional-sample rotation, output
		{
			constexpr int sL = N / RL;
			constexpr int J = (KB * 8) / RL;
			const uint2 *src = wb ? side1 : side0;
			wb ^= 1;
			// one value: fractional-sample (and order-0 fringe) rotation of effective
			// channel ce, y conjugated when cj < 0
			auto turned = [&](cf y, int ce, float cj) {
				const float fce = (float)ce;
				float th = fce * dhi;               // exact (split_turns)
				th -= rintf(th);
				float turns = th + fmaf(fce, dlo, postf + ph0);
				turns -= rintf(turns);
				float sn, cs;
				__sincosf(6.283185307179586f * turns, &sn, &cs);
				const float xr = y.x, xi = cj * y.y;
				if constexpr(TCO)
				{
					cs *= osc;
					sn *= osc;
				}
				return cf{xr * cs - xi * sn, xr * sn + xi * cs};
			};
			// the sideband: order-0 lower bands (and complex ones) mirror their bins
			const bool mirror = lsb && order == 0;
			if constexpr(TCO)
			{
				// A thread's outputs are N/8 apart, bins q0 + m N/8: the channels of a quad
				// of positions (chan_pos), stored at once.  One by one, a warp's 4-byte
				// stores met 32 sectors each: 14 stations x 1 band, 8 bits, F stage of 8192
				// channels 860 us and 600 now, of 4096 275 and 230, of 2048 (with a launch
				// of its own) 150 and 124, of 1024 82 and 82, of 256 54 and 49
				constexpr int JG = 8 / RL;
				const OutRow O = N > 8192 ? out : out_row(a.plans[g.freq], row0);
				uint32_t *const orow = (uint32_t *)a.spec + O.first + (int64_t)t * O.tstride;
				auto packed = [&](cf y, int ce, float cj) {
					const cf v = turned(y, ce, cj);
					return pack_spec(h16, v.x, v.y);
				};
				auto quad = [&](uint32_t p0, uint32_t h0, uint32_t h1, uint32_t h2, uint32_t h3) {
					store_quad(orow, p0, O.tcb, O.magic, O.bextra, make_uint4(h0, h1, h2, h3));
				};
#pragma unroll 1
				for(int kb = 0; kb < KB; kb++)
				{
					const int q0 = bt + kb * TPF;
					constexpr int NH = CPLX ? 8 : 4;
					uint32_t h[NH], edge = 0u;
#pragma unroll
					for(int g8 = 0; g8 < JG; g8++)
					{
						const int q = q0 + g8 * (N / 8);
						cf y[RL];
#pragma unroll
						for(int r = 0; r < RL; r++)
							y[r] = lds(src + st_index<sL, (N >= 8192)>(q, r));
						dftR<RL>(y);
						if(!tok || row0 < 0)
							continue;
#pragma unroll
						for(int r = 0; r < (CPLX ? RL : RL / 2); r++)
						{
							const int k = q + sL * r;
							uint32_t &o = h[g8 + r * JG];
							if constexpr(CPLX)
								o = packed(y[r], lsb ? (k == 0 ? -N : -k) : k, lsb && k != 0 ? -1.0f : 1.0f);
							else
							{
								const bool upper = lsb && !mirror;             // bins N/2 ..
								o = packed(cf{upper ? y[r + RL / 2].x : y[r].x, upper ? y[r + RL / 2].y : y[r].y},
								           mirror ? -k : (lsb ? k - nchan : k), mirror ? -1.0f : 1.0f);
							}
						}
						if constexpr(!CPLX)
							if(mirror && g8 == 0 && q0 == 0)
								edge = packed(y[RL / 2], -nchan, -1.0f);        // bin N/2, channel 0
					}
					if(!tok || row0 < 0)
						continue;
					const uint32_t p = 4u * (uint32_t)q0, pm = (uint32_t)(N / 2) - p, p8 = (uint32_t)(N / 2);
					if constexpr(CPLX)
					{
						if(!lsb)
						{
							quad(p, h[0], h[2], h[4], h[6]);
							quad(p + p8, h[1], h[3], h[5], h[7]);
						}
						else if(q0 == 0)
						{
							quad(0u, h[0], h[6], h[4], h[2]);
							quad(p8, h[7], h[5], h[3], h[1]);
						}
						else
						{
							quad(pm, h[7], h[5], h[3], h[1]);
							quad(pm + p8, h[6], h[4], h[2], h[0]);
						}
					}
					else if(!mirror)
						quad(p, h[0], h[1], h[2], h[3]);
					else if(q0 == 0)
						quad(0u, edge, h[3], h[2], h[1]);
					else
						quad(pm, h[3], h[2], h[1], h[0]);
				}
			}
			else
			{
				const int64_t obase = spec_off + (int64_t)t * prow * nchan;
#pragma unroll
				for(int jj = 0; jj < J; jj++)
				{
					const int q = bt + jj * TPF;
					cf y[RL];
#pragma unroll
					for(int r = 0; r < RL; r++)
						y[r] = lds(src + st_index<sL, (N >= 8192)>(q, r));
					dftR<RL>(y);
					if(!tok)
						continue;
#pragma unroll
					for(int r = 0; r < RL; r++)
					{
						const int k = q + sL * r;
						int c, ce;
						float cj = 1.0f;
						if constexpr(CPLX)
						{
							// every bin is a channel; the lower sideband keeps bin 0 and
							// mirrors and conjugates the rest (mode.cpp:1217-1226)
							if(!lsb)
							{
								c = k;
								ce = k;
							}
							else
							{
								c = k == 0 ? 0 : N - k;
								ce = c - nchan;
								cj = k == 0 ? 1.0f : -1.0f;
							}
						}
						else if(!lsb)
						{
							if(r >= RL / 2)
								continue;                  // bins >= nchan
							c = k;
							ce = k;
						}
						else if(!mirror)
						{
							if(r < RL / 2)
								continue;
							c = k - nchan;
							ce = c - nchan;
						}
						else
						{
							if(!(k >= 1 && k <= nchan))
								continue;
							c = nchan - k;
							ce = c - nchan;
							cj = -1.0f;
						}
						if(row0 < 0)
							continue;
						const float fce = (float)ce;
						float th = fce * dhi;               // exact (split_turns)
						th -= rintf(th);
						float turns = th + fmaf(fce, dlo, postf + ph0);
						turns -= rintf(turns);
						float sn, cs;
						__sincosf(6.283185307179586f * turns, &sn, &cs);
						const float xr = y[r].x, xi = cj * y[r].y;
						((float2 *)a.spec + obase + c)[(int64_t)row0 * nchan] = make_float2(xr * cs - xi * sn, xr * sn + xi * cs);
					}
				}
			}
		}
	}
}

// The units of a persistent launch's work-list class in turn (counter ctr,
// zero before the launch); the next unit's number is fetched while this one
// runs.  Every thread of the CTA calls; the calls are barriers.
struct UnitFeed {
	int32_t *ctr;
	int *slot;                           // [2], shared
	int k = 0;
	__device__ __forceinline__ UnitFeed(int32_t *c, int *s) : ctr(c), slot(s) {}
	__device__ __forceinline__ int first()
	{
		if(threadIdx.x == 0)
			slot[0] = atomicAdd(ctr, 1);
		return next();
	}
	__device__ __forceinline__ int next()
	{
		__syncthreads();
		const int u = slot[k];
		k ^= 1;
		if(threadIdx.x == 0)
			slot[k] = atomicAdd(ctr, 1);
		return u;
	}
};

static inline dim3 fstage_grid(const FKind &k, const FsArgs &a)
{
	const int per = k.tq * k.fpc, nt = (a.T + per - 1) / per;
	return a.items_fast ? dim3(k.count, nt) : dim3(nt, k.count);
}

template <typename K>
static void fs_launch_persistent(K kern, const FsMultiArgs &m, int cls, int ctas, int threads, size_t smem,
                                 cudaStream_t st)
{
	cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
	cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
	kern<<<m.nunit[cls] < ctas ? m.nunit[cls] : ctas, threads, smem, st>>>(m);
}

}  // namespace fxb
