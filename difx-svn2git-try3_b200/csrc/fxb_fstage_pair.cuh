// F stage of a work item with both polarisations of a subband (device code;
// fxb_fstage.cuh has the stage's description and its one-band form).
//
// The two bands of a subband share their FFT times, fringe rotation,
// fractional-sample rotation and twiddles; only their samples differ.  A value
// is therefore a pair of bands, held as two packed registers (band 0, band 1)
// of real and of imaginary parts:
//  - the butterflies' additions are packed FP32 (add.rn.f32x2), half the
//    instructions; products with a scalar (twiddles, rotators) use the two
//    halves as plain registers, which costs no moves;
//  - an exchange element is 16 bytes, so that a shared-memory instruction
//    carries both bands; element i sits at i + i / 8, free of bank conflicts
//    for every pass;
//  - the sideband's half of the last pass alone is computed: its outputs k and
//    k + N/2 differ by the sign of the odd inputs, which the packed FMA takes
//    as a factor, so that one code serves both sidebands;
//  - a thread's four output channels are N/8 apart: their fractional-sample
//    rotators follow from the first by one step per FFT, computed once;
//  - the window of a valid FFT in frames of at least N/8 samples is read with
//    one running bit position, bands side by side with one load a sample, bands
//    apart with two; other windows track frames and validity.  All of a thread's
//    loads are issued before the first value is used (one sample after the other: 10
//    stations x 8 subbands x 2 polarisations apart, 2048 points, FP32 383 us a launch,
//    370 before the pairs, 251 now; in FP16 415, 433 and 300; complex, 4 subbands, 1024
//    points, FP16 125 and 95; 30 % of the frames invalid, 8192 points 456 and 415).
// An FFT of up to 256 points lies within a warp and exchanges without CTA
// barriers, one of 512 or 1024 points synchronises its own threads only.
//
// Subbands of one polarisation pair up two by two, if they agree in sideband and
// spectra and carry no corrections of their own: the fringe rotations then differ
// too (kPTwo) and cost one packed product more per sample pair, against a whole
// second pass over the FFT.
//
// Bound: shared-memory data pipe (about 70 % busy) and instruction issue.  Launch
// times in us, one band a unit and now: 10 stations x 16 bands x 250 FFTs of 2048
// points FP32 342 and 239; 20 x 2 x 8192 points x 128 FFTs of 8 bits 290 and 220;
// 20 x 8 x 256 points x 4096 709 and 434; the first in FP16 from raw multi-thread
// reads 523 and 304; 7 x 16 bands of one polarisation x 128 points x 2005 154 and 71.
#pragma once

#include "fxb_fstage.cuh"

namespace fxb {

namespace {

// one complex value of both bands: (band 0, band 1) real and imaginary parts
struct cp {
	u64 re, im;
};

__device__ __forceinline__ cp add(cp a, cp b) { return {add2(a.re, b.re), add2(a.im, b.im)}; }
__device__ __forceinline__ cp sub(cp a, cp b) { return {sub2(a.re, b.re), sub2(a.im, b.im)}; }
__device__ __forceinline__ cp add_mi(cp a, cp b) { return {add2(a.re, b.im), sub2(a.im, b.re)}; }   // a - i b
__device__ __forceinline__ cp add_pi(cp a, cp b) { return {sub2(a.re, b.im), add2(a.im, b.re)}; }   // a + i b
__device__ __forceinline__ cp rot45(cp a)                                                            // a (1 - i) / sqrt2
{
	const u64 r = pk2(0.70710678118654752440f, 0.70710678118654752440f);
	return {mul2(add2(a.re, a.im), r), mul2(sub2(a.im, a.re), r)};
}
// rounded in one fixed way, so that every instance of the code agrees
__device__ __forceinline__ void rot1(float &x, float &y, float c, float s)
{
	const float xr = fmaf(x, c, -__fmul_rn(y, s)), xi = fmaf(x, s, __fmul_rn(y, c));
	x = xr;
	y = xi;
}
__device__ __forceinline__ cp twid(cp a, float2 w)
{
	float2 r = up2(a.re), i = up2(a.im);
	rot1(r.x, i.x, w.x, w.y);
	rot1(r.y, i.y, w.x, w.y);
	return {pk2(r.x, r.y), pk2(i.x, i.y)};
}

// outputs 0 .. R/2 - 1 of the R-point DFT with the odd inputs times sg (1: the
// first R/2 bins, -1: the second R/2); nsg = -sg
template <int R>
__device__ __forceinline__ void dft_half(const cp *x, cp *y, u64 sg, u64 nsg)
{
	if constexpr(R == 8)
	{
		const cp a0 = add(x[0], x[4]), d0 = sub(x[0], x[4]), a2 = add(x[2], x[6]), d2 = sub(x[2], x[6]);
		const cp a1 = add(x[1], x[5]), d1 = sub(x[1], x[5]), a3 = add(x[3], x[7]), d3 = sub(x[3], x[7]);
		const cp b0 = add(a0, a2), b2 = sub(a0, a2), b1 = add(a1, a3), b3 = sub(a1, a3);
		const cp f0 = add_mi(d0, d2), f2 = add_pi(d0, d2);
		const cp f1 = rot45(add_mi(d1, d3)), f3 = rot45(add_pi(d1, d3));
		y[0] = {fma2(b1.re, sg, b0.re), fma2(b1.im, sg, b0.im)};
		y[1] = {fma2(f1.re, sg, f0.re), fma2(f1.im, sg, f0.im)};
		y[2] = {fma2(b3.im, sg, b2.re), fma2(b3.re, nsg, b2.im)};
		y[3] = {fma2(f3.im, sg, f2.re), fma2(f3.re, nsg, f2.im)};
	}
	else if constexpr(R == 4)
	{
		const cp b0 = add(x[0], x[2]), b2 = sub(x[0], x[2]), b1 = add(x[1], x[3]), b3 = sub(x[1], x[3]);
		y[0] = {fma2(b1.re, sg, b0.re), fma2(b1.im, sg, b0.im)};
		y[1] = {fma2(b3.im, sg, b2.re), fma2(b3.re, nsg, b2.im)};
	}
	else
		y[0] = {fma2(x[1].re, sg, x[0].re), fma2(x[1].im, sg, x[0].im)};
}

__device__ __forceinline__ constexpr int ppad(int i) { return i + (i >> 3); }

__device__ __forceinline__ cp ldx(const ulonglong2 *p)
{
	const ulonglong2 v = *p;
	return {v.x, v.y};
}
__device__ __forceinline__ void stx(ulonglong2 *p, cp v) { *p = make_ulonglong2(v.re, v.im); }

// exp(2 pi i x) of a double, rounded once (the float angle's remainder enters
// to first order)
__device__ __forceinline__ float2 cispi2(double x)
{
	const double y = 2.0 * (x - rint(x));
	const float yf = (float)y, dy = (float)(y - (double)yf) * 3.14159265358979f;
	float s, c;
	sincospif(yf, &s, &c);
	return make_float2(fmaf(-s, dy, c), fmaf(c, dy, s));
}

// Threads, slots (FFTs side by side) and exchange buffer of length 2^LOGN.
template <int LOGN>
struct PShape {
	static constexpr int N = 1 << LOGN;
	static constexpr int TPF = N / 8;                        // threads per FFT, one butterfly each
	static constexpr int NT = TPF > 256 ? TPF : 256;
	static constexpr int FPC = NT / TPF;
	static constexpr int PADN = N + N / 8;                   // elements of 16 bytes
	static constexpr int NMID = (LOGN % 3 == 0) ? LOGN / 3 - 2 : LOGN / 3 - 1;
	static constexpr int RL = (LOGN % 3 == 0) ? 8 : (1 << (LOGN % 3));
	// CTAs per SM: 80 registers up to 2048 points, 64 above
	static constexpr int MINB = NT == 256 ? 3 : 1024 / NT;
};

// the threads of one FFT meet
template <int LOGN>
__device__ __forceinline__ void slot_sync(int slot)
{
	using SH = PShape<LOGN>;
	if constexpr(SH::TPF <= 32)
		__syncwarp();
	else if constexpr(SH::FPC > 1)
		asm volatile("bar.sync %0, %1;\n" ::"r"(1 + slot), "n"(SH::TPF) : "memory");
	else
		__syncthreads();
}

// One middle radix-8 pass (stride s = 2^LOGS, m = N / (8 s)): x_r = X[q + s (p
// + r m)], y = DFT8(x), Y[q + s (8 p + r)] = y_r w_N^(r p s).
template <int LOGN, int LOGS>
__device__ __forceinline__ void pair_mid(ulonglong2 *side, int slot, int b, const float2 *twp)
{
	using SH = PShape<LOGN>;
	constexpr int N = SH::N, s = 1 << LOGS, np = N / (8 * s);
	const int q = b & (s - 1), p8 = b >> LOGS;
	cp x[8];
#pragma unroll
	for(int r = 0; r < 8; r++)
	{
		// N/8 a multiple of 8 (N >= 64): the padding is a constant offset per r
		if constexpr(N >= 64)
			x[r] = ldx(side + ppad(b) + r * ppad(N / 8));
		else
			x[r] = ldx(side + ppad(b + r * (N / 8)));
	}
	float2 w[8];
#pragma unroll
	for(int r = 1; r < 8; r++)
		w[r] = ldtw(twp, (r - 1) * np + p8);
	dft8(x);
#pragma unroll
	for(int r = 1; r < 8; r++)
		x[r] = twid(x[r], w[r]);
	slot_sync<LOGN>(slot);
	// s is a multiple of 8, so is q + 8 s p8 + s r - q: constant offsets again
	ulonglong2 *o = side + ppad(q + s * 8 * p8);
#pragma unroll
	for(int r = 0; r < 8; r++)
		stx(o + r * ppad(s), x[r]);
	slot_sync<LOGN>(slot);
}

template <int LOGN, int PS>
__device__ __forceinline__ void pair_mids(ulonglong2 *side, int slot, int b, const float2 *tw)
{
	if constexpr(PS < PShape<LOGN>::NMID)
	{
		pair_mid<LOGN, 3 * (PS + 1)>(side, slot, b, tw + tw_offset(1 << LOGN, PS + 1));
		pair_mids<LOGN, PS + 1>(side, slot, b, tw);
	}
}

}  // namespace

// One work unit: FFT times t0 .. of an item of two bands, run by the CTA's
// PShape<LOGN>::NT threads in nit rounds.  I: the item, fcs: the constants of its
// FFTs from t0 on, both in shared memory.
// VAR 1: raw INTERLACEDVDIF reads; VAR 2: complex sampling.
template <int LOGN, bool TCO, int VAR>
__device__ __forceinline__ void fstage_pair_unit(const FsArgs &a, const PairItem &I, const PairConst *fcs,
                                                 const PairTwist *tws, const int t0, const int nit, const float2 *tw,
                                                 ulonglong2 *fsm, const float *lut8, const u64 *lut4)
{
	using SH = PShape<LOGN>;
	constexpr int N = SH::N, TPF = SH::TPF, FPC = SH::FPC, PADN = SH::PADN, RL = SH::RL;
	constexpr bool MUX = VAR == 1, CPLX = VAR == 2;
	constexpr int nchan = CPLX ? N : N / 2;
	constexpr uint32_t S8 = N / 8;
	const uint32_t fs = I.fs, bpt = I.bpt;
	const int nbits = I.nbits;
	const int slot = threadIdx.x / TPF, b = threadIdx.x - slot * TPF;
	ulonglong2 *const side = fsm + (size_t)slot * PADN;
	const bool lsb = I.lsb != 0;
	const int order = a.order;
	constexpr float osc = TCO ? 1.0f / (float)(1 << kTcSpecExp) : 1.0f;

	for(int it = 0; it < nit; it++)
	{
		const int t = t0 + it * FPC + slot;
		const PairConst &fc = fcs[it * FPC + slot];
		// constants past T are not there: such slots take part in the barriers only
		const int flags = t < a.T ? fc.flags : 0;
		// ---- 1. decode: the levels of samples b + r N/8 of both bands
		u64 lv[8], lu[CPLX ? 8 : 1];        // lu: imaginary parts (complex sampling)
		const uint32_t xs = fc.so + (uint32_t)b;
		// Every load is on its way before the first value is used.  A word holds the
		// fields of both bands side by side, or each band has a word of its own.
		// (the same code for 2 and 8 bits: kernels of many lengths fetch it over and over)
		auto levels = [&](int r, const float *tab, uint32_t w0, uint32_t w1) {
			const uint32_t mask = (1u << nbits) - 1u;
			lv[r] = pk2(tab[w0 & mask], tab[w1 & mask]);
			if constexpr(CPLX)
				lu[r] = pk2(tab[(w0 >> nbits) & mask], tab[(w1 >> nbits) & mask]);
		};
		auto table = [&]() { return lut8 + (nbits == 2 ? 256 : 0); };
		if(!MUX && (flags & kPFast))
		{
			// one running bit position: a frame boundary skips a header
			// (so < fs and b < N/8 <= fs: at most one boundary before sample b)
			const uint32_t hbits = I.hbits;
			uint32_t tin = xs, bit = xs * bpt + I.boff0;
			if(tin >= fs)
			{
				tin -= fs;
				bit += hbits;
			}
			const uint32_t *wp = (const uint32_t *)fc.wp;
			uint32_t raw[8], sh[8];
#pragma unroll
			for(int r = 0; r < 8; r++)
			{
				raw[r] = __ldg(wp + (bit >> 5));
				sh[r] = bit & 31u;
				tin += S8;
				bit += S8 * bpt;
				if(tin >= fs)
				{
					tin -= fs;
					bit += hbits;
				}
			}
			if constexpr(CPLX)
			{
				const float *tab = table();
				const uint32_t apart = I.boff1 - I.boff0;
#pragma unroll
				for(int r = 0; r < 8; r++)
				{
					const uint32_t w = raw[r] >> sh[r];
					levels(r, tab, w, w >> apart);
				}
			}
			else if(nbits == 2)
			{
#pragma unroll
				for(int r = 0; r < 8; r++)
					lv[r] = lut4[(raw[r] >> sh[r]) & 15u];
			}
			else
			{
#pragma unroll
				for(int r = 0; r < 8; r++)
				{
					const uint32_t w = raw[r] >> sh[r];
					lv[r] = pk2(lut8[w & 255u], lut8[(w >> 8) & 255u]);
				}
			}
		}
		else if(MUX && (flags & kPFast))
		{
			const uint8_t *buf = fc.wp + 32;
			const int minfb = I.minfb;
			const uint8_t *f00 = buf + (int64_t)fc.mi00 * minfb, *f01 = buf + (int64_t)fc.mi01 * minfb;
			const uint8_t *f10 = buf + (int64_t)fc.mi10 * minfb, *f11 = buf + (int64_t)fc.mi11 * minfb;
			uint32_t raw0[8], raw1[8], sh[8];
#pragma unroll
			for(int r = 0; r < 8; r++)
			{
				const uint32_t x = xs + r * S8;
				const bool second = x >= fs;
				const uint32_t bit = (second ? x - fs : x) * bpt;
				raw0[r] = __ldg((const uint32_t *)(second ? f10 : f00) + (bit >> 5));
				raw1[r] = __ldg((const uint32_t *)(second ? f11 : f01) + (bit >> 5));
				sh[r] = bit & 31u;
			}
			const float *tab = table();
#pragma unroll
			for(int r = 0; r < 8; r++)
				levels(r, tab, raw0[r] >> sh[r], raw1[r] >> sh[r]);
		}
		else if(!MUX && (flags & kPApart))
		{
			// the same with a word for each band
			const uint32_t hbits = I.hbits, apart = I.boff1 - I.boff0;
			uint32_t tin = xs, bit = xs * bpt + I.boff0;
			if(tin >= fs)
			{
				tin -= fs;
				bit += hbits;
			}
			const uint32_t *wp = (const uint32_t *)fc.wp;
			uint32_t raw0[8], raw1[8], sh[8];
#pragma unroll
			for(int r = 0; r < 8; r++)
			{
				raw0[r] = __ldg(wp + (bit >> 5));
				raw1[r] = __ldg(wp + ((bit + apart) >> 5));
				sh[r] = bit & 31u;
				tin += S8;
				bit += S8 * bpt;
				if(tin >= fs)
				{
					tin -= fs;
					bit += hbits;
				}
			}
			const float *tab = table();
#pragma unroll
			for(int r = 0; r < 8; r++)
				levels(r, tab, raw0[r] >> sh[r], raw1[r] >> ((sh[r] + apart) & 31u));
		}
		else if(flags & kPActive)
		{
			// frames, validity and blanking sample by sample
			const bool narrow = (flags & kPNarrow) != 0, blank = (flags & kPBlank) != 0;
			const int station = I.station, minfb = I.minfb;
			const uint8_t *buf = a.sub[station].buf, *vrow = a.valid + (int64_t)station * a.valid_stride;
			const int32_t *mslot = MUX ? a.sub[station].mux_slot : nullptr;
			const int64_t mk0 = MUX ? a.sub[station].mux_k0 : 0;
			const bool oneword = !MUX && bpt <= 32;              // all bands of a sample time in one word
			const uint32_t apart = MUX ? 0u : I.boff1 - I.boff0;
			uint32_t kf = xs / fs, tin = xs - kf * fs;
			const uint8_t *fp = MUX ? buf + 32 : buf + ((int64_t)fc.fa + kf) * I.framebytes + I.header;
			uint32_t raw0[8], raw1[8], pk[8];
#pragma unroll
			for(int r = 0; r < 8; r++)
			{
				const int n = b + r * (int)S8;
				const int64_t fr = (int64_t)fc.fa + kf;
				bool ok;
				if(narrow)
					ok = (fc.fmask >> kf) & 1u;
				else
					ok = fr < a.valid_stride && vrow[fr] != 0;
				ok = ok && n < fc.stuck;
				const uint32_t bit = tin * bpt + I.boff0;
				if constexpr(MUX)
				{
					const int32_t *slr = mslot + (mk0 + fr) * I.mnthr;
					const int i0 = ok ? __ldg(slr + I.band0) : -1, i1 = ok ? __ldg(slr + I.band1) : -1;
					raw0[r] = i0 >= 0 ? __ldg((const uint32_t *)(fp + (int64_t)i0 * minfb) + (bit >> 5)) : 0u;
					raw1[r] = i1 >= 0 ? __ldg((const uint32_t *)(fp + (int64_t)i1 * minfb) + (bit >> 5)) : 0u;
				}
				else
				{
					raw0[r] = ok ? __ldg((const uint32_t *)fp + (bit >> 5)) : 0u;
					raw1[r] = ok && !oneword ? __ldg((const uint32_t *)fp + ((bit + apart) >> 5)) : 0u;
				}
				pk[r] = (bit & 31u) | (ok ? 32u : 0u);
				tin += S8;
				while(tin >= fs)
				{
					tin -= fs;
					kf++;
					if constexpr(!MUX)
						fp += I.framebytes;
				}
			}
			const float *tab = table();
#pragma unroll
			for(int r = 0; r < 8; r++)
			{
				lv[r] = 0ull;
				if constexpr(CPLX)
					lu[r] = 0ull;
				if(!(pk[r] & 32u))
					continue;
				const uint32_t sh0 = pk[r] & 31u;
				levels(r, tab, raw0[r] >> sh0, (oneword ? raw0[r] : raw1[r]) >> ((sh0 + apart) & 31u));
				if(blank)
				{
					// bands of this sample's frame blanked by its EDV4 validity mask
					// (blank_vdif_EDV4, format_vdif.c:4699-4780)
					const uint32_t bo = a.bandok[(int64_t)station * a.valid_stride + fc.fa + (xs + r * S8) / fs];
					const bool v0 = (bo >> I.band0) & 1u, v1 = (bo >> I.band1) & 1u;
					const float2 l = up2(lv[r]);
					lv[r] = pk2(v0 ? l.x : 0.0f, v1 ? l.y : 0.0f);
					if constexpr(CPLX)
					{
						const float2 u = up2(lu[r]);
						lu[r] = pk2(v0 ? u.x : 0.0f, v1 ? u.y : 0.0f);
					}
				}
			}
		}
		else
		{
			// no FFT, or past T: nothing to read (as windows without a valid frame these
			// slots kept the last unit waiting for code that nothing else ran)
#pragma unroll
			for(int r = 0; r < 8; r++)
			{
				lv[r] = 0ull;
				if constexpr(CPLX)
					lu[r] = 0ull;
			}
		}
		// ---- 2. fringe rotation (order 1: the rotator of sample b, then one
		// complex step per N/8 samples), first radix-8 pass (butterfly b, twiddle
		// w_N^(r b))
		cp x[8];
		{
			// rotator of sample n: order 1 the start, order 2 every sample
			auto start = [&](float P0, float alpha, float &rc, float &rs) {
				float ph = fmaf((float)b, alpha, P0);
				ph -= rintf(ph);
				__sincosf(-6.283185307179586f * ph, &rs, &rc);
			};
			auto quadr = [&](int n, float P0, float alpha, float beta, float gamma, float eps, float &rc, float &rs) {
				const int asl = I.asl, kk = n / asl, jj = n - kk * asl;
				float ph = P0 + (float)jj * alpha + (float)(kk * jj) * beta + (float)kk * gamma + (float)(kk * kk) * eps;
				ph -= rintf(ph);
				__sincosf(-6.283185307179586f * ph, &rs, &rc);
			};
			auto value = [&](int r, float rc, float rs, float rcb, float rsb) {
				const float2 v = up2(lv[r]);
				if constexpr(CPLX)
				{
					const float2 u = up2(lu[r]);
					x[r].re = pk2(fmaf(v.x, rc, -__fmul_rn(u.x, rs)), fmaf(v.y, rcb, -__fmul_rn(u.y, rsb)));
					x[r].im = pk2(fmaf(v.x, rs, __fmul_rn(u.x, rc)), fmaf(v.y, rsb, __fmul_rn(u.y, rcb)));
				}
				else
				{
					x[r].re = pk2(__fmul_rn(v.x, rc), __fmul_rn(v.y, rcb));
					x[r].im = pk2(__fmul_rn(v.x, rs), __fmul_rn(v.y, rsb));
				}
			};
			float rc = 1.0f, rs = 0.0f;
			const float2 st = fc.st;
			if(order == 1)
				start(fc.P0, fc.alpha, rc, rs);
			if(!(flags & kPTwo))
			{
#pragma unroll
				for(int r = 0; r < 8; r++)
				{
					if(order == 2)
						quadr(b + r * (int)S8, fc.P0, fc.alpha, fc.beta, fc.gamma, fc.eps, rc, rs);
					value(r, rc, rs, rc, rs);
					if(order == 1 && r < 7)
						rot1(rc, rs, st.x, st.y);
				}
			}
			else
			{
				float rcb = 1.0f, rsb = 0.0f;
				const PairTwist &ft = tws[it * FPC + slot];
				const float2 stb = ft.st;
				if(order == 1)
					start(ft.P0, ft.alpha, rcb, rsb);
#pragma unroll
				for(int r = 0; r < 8; r++)
				{
					if(order == 2)
					{
						quadr(b + r * (int)S8, fc.P0, fc.alpha, fc.beta, fc.gamma, fc.eps, rc, rs);
						quadr(b + r * (int)S8, ft.P0, ft.alpha, ft.beta, ft.gamma, ft.eps, rcb, rsb);
					}
					value(r, rc, rs, rcb, rsb);
					if(order == 1 && r < 7)
					{
						rot1(rc, rs, st.x, st.y);
						rot1(rcb, rsb, stb.x, stb.y);
					}
				}
			}
		}
		dft8(x);
#pragma unroll
		for(int r = 1; r < 8; r++)
			x[r] = twid(x[r], ldtw(tw, (r - 1) * (N / 8) + b));
		slot_sync<LOGN>(slot);              // the exchange buffer has been read by the last FFT
		{
			ulonglong2 *o = side + ppad(8 * b);
#pragma unroll
			for(int r = 0; r < 8; r++)
				stx(o + r, x[r]);
		}
		slot_sync<LOGN>(slot);
		// ---- 3. middle radix-8 passes through shared memory
		pair_mids<LOGN, 0>(side, slot, b, tw);
		// ---- 4. last pass, sideband, fractional-sample rotation, output
		if(t >= a.T)
			continue;
		constexpr int sL = N / RL, J = 8 / RL;
		const bool same = (flags & kPSame) != 0;
		const int oflags = I.oflags;
		const bool h16 = (oflags & kOH16) != 0;
		const int64_t rowd = I.rowd;
		const int64_t base = I.first + (int64_t)t * I.tstride;
		auto put = [&](int c, const cp &y) {
			const float2 re = up2(y.re), im = up2(y.im);
			float2 *o = (float2 *)a.spec + base + c;
			if(oflags & kORow0)
				*o = make_float2(re.x, im.x);
			if(oflags & kORow1)
				o[rowd] = make_float2(re.y, im.y);
		};
		// Tensor-core form: the four values of each band at positions p0 .. p0 + 3
		// (chan_pos) at once; blocks of two channels whose rows of the two bands are an
		// aligned pair take both bands in one store.
		auto quad = [&](uint32_t p0, uint4 v0, uint4 v1) {
			uint32_t *o = (uint32_t *)a.spec + base;
			const uint32_t bextra = I.bextra;
			if(oflags & kOWide)
			{
				o += p0 + (p0 >> I.shift) * bextra;
				if(oflags & kORow0)
					*(uint4 *)o = v0;
				if(oflags & kORow1)
					*(uint4 *)(o + rowd) = v1;
			}
			else if(oflags & kOBoth)
			{
				o += p0 + (p0 >> 1) * bextra;
				*(uint4 *)o = make_uint4(v0.x, v0.y, v1.x, v1.y);
				*(uint4 *)(o + bextra + 2) = make_uint4(v0.z, v0.w, v1.z, v1.w);
			}
			else
			{
				if(oflags & kORow0)
					store_quad(o, p0, I.tcb, I.magic, bextra, v0);
				if(oflags & kORow1)
					store_quad(o + rowd, p0, I.tcb, I.magic, bextra, v1);
			}
		};
		auto packed = [&](const cp &y, uint32_t &h0, uint32_t &h1) {
			const float2 re = up2(y.re), im = up2(y.im);
			h0 = pack_spec(h16, re.x, im.x);
			h1 = pack_spec(h16, re.y, im.y);
		};
		// y conjugated when cj < 0, times the bands' rotators
		auto turn = [](const cp &y, float cj, float2 w0, float2 w1) {
			float2 re = up2(y.re), im = up2(y.im);
			im.x *= cj;
			im.y *= cj;
			rot1(re.x, im.x, w0.x, w0.y);
			rot1(re.y, im.y, w1.x, w1.y);
			return cp{pk2(re.x, re.y), pk2(im.x, im.y)};
		};
		// rotator exp(2 pi i (ce D + post)) of band j at effective channel ce,
		// D = hi + lo (ce hi exact), times the spectra's scale
		auto rotator = [&](int j, int ce) {
			const float fce = (float)ce;
			float h = fce * fc.dhi[j];
			h -= rintf(h);
			float turns = h + fmaf(fce, fc.dlo[j], fc.post[j]);
			turns -= rintf(turns);
			float2 w;
			__sincosf(6.283185307179586f * turns, &w.y, &w.x);
			w.x *= osc;
			w.y *= osc;
			return w;
		};
		if constexpr(CPLX)
		{
			// every bin is a channel; the lower sideband keeps bin 0 and mirrors and
			// conjugates the rest (mode.cpp:1217-1226).  Output m of the thread is bin b +
			// m N/8: the even ones are the channels of one quad of positions, the odd ones
			// of another, in descending order in the lower sideband.  Two bands of four
			// subbands, 1024 channels, 2 bits, 10 stations, F stage: 142 us in the order of
			// channels, 187 in that of chan_pos one by one, 125 a quad at a time.
			auto value = [&](const cp &y, int k) {
				const int ce = lsb ? (k == 0 ? -N : -k) : k;
				const float2 w0 = rotator(0, ce), w1 = same ? w0 : rotator(1, ce);
				return turn(y, !lsb || k == 0 ? 1.0f : -1.0f, w0, w1);
			};
			auto load = [&](cp *y, int jj) {
#pragma unroll
				for(int r = 0; r < RL; r++)
					y[r] = ldx(side + ppad(b + jj * TPF + sL * r));
				dftR<RL>(y);
			};
			if constexpr(!TCO)
			{
#pragma unroll
				for(int jj = 0; jj < J; jj++)
				{
					cp y[RL];
					load(y, jj);
#pragma unroll
					for(int r = 0; r < RL; r++)
					{
						const int k = b + jj * TPF + sL * r;
						put(!lsb || k == 0 ? k : N - k, value(y[r], k));
					}
				}
			}
			else
			{
				cp y[RL];
#pragma unroll
				for(int par = 0; par < 2; par++)
				{
					uint32_t h0[4], h1[4];
#pragma unroll
					for(int g = 0; g < (J + 1) / 2; g++)
					{
						// group jj holds the outputs m = jj + r J
						const int jj = J == 1 ? 0 : par + 2 * g;
						if(J > 1 || par == 0)
							load(y, jj);
#pragma unroll
						for(int r = 0; r < RL; r++)
						{
							const int m = jj + r * J;
							if((m & 1) == par)
								packed(value(y[r], b + m * (int)S8), h0[m >> 1], h1[m >> 1]);
						}
					}
					const uint4 up0 = make_uint4(h0[0], h0[1], h0[2], h0[3]), up1 = make_uint4(h1[0], h1[1], h1[2], h1[3]);
					const uint4 dn0 = make_uint4(h0[3], h0[2], h0[1], h0[0]), dn1 = make_uint4(h1[3], h1[2], h1[1], h1[0]);
					const uint32_t p = 4u * (uint32_t)b, half = (uint32_t)(N / 2);
					if(!lsb)
						quad(p + (par ? half : 0u), up0, up1);
					else if(b > 0)
						quad(half - p + (par ? 0u : half), dn0, dn1);
					else if(par)
						quad(half, dn0, dn1);
					else
						quad(0u, make_uint4(h0[0], h0[3], h0[2], h0[1]), make_uint4(h1[0], h1[3], h1[2], h1[1]));
				}
			}
		}
		else
		{
			// the thread's outputs are bins kb + b + m N/8, m = 0 .. 3: channel m N/8 +
			// b of the sideband; order-0 lower sideband: channel nchan - k, conjugated
			const bool mirror = lsb && order == 0;
			const float sgf = lsb && !mirror ? -1.0f : 1.0f;
			const u64 sg = pk2(sgf, sgf), nsg = pk2(-sgf, -sgf);
			const int ce = mirror ? -b : (lsb ? b - nchan : b);
			float2 w0 = rotator(0, ce), w1 = same ? w0 : rotator(1, ce);
			const float2 os0 = fc.os[0], os1 = fc.os[1];
			cp y[4];
#pragma unroll
			for(int jj = 0; jj < J; jj++)
			{
				cp z[RL], h[RL / 2];
#pragma unroll
				for(int r = 0; r < RL; r++)
				{
					if constexpr(N >= 64)
						z[r] = ldx(side + ppad(b) + jj * ppad(TPF) + r * ppad(sL));
					else
						z[r] = ldx(side + ppad(b + jj * TPF + sL * r));
				}
				dft_half<RL>(z, h, sg, nsg);
				// output r of group jj is bin b + jj N/8 + r N/RL
#pragma unroll
				for(int r = 0; r < RL / 2; r++)
					y[jj + r * J] = h[r];
				if(mirror && jj == 0 && b == 0)
				{
					// bin N/2, channel 0
					const float2 m0 = rotator(0, -nchan), m1 = same ? m0 : rotator(1, -nchan);
					dft_half<RL>(z, h, nsg, sg);
					const cp e = turn(h[0], -1.0f, m0, m1);
					if constexpr(TCO)
					{
						uint32_t *o = (uint32_t *)a.spec + base, e0, e1;
						packed(e, e0, e1);
						if(oflags & kORow0)
							*o = e0;
						if(oflags & kORow1)
							o[rowd] = e1;
					}
					else
						put(0, e);
				}
			}
#pragma unroll
			for(int m = 0; m < 4; m++)
			{
				if(mirror)
					y[m] = turn(y[m], -1.0f, w0, w1);
				else
				{
					float2 re = up2(y[m].re), im = up2(y[m].im);
					rot1(re.x, im.x, w0.x, w0.y);
					rot1(re.y, im.y, w1.x, w1.y);
					y[m] = cp{pk2(re.x, re.y), pk2(im.x, im.y)};
				}
				if(m < 3)
				{
					rot1(w0.x, w0.y, os0.x, os0.y);
					if(same)
						w1 = w0;
					else
						rot1(w1.x, w1.y, os1.x, os1.y);
				}
			}
			if constexpr(TCO)
			{
				uint32_t h0[4], h1[4];
#pragma unroll
				for(int m = 0; m < 4; m++)
					packed(y[m], h0[m], h1[m]);
				const uint32_t p = 4u * (uint32_t)b;
				const uint4 up0 = make_uint4(h0[0], h0[1], h0[2], h0[3]), up1 = make_uint4(h1[0], h1[1], h1[2], h1[3]);
				const uint4 dn0 = make_uint4(h0[3], h0[2], h0[1], h0[0]), dn1 = make_uint4(h1[3], h1[2], h1[1], h1[0]);
				if(!mirror)
					quad(p, up0, up1);
				else if(b > 0)
					quad((uint32_t)(N / 2) - p, dn0, dn1);
				else
				{
					// beside channel 0 (bin N/2, above)
#pragma unroll
					for(uint32_t m = 1; m < 4; m++)
					{
						uint32_t *o = (uint32_t *)a.spec + base + m + __umulhi(m, I.magic) * I.bextra;
						if(oflags & kORow0)
							*o = h0[4 - m];
						if(oflags & kORow1)
							o[rowd] = h1[4 - m];
					}
				}
			}
			else
			{
#pragma unroll
				for(int m = 0; m < 4; m++)
				{
					const int k = b + m * (int)S8;
					if(!mirror)
						put(k, y[m]);
					else if(k > 0)
						put(nchan - k, y[m]);
				}
			}
		}
	}
}

__device__ __forceinline__ void pair_cp16(void *dst, const void *src)
{
	asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void pair_cp_wait() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// a unit's item and constants into shared memory (pair_cp_wait and a barrier
// before they are read)
__device__ __forceinline__ void pair_fetch(PairItem *I, PairConst *fcs, PairTwist *tws, const void *item,
                                           const void *consts, const void *twists, int nfc)
{
	if(twists)
		for(int i = threadIdx.x; i < nfc * (int)(sizeof(PairTwist) / 16); i += blockDim.x)
			pair_cp16((char *)tws + 16 * i, (const char *)twists + 16 * i);
	for(int i = threadIdx.x; i < nfc * (int)(sizeof(PairConst) / 16); i += blockDim.x)
		pair_cp16((char *)fcs + 16 * i, (const char *)consts + 16 * i);
	if(threadIdx.x < sizeof(PairItem) / 16)
		pair_cp16((char *)I + 16 * threadIdx.x, (const char *)item + 16 * threadIdx.x);
}

// The units of a persistent launch's work-list class, CTAs striding over them
// (the units of a class cost about the same).  Fetched ahead: while unit k runs, the
// constants of k + 1 and the record of k + 2 are on their way, so that no unit
// waits for a chain of loads.
template <int NFC>
struct PairFeed {
	FsMultiUnit rec[3];
	PairItem item[2];
	PairConst fcs[2][NFC];
	PairTwist tws[2][NFC];
};

template <int NFC, class F>
__device__ __forceinline__ void pair_units(PairFeed<NFC> &s, const FsMultiArgs &m, const int cls, F &&run)
{
	static_assert(sizeof(FsMultiUnit) % 16 == 0 && sizeof(PairItem) % 16 == 0 && sizeof(PairConst) % 16 == 0, "copies");
	const FsMultiUnit *units = m.units + m.unit0[cls];
	const int n = m.nunit[cls], step = gridDim.x;
	constexpr int R16 = sizeof(FsMultiUnit) / 16;
	auto record = [&](int k, int u) {
		if(u < n && threadIdx.x < R16)
			pair_cp16((char *)&s.rec[k % 3] + 16 * threadIdx.x, (const char *)(units + u) + 16 * threadIdx.x);
	};
	auto consts = [&](int k, int u) {
		const FsMultiUnit &r = s.rec[k % 3];
		if(u < n)
			pair_fetch(&s.item[k & 1], s.fcs[k & 1], s.tws[k & 1], r.pitem, r.consts, r.twists, r.nfc);
	};
	int u = blockIdx.x;
	record(0, u);
	record(1, u + step);
	pair_cp_wait();
	__syncthreads();
	consts(0, u);
	for(int k = 0; u < n; k++, u += step)
	{
		pair_cp_wait();
		__syncthreads();
		consts(k + 1, u + step);
		record(k + 2, u + 2 * step);
		run(s.rec[k % 3], s.item[k & 1], s.fcs[k & 1], s.tws[k & 1]);
	}
}

// the level pairs of two adjacent 2-bit bands, and the 8-bit and 2-bit levels
__device__ __forceinline__ void fstage_pair_luts(float *lut8, u64 *lut4)
{
	for(int i = threadIdx.x; i < 256; i += blockDim.x)
		lut8[i] = (float)((i - 128) / 3.3);
	if(threadIdx.x < 4)
		lut8[256 + threadIdx.x] = level2(threadIdx.x);
	if(threadIdx.x < 16)
		lut4[threadIdx.x] = pk2(level2(threadIdx.x & 3u), level2(threadIdx.x >> 2u));
}

// One CTA per work unit (grid as k_fstage): the FP32 form, and complex sampling of the
// tensor-core forms, whose other kinds have persistent launches.
template <int LOGN, bool TCO, int VAR>
__global__ void __launch_bounds__(PShape<LOGN>::NT, PShape<LOGN>::MINB) k_fstage_pair(const FsArgs a)
{
	extern __shared__ __align__(16) ulonglong2 fsp[];
	constexpr int FPC = PShape<LOGN>::FPC;
	__shared__ float lut8[260];
	__shared__ u64 lut4[16];
	__shared__ PairConst fcs[kMaxTQ * FPC];
	__shared__ PairTwist tws[kMaxTQ * FPC];
	__shared__ PairItem I;
	const int item = a.pair0 + (a.items_fast ? blockIdx.x : blockIdx.y);
	const int t0 = (a.items_fast ? blockIdx.y : blockIdx.x) * a.tq * FPC, nfc = min(a.tq * FPC, a.T - t0);
	pair_fetch(&I, fcs, tws, a.pitems + item, a.pconst + (int64_t)item * a.T + t0,
	           a.two ? a.ptwist + (int64_t)(item - a.ptwist0) * a.T + t0 : nullptr, nfc);
	fstage_pair_luts(lut8, lut4);
	pair_cp_wait();
	__syncthreads();
	fstage_pair_unit<LOGN, TCO, VAR>(a, I, fcs, tws, t0, (nfc + FPC - 1) / FPC, (const float2 *)a.tw, fsp, lut8, lut4);
}

template <int LOGN, bool TCO, int VAR>
static void launch_t(const FKind &k, const FsArgs &a, cudaStream_t stream)
{
	cudaFuncSetAttribute(k_fstage_pair<LOGN, TCO, VAR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.smem);
	cudaFuncSetAttribute(k_fstage_pair<LOGN, TCO, VAR>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
	k_fstage_pair<LOGN, TCO, VAR><<<fstage_grid(k, a), k.threads, k.smem, stream>>>(a);
}

template <bool TCO, int VAR>
static void launch_var(const FKind &k, const FsArgs &a, cudaStream_t stream)
{
	switch(k.N)
	{
	case 32: launch_t<5, TCO, VAR>(k, a, stream); break;
	case 64: launch_t<6, TCO, VAR>(k, a, stream); break;
	case 128: launch_t<7, TCO, VAR>(k, a, stream); break;
	case 256: launch_t<8, TCO, VAR>(k, a, stream); break;
	case 512: launch_t<9, TCO, VAR>(k, a, stream); break;
	case 1024: launch_t<10, TCO, VAR>(k, a, stream); break;
	case 2048: launch_t<11, TCO, VAR>(k, a, stream); break;
	case 4096: launch_t<12, TCO, VAR>(k, a, stream); break;
	case 8192: launch_t<13, TCO, VAR>(k, a, stream); break;
	default: break;
	}
}

}  // namespace fxb
