// sm_100a kernels of the FX path: fused F stage, FP32 XMAC, weights,
// finalisation into the core-result layout, and the stand-alone VDIF decoder.

#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>

#include "fxb_internal.h"
#include "fxb_kernels.h"

namespace fxb {

// 2-bit code -> level, {-HiMag, -1, +1, +HiMag} with HiMag = 3.3359
// (libraries/mark5access/mark5access/format_vdif.c:48,78; mark5_stream.h:75).
__constant__ float c_lut2[4] = {-3.3359f, -1.0f, 1.0f, 3.3359f};
// 8-bit offset binary -> (b - 128) / 3.3 (format_vdif.c:122), filled from the host.
__constant__ float c_lut8[256];

cudaError_t upload_lut8(cudaStream_t stream);

__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
	return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// Sample (station-relative index g) of band `band`; 0 when its frame is invalid.
__device__ __forceinline__ float decode_sample(const DevStation &S, const uint8_t *__restrict__ buf,
                                               const uint8_t *__restrict__ valid, int64_t g, int band)
{
	int64_t fr = g / S.framesamples;
	int64_t tin = g - fr * S.framesamples;
	if(!valid[fr])
		return 0.0f;
	const uint8_t *pl = buf + fr * S.framebytes + S.header;
	int64_t q = tin * S.nband + band;
	if(S.nbits == 2)
	{
		int64_t bit = q * 2;
		unsigned int byte = __ldg(pl + (bit >> 3));
		return c_lut2[(byte >> (bit & 7)) & 3];
	}
	return c_lut8[__ldg(pl + q)];
}

// In-place radix-2 decimation-in-time FFT of N = 2^L points held in shared
// memory in bit-reversed order; tw holds exp(-2 pi i k / maxN), k < maxN/2.
__device__ void fft_dit_inplace(float2 *x, int L, const float2 *__restrict__ tw, int twscale)
{
	const int N = 1 << L;
	for(int s = 0; s < L; s++)
	{
		const int half = 1 << s;
		const int tstride = (N >> (s + 1)) * twscale;
		for(int q = threadIdx.x; q < (N >> 1); q += blockDim.x)
		{
			int k = q & (half - 1);
			int i = ((q >> s) << (s + 1)) + k;
			int j = i + half;
			float2 w = __ldg(tw + (int64_t)k * tstride);
			float2 a = x[i], b = x[j];
			float2 t = cmul(b, w);
			x[i] = make_float2(a.x + t.x, a.y + t.y);
			x[j] = make_float2(a.x - t.x, a.y - t.y);
		}
		__syncthreads();
	}
}

// One CTA per (FFT, station): Mode::process for every band of the station
// (mode.cpp:845-1308): decode, time-domain fringe rotation (orders 1, 2),
// complex FFT of 2*nchan points, sideband selection, fractional-sample
// rotation (with the post-F fringe phase for order 0).  Output row-major
// spectra [t][row][nchan] per frequency, FP32.
__global__ void __launch_bounds__(256) k_fstage(const DevStation *__restrict__ st, const DevSubintStation *__restrict__ sub,
                                                const DevBand *__restrict__ bands, int maxband,
                                                const DevFreqPlan *__restrict__ plans, const uint8_t *__restrict__ valid,
                                                int64_t valid_stride, const FftParam *__restrict__ params,
                                                const float2 *__restrict__ twiddle, int maxN, int T, int order,
                                                int fractionallofreq, float2 *__restrict__ spec)
{
	extern __shared__ float2 sx[];
	const int t = blockIdx.x, s = blockIdx.y;
	const DevStation &S = st[s];
	const FftParam p = params[(int64_t)s * T + t];
	const int N = S.fftchannels, nchan = S.nchan;
	const int L = 31 - __clz(N);
	const uint8_t *buf = sub[s].buf;
	const uint8_t *vrow = valid + (int64_t)s * valid_stride;
	const int twscale = maxN / N;

	for(int b = 0; b < S.nband; b++)
	{
		const DevBand bd = bands[s * maxband + b];
		if(bd.row < 0)
			continue;
		const DevFreqPlan &pl = plans[bd.freq];
		float2 *out = spec + pl.spec_off + ((int64_t)t * pl.nrow + bd.row) * nchan;
		if(p.status != kFftOk)
		{
			for(int c = threadIdx.x; c < nchan; c += blockDim.x)
				out[c] = make_float2(0.0f, 0.0f);
			continue;
		}
		// fringe phase of sample n in turns: P0 + ... (FP64 reduction of the
		// constant part, FP32 per sample); mode.cpp:790-1051
		const double lo = bd.lofreq;
		const double fraclo = fractionallofreq ? (lo - (int)lo) * (double)p.integerdelay : 0.0;
		float P0 = 0.0f, alpha = 0.0f, beta = 0.0f, gamma = 0.0f, eps = 0.0f;
		const int asl = S.asl;
		if(order == 1)
		{
			double ph0 = lo * p.b + fraclo;
			P0 = (float)(ph0 - floor(ph0));
			alpha = (float)(lo * p.a / N);
		}
		else if(order == 2)
		{
			double X1 = (double)asl / (double)N;
			double ph0 = lo * p.c + fraclo;
			P0 = (float)(ph0 - floor(ph0));
			alpha = (float)(lo * (p.b + p.a * X1) / N);
			beta = (float)(lo * 2.0 * p.a * X1 / N);
			gamma = (float)(lo * p.b * asl / N);
			eps = (float)(lo * p.a * X1 * X1);
		}
		for(int n = threadIdx.x; n < N; n += blockDim.x)
		{
			float v = 0.0f;
			if(n < p.stuck)
				v = decode_sample(S, buf, vrow, (int64_t)p.nearest + n, b);
			float2 z;
			if(order == 0)
				z = make_float2(v, 0.0f);
			else
			{
				float ph;
				if(order == 1)
					ph = P0 + (float)n * alpha;
				else
				{
					int k = n / asl, j = n - k * asl;
					ph = P0 + (float)j * alpha + (float)(k * j) * beta + (float)k * gamma + (float)(k * k) * eps;
				}
				ph -= floorf(ph);
				float sn, cs;
				sincospif(-2.0f * ph, &sn, &cs);
				z = make_float2(v * cs, v * sn);
			}
			sx[__brev(n) >> (32 - L)] = z;
		}
		__syncthreads();
		fft_dit_inplace(sx, L, twiddle, twscale);
		// fractional-sample correction exp(+2 pi i f_c fse), f_c in MHz
		// (mode.cpp:1053-1097, 1279-1286); post-F fringe phase for order 0
		// (mode.cpp:1061-1070)
		const float dfs = (float)(S.bw / nchan * (double)p.fse);
		float postf = 0.0f;
		if(order == 0)
		{
			double pr = (p.averagedelay - p.integerdelay) * lo;
			if(fractionallofreq)
				pr += p.integerdelay * (lo - (int)lo);
			postf = -(float)(pr - (int)pr);
		}
		for(int c = threadIdx.x; c < nchan; c += blockDim.x)
		{
			float2 x;
			int ce;
			if(bd.lsb)
			{
				ce = c - nchan;
				if(order == 0)
				{
					float2 y = sx[nchan - c];
					x = make_float2(y.x, -y.y);
				}
				else
					x = sx[nchan + c];
			}
			else
			{
				ce = c;
				x = sx[c];
			}
			float turns = (float)ce * dfs + postf;
			float sn, cs;
			sincospif(2.0f * turns, &sn, &cs);
			out[c] = cmul(x, make_float2(cs, sn));
		}
		__syncthreads();
	}
}

cudaError_t launch_fstage(const DevStation *st, const DevSubintStation *sub, const DevBand *bands, int maxband,
                   const DevFreqPlan *plans, const uint8_t *valid, int64_t valid_stride, const FftParam *params,
                   const float2 *twiddle, int maxN, int S, int T, int order, bool fractionallofreq, int maxfft,
                   float2 *spec, cudaStream_t stream)
{
	size_t smem = (size_t)maxfft * sizeof(float2);
	// the shared-memory limit is a per-device attribute: raised on every call
	// (cheap), so that a launch on any device of the process gets it
	const cudaError_t e = cudaFuncSetAttribute(k_fstage, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
	if(e != cudaSuccess)
		return e;
	dim3 grid(T, S);
	k_fstage<<<grid, 256, smem, stream>>>(st, sub, bands, maxband, plans, valid, valid_stride, params, twiddle, maxN, T,
	                                      order, fractionallofreq ? 1 : 0, spec);
	return cudaGetLastError();
}

// Weight sums of one subint: sum_t w1(t) w2(t) of a baseline (core.cpp:
// 998-1045) and sum_t w(t) of a station (mode.cpp:1304-1307; w is zero where
// the FFT is not valid), each the float sum in FFT order that Core forms,
// added to the running total (core.cpp:1068-1086, 1310-1363).  INTERLACEDVDIF
// stations weigh each band by its own data weight (Mode::getDataWeight,
// mode.h:168, mode.cpp:1300-1303).
//
// Bound: latency, of the loads and of a chain of T float additions.  One CTA per
// distinct sum (not per core-result slot: the products of a baseline share one)
// reads 2048 FFTs at a time from the packed weights.  Additions of zeros and ones
// to an integral sum below 2^23 are exact in any order, so a chunk, or a run of
// 32, of such weights (whole or invalid FFTs) is added by its count; other runs are
// added one by one by the first warp.  20 stations x 4 subbands, T = 4096: 87 us
// with a warp per slot, 53 us with a warp per sum, 9 us now; 5 stations, T =
// 38622: 740, 331, 58 us.
__global__ void __launch_bounds__(256) k_weights(const DevWeightSum *__restrict__ sums, const float *__restrict__ wts,
                                                 const float *__restrict__ pbw, int nbm, int T,
                                                 float *__restrict__ acc)
{
	constexpr int G = 8, kChunk = 256 * G;        // values per thread and chunk
	__shared__ __align__(16) float buf[kChunk];
	__shared__ int ones_s[kChunk / 32], clean_s[kChunk / 32], count_s[2][8];
	__shared__ float sum_s;
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const DevWeightSum u = sums[blockIdx.x];
	const float *wa = u.b1 >= 0 ? pbw + (int64_t)u.s1 * T * nbm + u.b1 : wts + (int64_t)u.s1 * T;
	const int sa = u.b1 >= 0 ? nbm : 1;
	const bool two = u.s2 >= 0;
	const float *wb = !two ? wa : (u.b2 >= 0 ? pbw + (int64_t)u.s2 * T * nbm + u.b2 : wts + (int64_t)u.s2 * T);
	const int sb = two && u.b2 >= 0 ? nbm : 1;
	float sum = 0.0f;                             // the same in every thread
	int par = 0;
	for(int t0 = 0; t0 < T; t0 += kChunk, par ^= 1)
	{
		float v[G];
#pragma unroll
		for(int g = 0; g < G; g++)
		{
			const int t = t0 + 256 * g + (int)threadIdx.x;
			v[g] = t < T ? __ldg(wa + (int64_t)t * sa) : 0.0f;
			if(two)
				v[g] = __fmul_rn(v[g], t < T ? __ldg(wb + (int64_t)t * sb) : 0.0f);
		}
		int count = 0;
		bool clean = true;
#pragma unroll
		for(int g = 0; g < G; g++)
		{
			count += __popc(__ballot_sync(0xffffffffu, v[g] == 1.0f));
			clean = clean && (v[g] == 1.0f || v[g] == 0.0f);
		}
		if(lane == 0)
			count_s[par][warp] = count;
		if(__syncthreads_and(clean) && sum == rintf(sum) && sum < 8388608.0f)
		{
			int n = 0;
#pragma unroll
			for(int w = 0; w < 8; w++)
				n += count_s[par][w];
			sum += (float)n;
			continue;
		}
		// run r of the chunk: FFTs t0 + 32 r .. + 31, held by warp r % 8
#pragma unroll
		for(int g = 0; g < G; g++)
		{
			const uint32_t ones = __ballot_sync(0xffffffffu, v[g] == 1.0f);
			const bool all = __all_sync(0xffffffffu, v[g] == 1.0f || v[g] == 0.0f);
			if(lane == 0)
			{
				ones_s[8 * g + warp] = __popc(ones);
				clean_s[8 * g + warp] = all;
			}
			buf[256 * g + threadIdx.x] = v[g];
		}
		__syncthreads();
		if(warp == 0)
		{
			const int nrun = min(kChunk, T - t0 + 31) / 32;
			for(int r = 0; r < nrun; r++)
			{
				if(clean_s[r] && sum == rintf(sum) && sum < 8388608.0f)
				{
					sum += (float)ones_s[r];
					continue;
				}
				// adding 0 (past T, or an invalid FFT) leaves a non-negative sum unchanged
#pragma unroll
				for(int j = 0; j < 32; j += 4)
				{
					const float4 q = *(const float4 *)(buf + 32 * r + j);
					sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, q.x), q.y), q.z), q.w);
				}
			}
			if(lane == 0)
				sum_s = sum;
		}
		__syncthreads();
		sum = sum_s;
	}
	if(threadIdx.x == 0)
		acc[blockIdx.x] = __fadd_rn(acc[blockIdx.x], sum);
}

void launch_weights(const DevWeightSum *sums, int nsum, const float *wts, const float *pbw, int nbm, int T, float *acc,
                    cudaStream_t stream)
{
	if(nsum > 0)
		k_weights<<<nsum, 256, 0, stream>>>(sums, wts, pbw, nbm, T, acc);
}

// Core-result assembly (core.cpp:1774-1802 channel averaging, 1266-1363):
// accumulators -> [freq][baseline][product][nchan/avg], autocorrelations,
// and the float weight slots.
__global__ void k_finalise(const DevOutMap *__restrict__ om, const float2 *__restrict__ acc, float2 *__restrict__ core)
{
	const DevOutMap m = om[blockIdx.x];
	const int nout = m.nchan / m.avg;
	for(int co = threadIdx.x; co < nout; co += blockDim.x)
	{
		float2 v = make_float2(0.0f, 0.0f);
		if(m.acc >= 0)
		{
			if(m.avg == 1)
				v = acc[m.acc + (int64_t)co * m.cstride];
			else
			{
				float sr = 0.0f, si = 0.0f;
				for(int k = 0; k < m.avg; k++)
				{
					float2 a = acc[m.acc + ((int64_t)co * m.avg + k) * m.cstride];
					sr += a.x;
					si += a.y;
				}
				v = make_float2(sr / m.avg, si / m.avg);
			}
		}
		core[m.core + co] = v;
	}
}

__global__ void k_finalise_weights(const DevWeightOut *__restrict__ wout, int n, const float *__restrict__ wacc,
                                   float *__restrict__ corefloat)
{
	const int k = blockIdx.x * blockDim.x + threadIdx.x;
	if(k < n)
		corefloat[wout[k].dst] = wacc[wout[k].sum];
}

void launch_finalise(const DevOutMap *om, int nom, const float2 *acc, const DevWeightOut *wout, int nwout,
                     const float *wacc, float2 *core, int64_t corelen, cudaStream_t stream)
{
	cudaMemsetAsync(core, 0, sizeof(float2) * corelen, stream);
	if(nom > 0)
		k_finalise<<<nom, 256, 0, stream>>>(om, acc, core);
	if(nwout > 0)
		k_finalise_weights<<<(nwout + 127) / 128, 128, 0, stream>>>(wout, nwout, wacc, (float *)core);
}

// Stand-alone decode with mark5_unpack_with_offset's contract
// (mark5_stream_unpacker.c:129-147): one CTA; frame validity first, then the
// good-sample count (with the 8-bit 2/4-channel blank semantics), then the
// samples.
__global__ void k_vdif_unpack(const uint8_t *__restrict__ data, int64_t nbytes, int payload, int header, int nchan,
                              int nbits, int64_t offsetsamples, int nsamp, float *__restrict__ out, int *good)
{
	extern __shared__ uint8_t fvalid[];
	__shared__ int firstblank;
	__shared__ int goodcount;
	const int64_t framebytes = payload + header;
	const int64_t fs = (int64_t)payload * 8 / (nchan * nbits);
	const int64_t f0 = offsetsamples / fs, f1 = (offsetsamples + nsamp - 1) / fs;
	const int nf = (int)(f1 - f0 + 1);
	const uint64_t FILL = 0x1122334411223344ULL;
	for(int k = threadIdx.x; k < nf; k += blockDim.x)
	{
		int64_t fr = f0 + k;
		uint8_t v = 0;
		if((fr + 1) * framebytes <= nbytes)
		{
			const uint8_t *f = data + fr * framebytes;
			uint32_t w0 = *(const uint32_t *)f, w2 = *(const uint32_t *)(f + 8);
			uint64_t first = *(const uint64_t *)(f + header);
			uint64_t last = *(const uint64_t *)(f + header + (payload / 8 - 1) * 8);
			v = (w2 != 0) && !((w0 >> 31) & 1) && first != FILL && last != FILL;
		}
		fvalid[k] = v;
	}
	__syncthreads();
	const bool sticky = nbits == 8 && (nchan == 2 || nchan == 4);
	if(threadIdx.x == 0)
	{
		int fb = nsamp, cnt = 0;
		for(int k = 0; k < nf; k++)
		{
			int64_t a = (f0 + k) * fs - offsetsamples, b = a + fs;
			if(a < 0) a = 0;
			if(b > nsamp) b = nsamp;
			if(!fvalid[k])
			{
				if(sticky && fb == nsamp) fb = (int)a;
				continue;
			}
			if(sticky && fb < nsamp) continue;
			cnt += (int)(b - a);
		}
		firstblank = sticky ? fb : nsamp;
		goodcount = cnt;
	}
	__syncthreads();
	for(int o = threadIdx.x; o < nsamp; o += blockDim.x)
	{
		int64_t g = offsetsamples + o;
		int64_t fr = g / fs, tin = g - fr * fs;
		bool v = fvalid[fr - f0] && o < firstblank;
		const uint8_t *pl = data + fr * framebytes + header;
		for(int c = 0; c < nchan; c++)
		{
			float val = 0.0f;
			if(v)
			{
				int64_t q = tin * nchan + c;
				if(nbits == 2)
				{
					int64_t bit = q * 2;
					val = c_lut2[(pl[bit >> 3] >> (bit & 7)) & 3];
				}
				else
					val = c_lut8[pl[q]];
			}
			out[(int64_t)c * nsamp + o] = val;
		}
	}
	if(threadIdx.x == 0)
		*good = goodcount;
}

void launch_vdif_unpack(const uint8_t *data, int64_t nbytes, int payload, int header, int nchan, int nbits,
                        int64_t offsetsamples, int nsamp, float *out, int *good, cudaStream_t stream)
{
	const int64_t fs = (int64_t)payload * 8 / (nchan * nbits);
	const int nf = (int)((offsetsamples + nsamp - 1) / fs - offsetsamples / fs + 1);
	k_vdif_unpack<<<1, 256, nf, stream>>>(data, nbytes, payload, header, nchan, nbits, offsetsamples, nsamp, out, good);
}

// ---------------------------------------------------------------- zoom bands
// A zoom band's spectra are the channels [choff, choff + nchan) of its parent
// band's (mode.cpp:169-208), copied into the zoom frequency's own rows.
constexpr int kZoomTimes = 8;

// FP32 form [t][row][chan]: one CTA per (8 FFTs, zoom row), a thread a channel of
// all eight.
__global__ void __launch_bounds__(256) k_zoom_gather(const DevZoomCopy *__restrict__ zc,
                                                     const DevFreqPlan *__restrict__ plans, int T,
                                                     float2 *__restrict__ spec)
{
	const DevZoomCopy z = zc[blockIdx.y];
	const DevFreqPlan &src = plans[z.src_plan], &dst = plans[z.dst_plan];
	const int t0 = blockIdx.x * kZoomTimes;
	const int64_t sts = (int64_t)src.nrow * src.nchan, dts = (int64_t)dst.nrow * dst.nchan;
	const float2 *s0 = spec + src.spec_off + t0 * sts + (int64_t)z.src_row * src.nchan + z.choff;
	float2 *d0 = spec + dst.spec_off + t0 * dts + (int64_t)z.dst_row * dst.nchan;
	for(int c = threadIdx.x; c < z.nchan; c += blockDim.x)
	{
		float2 v[kZoomTimes];
#pragma unroll
		for(int k = 0; k < kZoomTimes; k++)
			if(t0 + k < T)
				v[k] = s0[k * sts + c];
#pragma unroll
		for(int k = 0; k < kZoomTimes; k++)
			if(t0 + k < T)
				d0[k * dts + c] = v[k];
	}
}

// Tensor-core forms [t][block][trow][tcb], channels in the order of chan_pos: CTAs per
// (8 FFTs, zoom frequency, share of its quads), a thread the four channels of a quad
// of positions of one row, the lanes of a warp in neighbouring rows, whose quads lie
// side by side.
// Bound by L2: the quads of the parent hold one or two wanted channels of four.  A
// CTA a row and 4-byte loads and stores met a sector a value: two windows of 256
// channels on each of 8 subbands, 20 rows x 250 FFTs, F stage and gather 327 us, 185
// now (244 before the channels' present order).
__global__ void __launch_bounds__(256) k_zoom_quads(const DevZoomCopy *__restrict__ zc,
                                                    const DevZoomGroup *__restrict__ groups,
                                                    const DevFreqPlan *__restrict__ plans, int T,
                                                    uint32_t *__restrict__ spec)
{
	const DevZoomGroup g = groups[blockIdx.y];
	const int t0 = blockIdx.x * kZoomTimes, nq = zc[g.first].nchan >> 2, n = g.count * nq;
	for(int w = blockIdx.z * blockDim.x + threadIdx.x; w < n; w += gridDim.z * blockDim.x)
	{
		const int i = w / g.count;
		const DevZoomCopy z = zc[g.first + (w - i * g.count)];
		const DevFreqPlan &S = plans[z.src_plan], &D = plans[z.dst_plan];
		const int64_t sts = (int64_t)S.tnblk * S.trow * S.tcb, dts = (int64_t)D.tnblk * D.trow * D.tcb;
		const uint32_t *s = spec + S.spec_off + t0 * sts + (int64_t)z.src_row * S.tcb;
		uint32_t *d = spec + D.spec_off + t0 * dts + (int64_t)z.dst_row * D.tcb;
		const uint32_t sextra = (uint32_t)(S.trow - 1) * (uint32_t)S.tcb, dextra = (uint32_t)(D.trow - 1) * (uint32_t)D.tcb;
		uint32_t off[4];
#pragma unroll
		for(int m = 0; m < 4; m++)
		{
			const uint32_t q = (uint32_t)chan_pos(S.pbits, z.choff + i + m * nq);
			off[m] = q + __umulhi(q, S.magic) * sextra;
		}
		const uint32_t dtcb = (uint32_t)D.tcb, dmagic = D.magic;
		uint4 v[kZoomTimes];
#pragma unroll
		for(int k = 0; k < kZoomTimes; k++)
			if(t0 + k < T)
				v[k] = make_uint4(s[k * sts + off[0]], s[k * sts + off[1]], s[k * sts + off[2]], s[k * sts + off[3]]);
#pragma unroll
		for(int k = 0; k < kZoomTimes; k++)
			if(t0 + k < T)
				store_quad(d + k * dts, 4u * (uint32_t)i, dtcb, dmagic, dextra, v[k]);
	}
}

void launch_zoom_gather(const DevZoomCopy *zc, int nzc, const DevZoomGroup *groups, int ngroups, int maxquads,
                        const DevFreqPlan *plans, int T, bool tc, void *spec, cudaStream_t stream)
{
	if(nzc <= 0 || T <= 0)
		return;
	const int nt = (T + kZoomTimes - 1) / kZoomTimes;
	// few FFTs and frequencies: the quads of a frequency over more CTAs
	const int share = std::max(1, std::min((maxquads + 255) / 256, 1184 / (nt * std::max(ngroups, 1))));
	if(tc)
		k_zoom_quads<<<dim3(nt, ngroups, share), 256, 0, stream>>>(zc, groups, plans, T, (uint32_t *)spec);
	else
		k_zoom_gather<<<dim3(nt, nzc), 256, 0, stream>>>(zc, plans, T, (float2 *)spec);
}

// 8-bit levels (b - 128) / 3.3 (format_vdif.c:122) into the current
// device's constant table; pageable source, so the copy has been taken when
// this returns
cudaError_t upload_lut8(cudaStream_t stream)
{
	float lut[256];
	for(int b = 0; b < 256; b++)
		lut[b] = (float)((b - 128) / 3.3);
	return cudaMemcpyToSymbolAsync(c_lut8, lut, sizeof(lut), 0, cudaMemcpyHostToDevice, stream);
}

}  // namespace fxb
