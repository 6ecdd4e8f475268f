// FP32 cross-multiply-accumulate (Core::processdata, mpifxcorr/src/core.cpp:
// 877-972, with the autocorrelations of mode.cpp:1293-1369) for sm_100a.
//
// For one subband V[i][j] = sum_t X_i(t) X_j(t)^* over all input rows i, j is a
// complex Hermitian rank-T update per channel.  A CTA owns 32 channels of one
// subband, a share of the R x R tile pairs (ti <= tj) of its rows and a slice
// of the subint's times: one warp per tile pair, one channel per lane, so
// that each spectrum value is read from HBM once and reused by every tile pair
// in shared memory, through a ring of cp.async stages.
//
// Bound: the FP32 pipe and the shared-memory reads, R R complex products (4
// R R FFMA) per 2 R eight-byte loads of a warp; the registers (2 R R sums)
// decide how many warps hide each other's latencies.  20 rows x 1024 channels
// x 8 subbands x 250 times: R = 5 in 96 registers (20 warps per SM) 144 us,
// R = 4 in 64 (30 warps) 159 us, R = 5 in 80 161 us, R = 5 in 128 (10 warps)
// 210 us; the FFMAs alone take 53 us.  Packed FFMA2 (fma.rn.f32x2) runs at half
// the rate of FFMA and needs twice the sums: 160 us.  60 rows x 2048 x 2 x 26:
// R = 4 108 us, R = 5 148 us, so R = 5 is used where its tile pairs fit ten
// warps (20 rows); xmac_plan takes the R with the least work.
//
// Slices: 32 channels x the subbands of a group often make fewer CTAs than
// the chip holds (4 stations, one subband of 256 channels: 8 CTAs on 148 SMs).
// The times are then split over the CTAs of a cluster, and within a CTA over
// groups of warps where the rows give only a few tile pairs.  The partial
// sums meet in shared memory and over distributed shared memory in slice
// order, so a result depends on the job and the device's number of SMs (which
// chooses the slices), never on the schedule.
// Measured: 4 stations, 256 channels, T = 250: 142 -> 12 us; 7 rows x 64
// channels x 16 subbands, T = 2005: 552 -> 60 us; 10 stations x 8 x 1024
// channels, T = 250: 198 -> 144 us.

#include <cuda_runtime.h>
#include <cooperative_groups.h>
#include <cstdint>

#include "fxb_internal.h"
#include "fxb_kernels.h"

namespace fxb {

namespace {

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem)
{
	unsigned s = (unsigned)__cvta_generic_to_shared(smem);
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait()
{
	asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

constexpr int kCB = 32;        // channels per CTA
constexpr int kStages = 3;     // ring of time stages
constexpr int kMaxWarps = 16;
constexpr int kMaxWarps5 = 10;
constexpr int kMaxCluster = 8;

// tile pair p of nt row tiles, pairs (0,0) (0,1) .. (0,nt-1) (1,1) ..
__device__ __forceinline__ void pair_of(int p, int nt, int &ti, int &tj)
{
	ti = 0;
	while(p >= nt - ti)
	{
		p -= nt - ti;
		ti++;
	}
	tj = ti + p;
}

struct XPlan {
	int R, ntile, npair;       // rows per tile, tiles, tile pairs
	int npl, nz;               // tile pairs per CTA, CTAs sharing a subband's pairs
	int tsub, cluster;         // time slices within a CTA, over the CTAs of a cluster
	int TC;                    // times per stage
	size_t smem;
};

}  // namespace

// R = 5: 96 registers, at most kMaxWarps5 warps per CTA (two CTAs per SM)
template <int R>
__global__ void __launch_bounds__(R == 5 ? 32 * kMaxWarps5 : 32 * kMaxWarps, 2)
    k_xmac_fp32(const DevFreqPlan *__restrict__ plans, const int32_t *__restrict__ plan_idx, int T, XPlan xp,
                const float2 *__restrict__ spec, float2 *__restrict__ acc)
{
	extern __shared__ __align__(16) float2 sx[];
	const DevFreqPlan &P = plans[plan_idx[blockIdx.y]];
	const int cs = xp.cluster;
	const int rank = cs > 1 ? (int)(blockIdx.x % (unsigned)cs) : 0;
	const int c0 = (int)(blockIdx.x / (unsigned)cs) * kCB;
	const int nrow = P.nrow, nchan = P.nchan, TC = xp.TC;
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const int sub = warp / xp.npl, pl = warp - sub * xp.npl;
	const int pairidx = blockIdx.z * xp.npl + pl;
	const bool active = pairidx < xp.npair;
	int ti = 0, tj = 0;
	if(active)
		pair_of(pairidx, xp.ntile, ti, tj);
	const int stage = TC * nrow * kCB;
	const int t0 = (int)((int64_t)T * rank / cs), t1 = (int)((int64_t)T * (rank + 1) / cs);
	const int nv = min(kCB, nchan - c0) >> 1;               // 16-byte pieces of a row (channel counts are even)

	// A stage is [time][row][32 channels] without padding: rows past nrow (of
	// the last tile) and channels past nchan are whatever lies there, and only
	// products that are never written depend on them.  A thread copies the
	// same 16 bytes of every (blockDim / 16)th row.
	const int ch2 = threadIdx.x & (kCB / 2 - 1), tr0 = threadIdx.x / (kCB / 2), trs = blockDim.x / (kCB / 2);
	const float2 *X = spec + P.spec_off + c0 + 2 * ch2 + ((int64_t)t0 * nrow + tr0) * nchan;
	const int64_t xstep = (int64_t)trs * nchan;
	auto load_stage = [&](int buf, int tb) {
		if(ch2 >= nv)
			return;
		const int ntr = min(TC, t1 - tb) * nrow;
		float2 *dst = sx + buf * stage + tr0 * kCB + 2 * ch2;
		const float2 *src = X + (int64_t)(tb - t0) * nrow * nchan;
		for(int tr = tr0; tr < ntr; tr += trs, dst += trs * kCB, src += xstep)
			cp_async16(dst, src);
	};

	float vr[R][R], vi[R][R];
#pragma unroll
	for(int i = 0; i < R; i++)
#pragma unroll
		for(int j = 0; j < R; j++)
		{
			vr[i][j] = 0.0f;
			vi[i][j] = 0.0f;
		}

#pragma unroll
	for(int s = 0; s < kStages - 1; s++)
	{
		if(t0 + s * TC < t1)
			load_stage(s, t0 + s * TC);
		cp_async_commit();
	}
	int buf = 0;
	for(int tb = t0; tb < t1; tb += TC)
	{
		cp_async_wait<kStages - 2>();
		__syncthreads();                    // this stage has arrived, the one before it has been read by every warp
		const int nx = tb + (kStages - 1) * TC;
		if(nx < t1)
			load_stage(buf == 0 ? kStages - 1 : buf - 1, nx);
		cp_async_commit();
		if(active)
		{
			const int tcnt = min(TC, t1 - tb);
			const float2 *pa = sx + buf * stage + ti * R * kCB + lane, *pb = sx + buf * stage + tj * R * kCB + lane;
			for(int tt = sub; tt < tcnt; tt += xp.tsub)
			{
				const float2 *ra = pa + tt * nrow * kCB, *rb = pb + tt * nrow * kCB;
				float2 a[R], b[R];
#pragma unroll
				for(int i = 0; i < R; i++)
				{
					a[i] = ra[i * kCB];
					b[i] = rb[i * kCB];
				}
#pragma unroll
				for(int i = 0; i < R; i++)
#pragma unroll
					for(int j = 0; j < R; j++)
					{
						vr[i][j] = fmaf(a[i].x, b[j].x, fmaf(a[i].y, b[j].y, vr[i][j]));
						vi[i][j] = fmaf(a[i].y, b[j].x, fmaf(-a[i].x, b[j].y, vi[i][j]));
					}
			}
		}
		buf = buf + 1 == kStages ? 0 : buf + 1;
	}
	const int c = c0 + lane;
	// adds one value of this channel to its outputs
	auto emit = [&](int ri, int rj, float2 v) {
		if(ri >= nrow || rj >= nrow || ri > rj || c >= nchan)
			return;
		const int dA = P.destA[ri * nrow + rj], dB = P.destB[ri * nrow + rj];
		if(dA >= 0)
		{
			float2 *d = acc + P.acc_off + (int64_t)dA * P.acc_ostride + (int64_t)c * P.acc_cstride;
			const float2 o = *d;
			*d = make_float2(o.x + v.x, o.y + v.y);
		}
		if(dB >= 0)
		{
			float2 *d = acc + P.acc_off + (int64_t)dB * P.acc_ostride + (int64_t)c * P.acc_cstride;
			const float2 o = *d;
			*d = make_float2(o.x + v.x, o.y - v.y);
		}
	};
	if(xp.tsub * cs == 1)
	{
		if(active)
		{
#pragma unroll
			for(int i = 0; i < R; i++)
#pragma unroll
				for(int j = 0; j < R; j++)
					emit(ti * R + i, tj * R + j, make_float2(vr[i][j], vi[i][j]));
		}
		return;
	}
	// slices of the CTA in turn into part[pair][i][j][lane] (over the stages,
	// which every warp has finished reading), then each CTA of the cluster
	// sums its share of the values over the slices of all of them
	float2 *part = sx;
	for(int s = 0; s < xp.tsub; s++)
	{
		__syncthreads();
		if(s == sub && active)
		{
#pragma unroll
			for(int i = 0; i < R; i++)
#pragma unroll
				for(int j = 0; j < R; j++)
				{
					float2 *q = part + ((pl * R + i) * R + j) * 32 + lane;
					float2 v = make_float2(vr[i][j], vi[i][j]);
					if(s > 0)
					{
						const float2 o = *q;
						v = make_float2(o.x + v.x, o.y + v.y);
					}
					*q = v;
				}
		}
	}
	namespace cg = cooperative_groups;
	cg::cluster_group cl = cg::this_cluster();
	cl.sync();
	const int nval = min(xp.npl, xp.npair - (int)blockIdx.z * xp.npl) * R * R;
	for(int e = warp * cs + rank; e < nval; e += (blockDim.x >> 5) * cs)
	{
		float2 v = make_float2(0.0f, 0.0f);
		for(int q = 0; q < cs; q++)
		{
			const float2 o = *cl.map_shared_rank(part + e * 32 + lane, q);
			v = make_float2(v.x + o.x, v.y + o.y);
		}
		const int p = e / (R * R), ij = e - p * R * R;
		int ei, ej;
		pair_of(blockIdx.z * xp.npl + p, xp.ntile, ei, ej);
		emit(ei * R + ij / R, ej * R + ij % R, v);
	}
	cl.sync();                              // no CTA leaves while others read its sums
}

// Rows per tile, tile pairs per CTA and time slices of a group.
static XPlan xmac_plan(int nrow, int nchan, int nf, int T, int nsm)
{
	XPlan xp;
	int64_t best = -1;
	xp.R = 4;
	for(int R = 3; R <= 5; R++)
	{
		// FFMAs, and a third of the loads (they run beside the FFMAs)
		const int nt = (nrow + R - 1) / R, np = nt * (nt + 1) / 2;
		if(R == 5 && np > kMaxWarps5)
			continue;
		const int64_t cost = (int64_t)np * (3 * R * R + 4 * R);
		if(best < 0 || cost < best)
		{
			best = cost;
			xp.R = R;
		}
	}
	const int R = xp.R;
	xp.ntile = (nrow + R - 1) / R;
	xp.npair = xp.ntile * (xp.ntile + 1) / 2;
	xp.nz = (xp.npair + kMaxWarps - 1) / kMaxWarps;
	xp.npl = (xp.npair + xp.nz - 1) / xp.nz;
	// few tile pairs: up to 12 (10) warps take the times in turn
	const int want = R == 5 ? kMaxWarps5 : 12;
	xp.tsub = want / xp.npl > 1 ? want / xp.npl : 1;
	if(xp.tsub > T)
		xp.tsub = T;
	// CTAs of a cluster: rounds of CTAs over the SMs x times per CTA, each
	// round with the merge of its slices at the cost of about kMerge times (20
	// rows, T = 250: slices over two CTAs of a cluster cost 13 us on 147)
	constexpr int kMerge = 12;
	const int64_t units = (int64_t)((nchan + kCB - 1) / kCB) * nf * xp.nz;
	xp.cluster = 1;
	int64_t least = -1;
	for(int cs = 1; cs <= kMaxCluster; cs *= 2)
	{
		const int64_t times = (T + cs * xp.tsub - 1) / (cs * xp.tsub);
		if(cs > 1 && times < 4)
			break;
		const int64_t cost = (units * cs + nsm - 1) / nsm * (times + (cs > 1 || xp.tsub > 1 ? kMerge : 2));
		if(least < 0 || cost < least)
		{
			least = cost;
			xp.cluster = cs;
		}
	}
	const int trow = nrow * kCB * (int)sizeof(float2);
	xp.TC = (96 * 1024) / (kStages * trow);
	const int cap = 4 * xp.tsub > 16 ? 4 * xp.tsub : 16;
	xp.TC = xp.TC > cap ? cap : (xp.TC < 1 ? 1 : xp.TC);
	// the last tile's rows past nrow are read past the last stage
	xp.smem = (size_t)kStages * xp.TC * trow + (size_t)(xp.ntile * R - nrow) * kCB * sizeof(float2);
	const size_t part = (size_t)xp.npl * R * R * 32 * sizeof(float2);
	if(xp.tsub * xp.cluster > 1 && part > xp.smem)
		xp.smem = part;
	return xp;
}

void launch_xmac_fp32(const DevFreqPlan &plan0, const DevFreqPlan *dplans, const int32_t *plan_idx, int nf, int T,
                      int nsm, const float2 *spec, float2 *acc, cudaStream_t stream)
{
	const XPlan xp = xmac_plan(plan0.nrow, plan0.nchan, nf, T, nsm);
	auto go = [&](auto kern) {
		cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024);
		cudaLaunchConfig_t cfg = {};
		cfg.gridDim = dim3((plan0.nchan + kCB - 1) / kCB * xp.cluster, nf, xp.nz);
		cfg.blockDim = dim3(32 * xp.npl * xp.tsub);
		cfg.dynamicSmemBytes = xp.smem;
		cfg.stream = stream;
		cudaLaunchAttribute at;
		at.id = cudaLaunchAttributeClusterDimension;
		at.val.clusterDim.x = xp.cluster;
		at.val.clusterDim.y = 1;
		at.val.clusterDim.z = 1;
		cfg.attrs = &at;
		cfg.numAttrs = 1;
		cudaLaunchKernelEx(&cfg, kern, dplans, plan_idx, T, xp, spec, acc);
	};
	if(xp.R == 3)
		go(k_xmac_fp32<3>);
	else if(xp.R == 4)
		go(k_xmac_fp32<4>);
	else
		go(k_xmac_fp32<5>);
}

}  // namespace fxb
