// FP16 / BF16 form of the tensor-core cross-multiply-accumulate for sm_100a
// (tcgen05 + TMA).
//
// Core::processdata's XMAC (mpifxcorr/src/core.cpp:877-972) and the Mode
// autocorrelations (mode.cpp:1293-1369) per channel are V = X X^H, with X the
// [inputs x time] matrix of one channel's spectra.  With X written as real rows
// (2 per input: real and imaginary part, interleaved), A A^T holds every
// product: for inputs a, b
//     Re V[a][b] = P[2a][2b] + P[2a+1][2b+1],  Im V[a][b] = P[2a+1][2b] - P[2a][2b+1].
//
// Input: the F stage's half2 (or bf16x2) spectra X 2^-kTcSpecExp, per group of
// equally shaped subbands one block [subband][Tpad][block][trow][CB] (times T ..
// Tpad-1 and rows nrow .. trow-1 zero).  The Wh = 2 trow CB real values of a
// block at one time are one contiguous run, which is an MN-major operand row as
// it stands: TMA puts the run's 64-byte pieces where tcgen05 wants them (atoms
// of 8 times x 32 values, 64-byte swizzle), and the same shared memory serves as
// A and as B.  Nothing is transposed or copied by threads.  The price is
// that a block's CB channels meet in one product, of which only the terms of
// equal channels are used (1 / CB); with CB = 8, 4 or 2 for up to 12, 24 and 64
// inputs the matrix work is that of packing G diagonal blocks into 128 rows.
// A unit is one block over one slice of the subint's times: rows 0 - 127 against
// all Wh columns, and rows 128 - Wh-1 against columns 128 - Wh-1 (the rest is
// the mirror image).  The epilogue scales every product by 2^(2 kTcSpecExp),
// which undoes the spectra's scale exactly.
//
// Persistent CTAs (two per SM where the accumulators fit 256 tensor-memory
// columns), warp-specialised:
//   warp 0     TMA producer: boxes of 32 times into a ring of stages,
//   warp 1     tensor-memory owner and MMA issuer,
//   warps 2-9  epilogue: two warps per tensor-memory quadrant.  A lane holds the
//              real or imaginary row of one input and channel; it picks its
//              channel's columns of two inputs, trades with its neighbour so
//              that each of the two lanes holds one complex output, and adds it
//              to the [channel][output] accumulators (vector reduction).
// Few units (few channels, many FFTs): a unit's times are cut into slices, whose
// sums go to a workspace and are added in slice order by k_xmac_merge, so that a
// result never depends on the schedule.  Slices are chosen from the group's own
// extents and the device's number of SMs, so a context alone and in a batch agree.
//
// Bound: HBM / L2 reads of the spectra at up to about 20 inputs, the epilogue's
// reductions and the matrix work above.  Launch times in us with K-major operands
// made by transposer warps, and now: 20 inputs x 8 x 1024 channels x 250 FFTs 69 and
// 47 (the loads alone take 31); 40 x 4 x 128 x 4096 180 and 79; 10 x 2 x 64 x 38622
// 1720 and 81 (time slices); 64 x 4 x 1024 x 250 125 and 134 (two reads).
// Every wait is bounded: on timeout the CTA records an error code, drains its
// TMA loads and MMAs, and still releases its tensor memory.

#include <cuda_runtime.h>
#include <cstdint>
#include <cstring>

#include "fxb_xmac_tc.cuh"

namespace fxb {

namespace {

constexpr int kKT = 32;                    // times per stage (two MMA steps of 16)
constexpr int kMaxStages = 12;
constexpr int kThreads = 320;
constexpr int kChunk = kKT * 64;           // 32 values (64 bytes) x 32 times
constexpr int kMaxSlice = 16;

__device__ __forceinline__ void tma_load_4d(void *dst, const CUtensorMap *map, int x, int y, int z, int w, uint64_t *bar)
{
	asm volatile(
	    "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
	    "[%6];\n" ::"r"(smem_u32(dst)),
	    "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(smem_u32(bar))
	    : "memory");
}

// shared-memory matrix descriptor: MN-major, 64-byte swizzle.  Atoms of 8 times
// x 32 values (512 bytes); the next 32 values kChunk bytes on (leading byte
// offset), the next 8 times 512 bytes on (stride byte offset)
__device__ __forceinline__ uint64_t desc_mn64(uint32_t saddr)
{
	uint64_t d = 0;
	d |= (uint64_t)((saddr >> 4) & 0x3FFF);
	d |= (uint64_t)(kChunk >> 4) << 16;
	d |= (uint64_t)(512 >> 4) << 32;
	d |= (uint64_t)1 << 46;                // descriptor version
	d |= (uint64_t)4 << 61;                // SWIZZLE_64B
	return d;
}

__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate)
{
	asm volatile(
	    "{\n\t.reg .pred p;\n\t"
	    "setp.ne.b32 p, %4, 0;\n\t"
	    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(tmem_d),
	    "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
}

template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, float *v)
{
	uint32_t r[N];
	if constexpr(N == 8)
		asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
		             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
		             : "r"(taddr));
	else if constexpr(N == 16)
		asm volatile(
		    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
		    "%15}, [%16];\n"
		    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
		      "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
		    : "r"(taddr));
	else
		asm volatile(
		    "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
		    "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
		    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
		      "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
		      "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
		      "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
		    : "r"(taddr));
#pragma unroll
	for(int i = 0; i < N; i++)
		v[i] = __uint_as_float(r[i]);
}

// element i (a power of two of them, stride 2) of v by a lane-dependent index
template <int CB>
__device__ __forceinline__ float pick(const float *v, int i)
{
	if constexpr(CB == 1)
		return v[0];
	else
	{
		const float lo = pick<CB / 2>(v, i & (CB / 2 - 1)), hi = pick<CB / 2>(v + CB, i & (CB / 2 - 1));
		return (i & (CB / 2)) ? hi : lo;
	}
}

}  // namespace

// the launch's common shape (every group has the same rows); the groups' own
// extents are in XMultiArgs
struct XhParams {
	int32_t nrow, nch;              // inputs; 64-byte pieces of a block's run
	int32_t stage_bytes, nst;       // one stage; stages in use
	int32_t nbuf, cols, tcols;      // accumulator buffers, columns of one, columns allocated
	int32_t h16;                    // FP16 operands (else BF16)
	int32_t *err;
};

// Work units of every group of the launch in turn, CTAs striding over them.
template <int CB>
__global__ void __launch_bounds__(kThreads, 2) k_xmac_h(const __grid_constant__ XMultiArgs xm, XhParams tp)
{
	extern __shared__ __align__(1024) unsigned char smem_h[];
	__shared__ uint64_t full[kMaxStages], empty[kMaxStages], acc_full[2], acc_empty[2], mma_done;
	__shared__ uint32_t tmem_base_s;
	__shared__ volatile int fail_s;
	__shared__ int issued_s, consumed_s;

	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	unsigned char *ring = (unsigned char *)(((uintptr_t)smem_h + 1023) & ~(uintptr_t)1023);
	const int nst = tp.nst, nbuf = tp.nbuf;
	if(threadIdx.x == 0)
	{
		for(int s = 0; s < nst; s++)
		{
			mbar_init(&full[s], 1);
			mbar_init(&empty[s], 1);
		}
		for(int b = 0; b < 2; b++)
		{
			mbar_init(&acc_full[b], 1);
			mbar_init(&acc_empty[b], 8);
		}
		mbar_init(&mma_done, 1);
		fail_s = 0;
		issued_s = 0;
		consumed_s = 0;
		asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
	}
	if(warp == 1)
	{
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_base_s)),
		             "r"((uint32_t)tp.tcols));
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
	}
	asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
	__syncthreads();
	asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
	const uint32_t tmem = tmem_base_s;
	const int Wh = 32 * tp.nch;

	if(warp == 0)
	{
		if(lane == 0)
		{
			// ---- TMA producer
			int kk = 0;
			bool ok = true;
			for(int u = blockIdx.x; u < xm.nunits && ok; u += gridDim.x)
			{
				const UnitLoc L = locate(xm, u);
				const XGroupRec &G = xm.g[L.gi];
				const CUtensorMap *map = (const CUtensorMap *)&xm.map[L.gi];
				const int k0 = G.nkt * L.slice / G.nslice, k1 = G.nkt * (L.slice + 1) / G.nslice;
				for(int kt = k0; kt < k1; kt++, kk++)
				{
					const int s = kk % nst;
					if(kk >= nst && !mbar_wait(&empty[s], ((kk / nst) - 1) & 1, &fail_s))
					{
						fail_s = 1;
						ok = false;
						break;
					}
					mbar_expect_tx(&full[s], (uint32_t)tp.stage_bytes);
					tma_load_4d(ring + (size_t)s * tp.stage_bytes, map, 0, (L.fi * G.nkt + kt) * kKT, 0, L.blk, &full[s]);
					issued_s = kk + 1;
				}
			}
		}
	}
	else if(warp == 1)
	{
		if(lane == 0)
		{
			// ---- MMA issuer.  Instruction descriptor: D format F32 (bit 4), A / B
			// formats (bits 7-9 / 10-12: 0 F16, 1 BF16), A and B MN-major (bits 15,
			// 16), N >> 3 (bits 17-22), M = 128 (bits 24-28: M >> 4).  Rows of the
			// second tile past Wh are whatever follows the stage in shared memory;
			// their products are never read.
			const uint32_t fixed = (1u << 4) | (tp.h16 ? 0u : (1u << 7) | (1u << 10)) | (1u << 15) | (1u << 16) |
			                       ((128u >> 4) << 24);
			const uint32_t id0 = fixed | ((uint32_t)(Wh >> 3) << 17);
			const uint32_t id1 = fixed | ((uint32_t)((Wh - 128) >> 3) << 17);
			int kk = 0, ku = 0;
			bool ok = true;
			for(int u = blockIdx.x; u < xm.nunits && ok; u += gridDim.x, ku++)
			{
				const UnitLoc L = locate(xm, u);
				const XGroupRec &G = xm.g[L.gi];
				const int nk = G.nkt * (L.slice + 1) / G.nslice - G.nkt * L.slice / G.nslice;
				const int buf = nbuf == 2 ? ku & 1 : 0;
				const int round = nbuf == 2 ? ku >> 1 : ku;
				if(round > 0)
				{
					// the epilogue has read this buffer's previous unit
					if(!mbar_wait(&acc_empty[buf], (round - 1) & 1, &fail_s))
					{
						fail_s = 3;
						ok = false;
						break;
					}
					asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
				}
				const uint32_t d0 = tmem + (uint32_t)(buf * tp.cols), d1 = L.tile == 1 ? d0 : d0 + (uint32_t)Wh;
				for(int kt = 0; kt < nk; kt++, kk++)
				{
					const int s = kk % nst;
					if(!mbar_wait(&full[s], (kk / nst) & 1, &fail_s))
					{
						fail_s = 2;
						ok = false;
						break;
					}
					consumed_s = kk + 1;
					asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
					const uint32_t sb = smem_u32(ring + (size_t)s * tp.stage_bytes);
#pragma unroll
					for(int ks = 0; ks < kKT / 16; ks++)
					{
						const uint32_t more = (kt > 0 || ks > 0) ? 1u : 0u;
						if(L.tile != 1)
						{
							const uint64_t da = desc_mn64(sb + ks * 1024);
							mma_f16(d0, da, da, id0, more);
						}
						if(L.tile != 0 && Wh > 128)
						{
							const uint64_t db = desc_mn64(sb + 4 * kChunk + ks * 1024);
							mma_f16(d1, db, db, id1, more);
						}
					}
					mma_commit(&empty[s]);
				}
				if(ok)
					mma_commit(&acc_full[buf]);
			}
			// every MMA issued by this thread has completed once this arrives
			mma_commit(&mma_done);
			if(!mbar_wait(&mma_done, 0, &fail_s))
				fail_s = 4;
		}
	}
	else
	{
		// ---- epilogue: warps of quadrant q read tensor-memory lanes 32 q .. + 31,
		// taking every other pair of columns inputs
		constexpr int LR = 2 * CB;               // operand rows (and columns) of one input
		const int q = warp & 3, half = (warp - 2) >> 2;
		const int cl = (lane >> 1) & (CB - 1), p = lane & 1;
		const int nin = tp.nrow;
		constexpr float unscale = (float)(1 << (2 * kTcSpecExp));
		int ku = 0;
		for(int u = blockIdx.x; u < xm.nunits; u += gridDim.x, ku++)
		{
			const int buf = nbuf == 2 ? ku & 1 : 0;
			const int round = nbuf == 2 ? ku >> 1 : ku;
			const UnitLoc L = locate(xm, u);
			const XGroupRec &G = xm.g[L.gi];
			const DevFreqPlan &P = G.plans[G.plan_idx[L.fi]];
			const int nout = P.acc_cstride, c = pos_chan(P.pbits, L.blk * CB + cl);
			const int32_t *dA = P.destA, *dB = P.destB;
			// one slice: added to the accumulators; more: stored into the slice's sums
			const bool sliced = G.nslice > 1;
			float2 *dst = sliced ? G.ws + (int64_t)L.slice * G.ws_slice + ((int64_t)L.fi * G.nchan + c) * G.ws_nout
			                     : G.acc + P.acc_off + (int64_t)c * nout;
			if(!__all_sync(0xffffffffu, mbar_wait(&acc_full[buf], round & 1, &fail_s)))
			{
				fail_s = 6;
				break;                        // the warp leaves together
			}
			asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
			for(int i = L.tile == 1 ? 1 : 0; 128 * i < Wh && (L.tile < 0 || i == L.tile); i++)
			{
				const int rb = (128 * i + 32 * q) / LR;      // first input of this warp's lanes
				if(rb >= nin)
					break;
				const int row = rb + lane / LR;
				const uint32_t tb = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(buf * tp.cols + (L.tile == 1 ? -128 : i * (Wh - 128)));
				for(int a = rb + 2 * half; a < nin; a += 4)
				{
					// columns of inputs a and a + 1 (column n of the block is column n
					// of tile 0 and n - 128 of tile 1, which starts at Wh, or at 0 alone)
					float v[2 * LR];
					tmem_ld<2 * LR>(tb + (uint32_t)(a * LR), v);
					tmem_ld_wait();
					const float xa = pick<CB>(v, cl), ya = pick<CB>(v + 1, cl);
					const float xb = pick<CB>(v + LR, cl), yb = pick<CB>(v + LR + 1, cl);
					// the even lane (real row) makes the output of a, the odd one that of a + 1
					const float rx = __shfl_xor_sync(0xffffffffu, p ? xa : xb, 1);
					const float ry = __shfl_xor_sync(0xffffffffu, p ? ya : yb, 1);
					const int b = a + p;
					float2 o;
					o.x = (p ? rx + yb : xa + ry) * unscale;
					o.y = (p ? xb - ry : rx - ya) * unscale;
					if(row <= b && b < nin)
					{
						const int oa = __ldg(dA + row * nin + b), ob = __ldg(dB + row * nin + b);
						if(sliced)
						{
							if(oa >= 0)
								dst[oa] = o;
							if(ob >= 0)
								dst[ob] = make_float2(o.x, -o.y);
						}
						else
						{
							if(oa >= 0)
								atomicAdd(dst + oa, o);
							if(ob >= 0)
								atomicAdd(dst + ob, make_float2(o.x, -o.y));
						}
					}
					__syncwarp();             // the next load is the whole warp's
				}
			}
			asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
			__syncwarp();
			if(lane == 0)
				mbar_arrive(&acc_empty[buf]);
		}
	}

	asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
	__syncthreads();
	if(threadIdx.x == 0)
	{
		// on the error path, wait (bounded) for TMA loads that nobody consumed
		for(int kk = consumed_s; kk < issued_s; kk++)
			mbar_wait(&full[kk % nst], (kk / nst) & 1, &fail_s);
		if(fail_s && tp.err)
			atomicExch(tp.err, fail_s);
	}
	__syncthreads();
	asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
	if(warp == 1)
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"((uint32_t)tp.tcols));
}

// adds the slices' sums of one group, in slice order, to the accumulators
__global__ void __launch_bounds__(256) k_xmac_merge(const DevFreqPlan *__restrict__ plans,
                                                    const int32_t *__restrict__ plan_idx, int nslice, int64_t ws_slice,
                                                    int ws_nout, const float2 *__restrict__ ws, float2 *__restrict__ acc)
{
	const DevFreqPlan &P = plans[plan_idx[blockIdx.z]];
	const int c = blockIdx.y, o = blockIdx.x * blockDim.x + threadIdx.x, nout = P.acc_cstride;
	if(c >= P.nchan || o >= nout || P.outsrc[o] < 0)
		return;
	const float2 *w = ws + ((int64_t)blockIdx.z * P.nchan + c) * ws_nout + o;
	float2 s = w[0];
	for(int k = 1; k < nslice; k++)
	{
		const float2 v = w[k * ws_slice];
		s.x += v.x;
		s.y += v.y;
	}
	float2 *d = acc + P.acc_off + (int64_t)c * nout + o;
	const float2 t = *d;
	*d = make_float2(t.x + s.x, t.y + s.y);
}

// ---------------------------------------------------------------- host side
static int h_halves(const TcShape &s) { return 2 * s.trow * s.CB; }
static int h_cols(const TcShape &s)
{
	const int Wh = h_halves(s);
	return Wh > 128 && !s.split ? 2 * Wh - 128 : Wh;
}

static bool h_stages(TcShape *s, int nst, int nb)
{
	const int stage = h_halves(*s) / 32 * kChunk;
	// two CTAs per SM: 256 tensor-memory columns each
	if(nst < 2 || nst > kMaxStages || nb < 1 || nb > 2 || (nb == 1 && h_cols(*s) > 256))
		return false;
	// the second tile's operand is read up to three pieces past the last stage
	const size_t smem = 1024 + (size_t)nst * stage + 3 * kChunk;
	if(smem > (size_t)(nb == 2 ? 227 : 112) * 1024)
		return false;
	s->nrs = nst;
	s->nas = 0;
	s->nb = nb;
	s->smem = smem;
	return true;
}

// Time slices of a group: rounds of units over the resident CTAs times the K
// tiles of each, every unit with an epilogue worth about kEpi K tiles, and the
// sums of more than one slice written and read once more (kMerge K tiles each).
// 40 inputs x 128 channels x 4 subbands, T = 4096 (256 units): 180 us whole, 79 us
// in slices.
static int h_slices(const TcShape &s, int nf, int nsm)
{
	constexpr int kEpi = 6, kMerge = 2;
	const int64_t units = (int64_t)(s.nchan / s.CB) * nf * (1 + s.split), ctas = (int64_t)nsm * (s.nb == 1 ? 2 : 1);
	int best = 1;
	int64_t least = -1;
	for(int n = 1; n <= kMaxSlice && n <= s.nkt; n++)
	{
		const int64_t cost = (units * n + ctas - 1) / ctas * ((s.nkt + n - 1) / n + kEpi + (n > 1 ? kMerge : 0));
		if(least < 0 || cost * 16 < least * 15)
		{
			least = cost;
			best = n;
		}
	}
	return best;
}

bool tc_shape(int nrow, int nchan, int nf, int T, int nsm, bool f8, bool h16, TcShape *s)
{
	memset(s, 0, sizeof(*s));
	s->f8 = f8 ? 1 : 0;
	s->h16 = h16 ? 1 : 0;
	s->nrow = nrow;
	s->nchan = nchan;
	s->T = T;
	if(nrow <= 0 || nrow > 64)
		return false;
	if(f8)
		return f8_shape(s);
	// channels per block, and rows padded to whole 64-byte pieces
	s->CB = nrow <= 12 ? 8 : (nrow <= 24 ? 4 : 2);
	const int m = 16 / s->CB;
	s->trow = (nrow + m - 1) / m * m;
	s->Tpad = (T + kKT - 1) / kKT * kKT;
	s->nkt = s->Tpad / kKT;
	// accumulators of more than 256 columns (more than 48 inputs) would leave one
	// CTA per SM and nothing to run beside its epilogue: each of the two operand
	// tiles becomes a unit of its own, at the price of reading the spectra twice
	// (64 inputs x 4 x 1024 channels, T = 250: 156 us whole, 134 us split)
	s->split = h_cols(*s) > 256 ? 1 : 0;
	// two CTAs per SM where their accumulators fit, the deepest ring
	bool ok = false;
	for(int nb = h_cols(*s) <= 256 ? 1 : 2; nb <= 2 && !ok; nb++)
		for(int nst = nb == 1 ? 8 : kMaxStages; nst >= 2 && !ok; nst--)
			ok = h_stages(s, nst, nb);
	s->nslice = ok ? h_slices(*s, nf, nsm) : 1;
	return ok;
}

// ring depth and CTAs per SM (nb 1: two CTAs; 2: one).  The slices stay as
// they are: they belong to the result.
bool tc_stages(TcShape *s, int nrs, int nas, int nb) { return s->f8 ? f8_stages(s, nrs, nas, nb) : h_stages(s, nrs, nb); }

size_t tc_tensormap_size() { return sizeof(CUtensorMap); }

// 4D map over one group's spectra [nf * Tpad][nblk][trow * CB] of 4-byte values:
// 16 values (64 bytes) x times x pieces of the run x blocks; box {16, 32, all
// pieces, 1}, 64-byte swizzle.
bool tc_make_tensormap(void *map_out, const void *spec, const TcShape &s, int nf)
{
	if(((uintptr_t)map_out & 63) != 0 || ((uintptr_t)spec & 15) != 0)
		return false;
	if(s.f8)
		return f8_tensormap(map_out, spec, s, nf);
	const PFN_encodeTiled encode = tensormap_encoder();
	if(!encode)
		return false;
	const cuuint64_t W = (cuuint64_t)s.trow * s.CB, nch = W / 16, nblk = (cuuint64_t)(s.nchan / s.CB);
	cuuint64_t dims[4] = {16, (cuuint64_t)s.Tpad * nf, nch, nblk};
	cuuint64_t strides[3] = {nblk * W * 4, 64, W * 4};
	cuuint32_t box[4] = {16, (cuuint32_t)kKT, (cuuint32_t)nch, 1};
	cuuint32_t estr[4] = {1, 1, 1, 1};
	return encode((CUtensorMap *)map_out, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, (void *)spec, dims, strides, box, estr,
	              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
	              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// complex values of the slices' sums of one group (0: one slice)
int64_t tc_workspace(const TcShape &s, int nf, int maxout)
{
	return s.nslice > 1 ? (int64_t)s.nslice * nf * s.nchan * maxout : 0;
}

bool xmac_multi_add(XMultiArgs *xm, const void *tmap, const TcShape &s, const DevFreqPlan *dplans,
                    const int32_t *plan_idx, int nf, float2 *ws, int maxout, float2 *acc)
{
	if(xm->ngroups >= kXMultiGroups || ((uintptr_t)tmap & 63) != 0 || nf <= 0)
		return false;
	XGroupRec &g = xm->g[xm->ngroups];
	memcpy(&xm->map[xm->ngroups], tmap, sizeof(CUtensorMap));
	g.plans = dplans;
	g.plan_idx = plan_idx;
	g.acc = acc;
	g.ws = ws;
	g.ws_nout = maxout;
	g.ws_slice = (int64_t)nf * s.nchan * maxout;
	g.nchan = s.nchan;
	g.nkt = s.nkt;
	g.nblk = (s.nchan + s.CB - 1) / s.CB;
	g.nslice = s.nslice;
	g.nf = nf;
	g.split = s.split;
	g.unit0 = xm->nunits;
	xm->nunits += g.nblk * nf * s.nslice * (1 + s.split);
	xm->ngroups++;
	return true;
}

void launch_xmac_tc_multi(const XMultiArgs &xm, const TcShape &s, int nsm, int32_t *err, cudaStream_t stream)
{
	if(xm.ngroups <= 0 || xm.nunits <= 0)
		return;
	if(s.f8)
	{
		f8_launch(xm, s, nsm, err, stream);
		return;
	}
	XhParams tp;
	tp.nrow = s.nrow;
	tp.nch = h_halves(s) / 32;
	tp.stage_bytes = tp.nch * kChunk;
	tp.nst = s.nrs;
	tp.cols = h_cols(s);
	const int room = s.nb == 1 ? 256 : 512;
	tp.nbuf = 2 * tp.cols <= room ? 2 : 1;
	tp.tcols = 32;
	while(tp.tcols < tp.nbuf * tp.cols)
		tp.tcols *= 2;
	tp.h16 = s.h16;
	tp.err = err;
	const int ctas = nsm * (s.nb == 1 ? 2 : 1);
	auto go = [&](auto kern) {
		cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s.smem);
		kern<<<xm.nunits < ctas ? xm.nunits : ctas, kThreads, s.smem, stream>>>(xm, tp);
	};
	if(s.CB == 8)
		go(k_xmac_h<8>);
	else if(s.CB == 4)
		go(k_xmac_h<4>);
	else
		go(k_xmac_h<2>);
	for(int i = 0; i < xm.ngroups; i++)
	{
		const XGroupRec &g = xm.g[i];
		if(g.nslice > 1)
			k_xmac_merge<<<dim3((g.ws_nout + 255) / 256, g.nchan, g.nf), 256, 0, stream>>>(
			    g.plans, g.plan_idx, g.nslice, g.ws_slice, g.ws_nout, g.ws, g.acc);
	}
}

void launch_xmac_tc(const void *tmap, const TcShape &s, const DevFreqPlan *dplans, const int32_t *plan_idx, int nf,
                    float2 *ws, int maxout, int nsm, int32_t *err, float2 *acc, cudaStream_t stream)
{
	XMultiArgs xm;
	memset(&xm, 0, sizeof(xm));
	if(!xmac_multi_add(&xm, tmap, s, dplans, plan_idx, nf, ws, maxout, acc))
		return;                      // refused by tc_make_tensormap at set-up already
	launch_xmac_tc_multi(xm, s, nsm, err, stream);
}

}  // namespace fxb
