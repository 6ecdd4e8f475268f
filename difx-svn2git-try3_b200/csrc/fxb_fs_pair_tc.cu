// F stage of two-band work items, tensor-core-form spectra (see
// fxb_fstage_pair.cuh): the persistent launches, and complex sampling.
#include "fxb_fstage_pair.cuh"

namespace fxb {

// One CTA per work unit (grid as k_fstage).
template <int LOGN, bool TCO, int VAR>
__global__ void __launch_bounds__(PShape<LOGN>::NT, PShape<LOGN>::MINB) k_fstage_pair(const FsArgs a)
{
	extern __shared__ __align__(16) ulonglong2 fsp[];
	__shared__ float lut8[256];
	__shared__ u64 lut4[16];
	__shared__ PairConst fcs[kMaxTQ * PShape<LOGN>::FPC];
	__shared__ PairOut po;
	const int item = a.items_fast ? blockIdx.x : blockIdx.y;
	const int tchunk = a.items_fast ? blockIdx.y : blockIdx.x;
	fstage_pair_luts(lut8, lut4);
	__syncthreads();
	fstage_pair_unit<LOGN, TCO, VAR>(a, a.first + item, tchunk, a.tq, (const float2 *)a.tw, fsp, lut8, lut4, fcs, &po);
}

template <int LOGN, bool TCO, int VAR>
static void launch_t(const FKind &k, const FsArgs &a, cudaStream_t stream)
{
	cudaFuncSetAttribute(k_fstage_pair<LOGN, TCO, VAR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.smem);
	cudaFuncSetAttribute(k_fstage_pair<LOGN, TCO, VAR>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
	k_fstage_pair<LOGN, TCO, VAR><<<fstage_grid(k, a), k.threads, k.smem, stream>>>(a);
}

constexpr size_t kPairSide = 2304 * 16;          // exchange buffers of 2048 points in all, padded

// Work-list class 5 VAR + 3: every length up to 2048 points in CTAs of 256
// threads.  VAR 0: plain VDIF, 1: raw INTERLACEDVDIF reads.
template <int VAR>
__global__ void __launch_bounds__(256, 3) k_fstage_pair_pn(const __grid_constant__ FsMultiArgs m)
{
	extern __shared__ __align__(16) ulonglong2 fsp[];
	__shared__ float lut8[256];
	__shared__ u64 lut4[16];
	__shared__ PairConst fcs[kFsMultiFc];
	__shared__ PairOut po;
	__shared__ int unit_s[2];
	constexpr int cls = kFsMultiPer * VAR + 3;
	fstage_pair_luts(lut8, lut4);
	UnitFeed feed(m.ctr + cls, unit_s);
	for(int u = feed.first(); u < m.nunit[cls]; u = feed.next())
	{
		const FsMultiUnit w = m.units[m.unit0[cls] + u];
		const FsMultiKind k = m.kinds[w.kind];
		const float2 *tw = (const float2 *)k.tw;
		const int gi = k.first + w.item;
		switch(k.code & 31)
		{
		case 5: fstage_pair_unit<5, true, VAR>(m.m[k.member], gi, w.tchunk, k.tq, tw, fsp, lut8, lut4, fcs, &po); break;
		case 6: fstage_pair_unit<6, true, VAR>(m.m[k.member], gi, w.tchunk, k.tq, tw, fsp, lut8, lut4, fcs, &po); break;
		case 7: fstage_pair_unit<7, true, VAR>(m.m[k.member], gi, w.tchunk, k.tq, tw, fsp, lut8, lut4, fcs, &po); break;
		case 8: fstage_pair_unit<8, true, VAR>(m.m[k.member], gi, w.tchunk, k.tq, tw, fsp, lut8, lut4, fcs, &po); break;
		case 9: fstage_pair_unit<9, true, VAR>(m.m[k.member], gi, w.tchunk, k.tq, tw, fsp, lut8, lut4, fcs, &po); break;
		case 10: fstage_pair_unit<10, true, VAR>(m.m[k.member], gi, w.tchunk, k.tq, tw, fsp, lut8, lut4, fcs, &po); break;
		case 11: fstage_pair_unit<11, true, VAR>(m.m[k.member], gi, w.tchunk, k.tq, tw, fsp, lut8, lut4, fcs, &po); break;
		default: break;
		}
	}
}

// 4096 points (class 5 VAR + 2) in CTAs of 512 threads, 8192 (class 5 VAR) of 1024
template <int VAR, int LOGN>
__global__ void __launch_bounds__(PShape<LOGN>::NT, PShape<LOGN>::MINB)
    k_fstage_pair_pw(const __grid_constant__ FsMultiArgs m)
{
	extern __shared__ __align__(16) ulonglong2 fsp[];
	__shared__ float lut8[256];
	__shared__ u64 lut4[16];
	__shared__ PairConst fcs[kMaxTQ];
	__shared__ PairOut po;
	__shared__ int unit_s[2];
	constexpr int cls = kFsMultiPer * VAR + (LOGN == 12 ? 2 : 0);
	fstage_pair_luts(lut8, lut4);
	UnitFeed feed(m.ctr + cls, unit_s);
	for(int u = feed.first(); u < m.nunit[cls]; u = feed.next())
	{
		const FsMultiUnit w = m.units[m.unit0[cls] + u];
		const FsMultiKind k = m.kinds[w.kind];
		fstage_pair_unit<LOGN, true, VAR>(m.m[k.member], k.first + w.item, w.tchunk, k.tq, (const float2 *)k.tw, fsp, lut8,
		                                  lut4, fcs, &po);
	}
}

template <int VAR>
static void launch_cls(const FsMultiArgs &m, int c, int nsm, cudaStream_t st)
{
	if(c == 3)
		fs_launch_persistent(k_fstage_pair_pn<VAR>, m, kFsMultiPer * VAR + c, 3 * nsm, 256, kPairSide, st);
	else if(c == 2)
		fs_launch_persistent(k_fstage_pair_pw<VAR, 12>, m, kFsMultiPer * VAR + c, 2 * nsm, 512, 2 * kPairSide, st);
	else
		fs_launch_persistent(k_fstage_pair_pw<VAR, 13>, m, kFsMultiPer * VAR + c, nsm, 1024, 4 * kPairSide, st);
}

void launch_fs_pair_multi(const FsMultiArgs &m, int cls, int nsm, cudaStream_t st)
{
	if(cls >= kFsMultiPer)
		launch_cls<1>(m, cls - kFsMultiPer, nsm, st);
	else
		launch_cls<0>(m, cls, nsm, st);
}

void launch_fs_pair_tc(const FKind &k, const FsArgs &a, cudaStream_t stream)
{
	if(!k.cplx)
		return;
	switch(k.N)
	{
	case 32: launch_t<5, true, 2>(k, a, stream); break;
	case 64: launch_t<6, true, 2>(k, a, stream); break;
	case 128: launch_t<7, true, 2>(k, a, stream); break;
	case 256: launch_t<8, true, 2>(k, a, stream); break;
	case 512: launch_t<9, true, 2>(k, a, stream); break;
	case 1024: launch_t<10, true, 2>(k, a, stream); break;
	case 2048: launch_t<11, true, 2>(k, a, stream); break;
	case 4096: launch_t<12, true, 2>(k, a, stream); break;
	case 8192: launch_t<13, true, 2>(k, a, stream); break;
	default: break;
	}
}

}  // namespace fxb
