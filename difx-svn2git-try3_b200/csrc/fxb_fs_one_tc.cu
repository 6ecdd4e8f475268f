// F stage of one-band work items, tensor-core-form spectra (see
// fxb_fstage.cuh): the persistent launches, and the kinds outside them
// (complex sampling, 16384-point FFTs).
#include "fxb_fstage.cuh"

namespace fxb {

// One CTA per work unit.  grid: (time chunks, items), or (items, time chunks)
// when the stations of a subband should run side by side (blocked
// tensor-core spectra).
template <int LOGN, bool TCO, int VAR>
__global__ void __launch_bounds__(FShape<LOGN>::NT, FShape<LOGN>::MINB) k_fstage(const FsArgs a)
{
	extern __shared__ __align__(16) uint2 fsm[];
	__shared__ float lut8[256];
	__shared__ FftConst fcs[kMaxTQ * FShape<LOGN>::FPC];
	const int item = a.items_fast ? blockIdx.x : blockIdx.y;
	const int tchunk = a.items_fast ? blockIdx.y : blockIdx.x;
	fstage_luts(lut8);
	__syncthreads();
	fstage_unit<LOGN, TCO, VAR>(a, a.first + item, tchunk, a.tq, a.pp, (const float2 *)a.tw, fsm, lut8, fcs);
}

template <int LOGN, bool TCO, int VAR>
static void launch_t(const FKind &k, const FsArgs &a, cudaStream_t stream)
{
	cudaFuncSetAttribute(k_fstage<LOGN, TCO, VAR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.smem);
	cudaFuncSetAttribute(k_fstage<LOGN, TCO, VAR>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
	k_fstage<LOGN, TCO, VAR><<<fstage_grid(k, a), k.threads, k.smem, stream>>>(a);
}

constexpr size_t kNarrowSide = 18432;            // exchange buffer: 2048 points of one band, padded
constexpr size_t kMidSide = 36864;               // 4096 points
constexpr size_t kWideSmem = 73728;              // 8192 points of one band, padded

// Work-list class 7 VAR + 5: every length up to 2048 points in CTAs of 256
// threads (the shape of k_fstage for those lengths), one exchange buffer per
// unit (three CTAs per SM): faster than two buffers at two CTAs per SM on every
// length measured.  VAR 0: plain VDIF, 1: raw INTERLACEDVDIF reads.
template <int VAR>
__global__ void __launch_bounds__(256, 3) k_fstage_pn(const __grid_constant__ FsMultiArgs m)
{
	extern __shared__ __align__(16) uint2 fsm[];
	__shared__ float lut8[256];
	__shared__ FftConst fcs[kFsMultiFc];
	__shared__ int unit_s[2];
	constexpr int cls = kFsMultiPer * VAR + 5;
	fstage_luts(lut8);
	UnitFeed feed(m.ctr + cls, unit_s);
	for(int u = feed.first(); u < m.nunit[cls]; u = feed.next())
	{
		const FsMultiUnit w = m.units[m.unit0[cls] + u];
		const FsMultiKind k = m.kinds[w.kind];
		const float2 *tw = (const float2 *)k.tw;
		const int gi = k.first + w.item;
		switch(k.code & 31)
		{
		case 5: fstage_unit<5, true, VAR>(m.m[k.member], gi, w.tchunk, k.tq, 0, tw, fsm, lut8, fcs); break;
		case 6: fstage_unit<6, true, VAR>(m.m[k.member], gi, w.tchunk, k.tq, 0, tw, fsm, lut8, fcs); break;
		case 7: fstage_unit<7, true, VAR>(m.m[k.member], gi, w.tchunk, k.tq, 0, tw, fsm, lut8, fcs); break;
		case 8: fstage_unit<8, true, VAR>(m.m[k.member], gi, w.tchunk, k.tq, 0, tw, fsm, lut8, fcs); break;
		case 9: fstage_unit<9, true, VAR>(m.m[k.member], gi, w.tchunk, k.tq, 0, tw, fsm, lut8, fcs); break;
		case 10: fstage_unit<10, true, VAR>(m.m[k.member], gi, w.tchunk, k.tq, 0, tw, fsm, lut8, fcs); break;
		case 11: fstage_unit<11, true, VAR>(m.m[k.member], gi, w.tchunk, k.tq, 0, tw, fsm, lut8, fcs); break;
		default: break;
		}
	}
}

// 4096 points (class 7 VAR + 3) in CTAs of 256 threads, 8192 (class 7 VAR + 1) of 512
template <int VAR, int LOGN>
__global__ void __launch_bounds__(FShape<LOGN>::NT, LOGN == 12 ? 3 : 2) k_fstage_pw(const __grid_constant__ FsMultiArgs m)
{
	extern __shared__ __align__(16) uint2 fsm[];
	__shared__ float lut8[256];
	__shared__ FftConst fcs[kMaxTQ];
	__shared__ int unit_s[2];
	constexpr int cls = kFsMultiPer * VAR + (LOGN == 12 ? 3 : 1);
	fstage_luts(lut8);
	UnitFeed feed(m.ctr + cls, unit_s);
	for(int u = feed.first(); u < m.nunit[cls]; u = feed.next())
	{
		const FsMultiUnit w = m.units[m.unit0[cls] + u];
		const FsMultiKind k = m.kinds[w.kind];
		fstage_unit<LOGN, true, VAR>(m.m[k.member], k.first + w.item, w.tchunk, k.tq, 0, (const float2 *)k.tw, fsm, lut8, fcs);
	}
}

template <int VAR>
static void launch_cls(const FsMultiArgs &m, int c, int nsm, cudaStream_t st)
{
	if(c == 5)
		fs_launch_persistent(k_fstage_pn<VAR>, m, kFsMultiPer * VAR + c, 3 * nsm, 256, kNarrowSide, st);
	else if(c == 3)
		fs_launch_persistent(k_fstage_pw<VAR, 12>, m, kFsMultiPer * VAR + c, 3 * nsm, 256, kMidSide, st);
	else
		fs_launch_persistent(k_fstage_pw<VAR, 13>, m, kFsMultiPer * VAR + c, 2 * nsm, 512, kWideSmem, st);
}

void launch_fs_one_multi(const FsMultiArgs &m, int cls, int nsm, cudaStream_t st)
{
	if(cls >= kFsMultiPer)
		launch_cls<1>(m, cls - kFsMultiPer, nsm, st);
	else
		launch_cls<0>(m, cls, nsm, st);
}

void launch_fs_one_tc(const FKind &k, const FsArgs &a, cudaStream_t stream)
{
	if(!k.cplx)
	{
		if(k.N == 16384 && k.muxraw)
			launch_t<14, true, 1>(k, a, stream);
		else if(k.N == 16384)
			launch_t<14, true, 0>(k, a, stream);
		return;
	}
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
	case 16384: launch_t<14, true, 2>(k, a, stream); break;
	default: break;
	}
}

}  // namespace fxb
