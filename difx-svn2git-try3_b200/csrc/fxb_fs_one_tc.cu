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

// CTAs per SM of a persistent launch: one exchange buffer each, three up to 4096
// points (faster than two buffers at two CTAs per SM on every length measured)
template <int LOGN>
struct OneShape {
	static constexpr int MINB = LOGN <= 12 ? 3 : 2;
};

// The units of one length (class 2 (13 - LOGN) + 1 of VAR 0: plain VDIF, 1: raw
// INTERLACEDVDIF reads), each in a kernel of its own: 14 stations x 1 band of 8 bits, F
// stage among the other lengths' code and alone, 4096 points 137 and 124 us, 2048
// points 82 and 68.
template <int VAR, int LOGN>
__global__ void __launch_bounds__(FShape<LOGN>::NT, OneShape<LOGN>::MINB) k_fstage_pw(const __grid_constant__ FsMultiArgs m)
{
	extern __shared__ __align__(16) uint2 fsm[];
	constexpr int FPC = FShape<LOGN>::FPC, NFC = kMaxTQ * FPC < kFsMultiFc ? kMaxTQ * FPC : kFsMultiFc;
	__shared__ float lut8[256];
	__shared__ FftConst fcs[NFC];
	__shared__ int unit_s[2];
	constexpr int cls = kFsMultiPer * VAR + 2 * (13 - LOGN) + 1;
	fstage_luts(lut8);
	UnitFeed feed(m.ctr + cls, unit_s);
	for(int u = feed.first(); u < m.nunit[cls]; u = feed.next())
	{
		const FsMultiUnit w = m.units[m.unit0[cls] + u];
		const FsMultiKind k = m.kinds[w.kind];
		fstage_unit<LOGN, true, VAR>(m.m[k.member], k.first + w.item, w.tchunk, k.tq, 0, (const float2 *)k.tw, fsm, lut8, fcs);
	}
}

template <int VAR, int LOGN>
static void launch_len(const FsMultiArgs &m, int nsm, cudaStream_t st)
{
	using SH = FShape<LOGN>;
	fs_launch_persistent(k_fstage_pw<VAR, LOGN>, m, kFsMultiPer * VAR + 2 * (13 - LOGN) + 1, OneShape<LOGN>::MINB * nsm,
	                     SH::NT, (size_t)SH::FPC * SH::PADN * 8, st);
}

template <int VAR>
static void launch_cls(const FsMultiArgs &m, int c, int nsm, cudaStream_t st)
{
	switch(13 - c / 2)
	{
	case 5: launch_len<VAR, 5>(m, nsm, st); break;
	case 6: launch_len<VAR, 6>(m, nsm, st); break;
	case 7: launch_len<VAR, 7>(m, nsm, st); break;
	case 8: launch_len<VAR, 8>(m, nsm, st); break;
	case 9: launch_len<VAR, 9>(m, nsm, st); break;
	case 10: launch_len<VAR, 10>(m, nsm, st); break;
	case 11: launch_len<VAR, 11>(m, nsm, st); break;
	case 12: launch_len<VAR, 12>(m, nsm, st); break;
	default: launch_len<VAR, 13>(m, nsm, st); break;
	}
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
