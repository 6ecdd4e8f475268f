// F stage of two-band work items, FP32 spectra (see fxb_fstage_pair.cuh).
#include "fxb_fstage_pair.cuh"

namespace fxb {

// One CTA per work unit (grid as k_fstage).
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

template <int VAR>
static void launch_var(const FKind &k, const FsArgs &a, cudaStream_t stream)
{
	switch(k.N)
	{
	case 32: launch_t<5, false, VAR>(k, a, stream); break;
	case 64: launch_t<6, false, VAR>(k, a, stream); break;
	case 128: launch_t<7, false, VAR>(k, a, stream); break;
	case 256: launch_t<8, false, VAR>(k, a, stream); break;
	case 512: launch_t<9, false, VAR>(k, a, stream); break;
	case 1024: launch_t<10, false, VAR>(k, a, stream); break;
	case 2048: launch_t<11, false, VAR>(k, a, stream); break;
	case 4096: launch_t<12, false, VAR>(k, a, stream); break;
	case 8192: launch_t<13, false, VAR>(k, a, stream); break;
	default: break;
	}
}

void launch_fs_pair_f32(const FKind &k, const FsArgs &a, cudaStream_t stream)
{
	if(k.muxraw)
		launch_var<1>(k, a, stream);
	else if(k.cplx)
		launch_var<2>(k, a, stream);
	else
		launch_var<0>(k, a, stream);
}

}  // namespace fxb
