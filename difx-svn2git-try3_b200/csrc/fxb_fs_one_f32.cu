// F stage of one-band work items, FP32 spectra (see fxb_fstage.cuh).
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
	case 16384: launch_t<14, false, VAR>(k, a, stream); break;
	default: break;
	}
}

void launch_fs_one_f32(const FKind &k, const FsArgs &a, cudaStream_t stream)
{
	if(k.muxraw)
		launch_var<1>(k, a, stream);
	else if(k.cplx)
		launch_var<2>(k, a, stream);
	else
		launch_var<0>(k, a, stream);
}

}  // namespace fxb
