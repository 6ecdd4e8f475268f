// Device code shared by the tensor-core XMAC kernels (sm_100a).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdint>

#include "fxb_internal.h"
#include "fxb_kernels.h"
#include "fxb_ptx.cuh"

namespace fxb {

namespace {

__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, int x, int y, int z, uint64_t *bar)
{
	asm volatile(
	    "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(
	        smem_u32(dst)),
	    "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
	    : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t *bar)
{
	asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_u32(bar))
	             : "memory");
}

__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }

// tensor maps are encoded through the driver entry point (no link to libcuda)
typedef CUresult (*PFN_encodeTiled)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                     const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                     CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline PFN_encodeTiled tensormap_encoder()
{
	static PFN_encodeTiled encode = nullptr;
	if(!encode)
	{
		void *fn = nullptr;
		cudaDriverEntryPointQueryResult q;
		if(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess &&
		   q == cudaDriverEntryPointSuccess)
			encode = (PFN_encodeTiled)fn;
	}
	return encode;
}

// unit u of a launch: its group, subband of the group, channel block, time slice
// and operand tile (-1: all of them)
struct UnitLoc {
	int gi, fi, blk, slice, tile;
};
__device__ __forceinline__ UnitLoc locate(const XMultiArgs &xm, int u)
{
	int gi = 0;
	while(gi + 1 < xm.ngroups && u >= xm.g[gi + 1].unit0)
		gi++;
	int lu = u - xm.g[gi].unit0, tile = -1;
	if(xm.g[gi].split)
	{
		tile = lu & 1;
		lu >>= 1;
	}
	const int nblk = xm.g[gi].nblk, ns = xm.g[gi].nslice;
	const int r = lu / ns, fi = r / nblk;
	return UnitLoc{gi, fi, r - fi * nblk, lu - r * ns, tile};
}

}  // namespace

}  // namespace fxb
