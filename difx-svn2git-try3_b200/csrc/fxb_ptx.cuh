// Wrappers of PTX instructions that several kernels use (sm_100a): mbarriers,
// packed pairs of FP32 values, and the rounding of spectra to 16 bits.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cstdint>

namespace fxb {

constexpr uint32_t kWaitLimit = 1u << 22;

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
	asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes)
{
	asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes)
	             : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
	asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}

// bounded wait for the phase with parity `parity`; gives up early once
// another role has recorded a failure
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, volatile int *fail)
{
	const uint32_t a = smem_u32(bar);
	for(uint32_t it = 0; it < kWaitLimit; it++)
	{
		uint32_t done;
		asm volatile(
		    "{\n\t.reg .pred p;\n\t"
		    "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
		    "selp.u32 %0, 1, 0, p;\n\t}\n"
		    : "=r"(done)
		    : "r"(a), "r"(parity)
		    : "memory");
		if(done)
			return true;
		if((it & 255u) == 255u && *fail)
			return false;
	}
	return false;
}

// two FP32 values in one register pair
typedef unsigned long long u64;

__device__ __forceinline__ u64 pk2(float a, float b)
{
	u64 d;
	asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
	return d;
}
__device__ __forceinline__ float2 up2(u64 v)
{
	float2 r;
	asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
	return r;
}
__device__ __forceinline__ u64 add2(u64 a, u64 b)
{
	u64 d;
	asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
	return d;
}
__device__ __forceinline__ u64 sub2(u64 a, u64 b)
{
	u64 d;
	asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
	return d;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b)
{
	u64 d;
	asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
	return d;
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c)
{
	u64 d;
	asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
	return d;
}

__device__ __forceinline__ uint32_t pack_h2(float a, float b)
{
	const __half2 h = __floats2half2_rn(a, b);
	return *(const uint32_t *)&h;
}
__device__ __forceinline__ uint32_t pack_h2(u64 v)
{
	const float2 f = up2(v);
	return pack_h2(f.x, f.y);
}

// one spectral value of the tensor-core forms: (re, im) as half2 or bf16x2
__device__ __forceinline__ uint32_t pack_spec(bool h16, float re, float im)
{
	if(h16)
		return pack_h2(re, im);
	const __nv_bfloat162 b = __floats2bfloat162_rn(re, im);
	return *(const uint32_t *)&b;
}

}  // namespace fxb
