// What the kernels that split both operands themselves share (cn_gemm_small.cu, cn_gemm_outer.cu): fp32 rounded to TF32, stores of 16 bytes to
// shared memory, the rows of a tile and the k of a block.
#pragma once
#include "cn_gemm.h"
#include "cn_tc.cuh"

#define SM_BM 128
#define SM_BK 32

// fp32 -> TF32, round to nearest with ties away from zero: add half a TF32 ulp to the magnitude bits and truncate.  That carry takes
// the finite values from 0x7f7ff000 up to infinity and a NaN with a full mantissa (0x7fffffff, the one GPU arithmetic makes)
// over into the sign bit, to -0.  CAREFUL truncates those instead, NaNs after an addition that makes them the canonical one.
template <bool CAREFUL>
__device__ __forceinline__ uint32_t sm_tf32(float x)
{
    if (!CAREFUL) return (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
    const float top = __uint_as_float(0x7f7ff000u);
    return (fabsf(x) < top ? __float_as_uint(x) + 0x1000u : __float_as_uint(__fadd_rn(x, 0.0f))) & 0xffffe000u;
}

__device__ __forceinline__ void sts4u(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w)
{
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

__device__ __forceinline__ void sts4f(uint32_t a, const float *v)
{
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]) : "memory");
}
