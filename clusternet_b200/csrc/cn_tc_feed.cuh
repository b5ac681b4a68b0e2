// What the kernels that split both operands themselves share (cn_gemm_small.cu, cn_gemm_outer.cu): operands in any layout and alignment as TF32
// hi / lo parts.
#pragma once
#include "cn_gemm.h"
#include "cn_tc.cuh"

#define SM_BM 128
#define SM_BK 32

// An operand: element (row, k) at p[row * sr + k * sk].
struct SmOperand {
    const float *p;
    int64_t sr, sk;
    int vec;                // 16-byte aligned along the contiguous one of the two
};
static inline SmOperand sm_operand(const float *p, bool k_contiguous, int64_t ld)
{
    SmOperand o;
    o.p = p;
    o.sr = k_contiguous ? ld : 1;
    o.sk = k_contiguous ? 1 : ld;
    o.vec = (ld & 3) == 0 && ((uintptr_t)p & 15u) == 0;
    return o;
}

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

// D[tmem] (+)= A[smem] * B[smem], both K-major TF32 tiles.
__device__ __forceinline__ void sm_mma_ss(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t desc_hi, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 ad, bd;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 ad, {%1, %3};\n\t"
        "mov.b64 bd, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], ad, bd, %4, p;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate) : "memory");
}
