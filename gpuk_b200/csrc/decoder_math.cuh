// Arithmetic of a decoder layer's elementwise steps, shared by their kernels and by the epilogues of the projections in front of them.
#pragma once

#include <cuda_runtime.h>

namespace gpuk {

// f / (1 + exp(-f)): the quotient by reciprocal and one exact-residual correction (bf16 results as with the division on everything tried), the
// division itself for zeros, infinities and where the residual could leave the range.
__device__ __forceinline__ float silu(float f) {
    const float b = 1.0f + expf(-f);
    if (!(fabsf(f) > 1e-30f && fabsf(f) < 1e30f && b < 1e30f)) return f / b;
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
    const float q = f * y;
    return fmaf(fmaf(-q, b, f), y, q);
}

// One pair of a rotary embedding: products and sums each rounded, no fused multiply-add, as a chain of operators rounds them.
__device__ __forceinline__ void rotate(float x1, float x2, float c, float s, float &lo, float &hi) {
    lo = __fsub_rn(__fmul_rn(x1, c), __fmul_rn(x2, s));
    hi = __fadd_rn(__fmul_rn(x2, c), __fmul_rn(x1, s));
}

}  // namespace gpuk
