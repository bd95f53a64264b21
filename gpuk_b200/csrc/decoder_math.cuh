// Arithmetic of a decoder layer's elementwise steps, shared by their kernels and by the epilogues of the projections in front of them.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace gpuk {

// f / (1 + exp(-f)).  The quotient is that of an approximate reciprocal, corrected once by the residual f - q b, which a fused multiply-add gives without rounding (P. Markstein,
// Computation of elementary functions on the IBM RISC System/6000 processor, IBM Journal of Research and Development 34, 1990); the division operator for zeros,
// infinities and where the residual could leave the range.  Rounded to bf16 the same as silu by the operator for each of the 65536 inputs.
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

// Where a position points in the cache and in the table of angles.  A negative one counts from the end of what it indexes, as in an indexed tensor.
struct Place {
    int64_t at, angle;
    bool valid;      // inside both: otherwise nothing goes to the caches, the queries become NaN, and the status word says so
};
__device__ __forceinline__ Place place_of(int64_t position, int max_seq, int table_rows) {
    Place p = {position < 0 ? position + max_seq : position, position < 0 ? position + table_rows : position, false};
    p.valid = p.at >= 0 && p.at < max_seq && p.angle >= 0 && p.angle < table_rows;
    return p;
}
constexpr uint32_t kNan2 = 0x7fff7fffu;      // two bf16

}  // namespace gpuk
