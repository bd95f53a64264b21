// The elementwise steps of a decoder layer between its projections, one launch each:
//
//   rope_append_kernel   rotary embedding of q and k and the write of k and v into the KV cache, straight from the
//                        q|k|v projection's output.  As PyTorch operators: slicing, four multiplications, two additions
//                        and a concatenation each for q and k, two casts, two indexed stores.
//   silu_mul_kernel      silu(w1 x) * (w3 x) from the joint w1|w3 output.
//
// 2048 tokens: silu of 28672 channels 58.5 us (6.0 TB/s; 86 with one vector a thread, 64-bit index divisions and IEEE quotients), rope of
// 64 + 16 heads 16.1 us (5.2 TB/s; 22 with 64-bit divisions).  A decode step: 2.4 and 2.3 us, all launch.
//
// Both are bound by their bytes for long prompts and by launch latency for a decode step, so what counts is one pass and
// one launch.  Rounding points are those of the operator chains: fp32 products and sums each rounded (no fused
// multiply-add), one rounding to bf16; silu rounded to bf16 before the multiplication.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/gpuk_b200.h"
#include "decoder_math.cuh"
#include "launch.cuh"
#include "linear.cuh"

namespace gpuk {
namespace {

using bf16 = __nv_bfloat16;
constexpr int kRopeVec = 16;      // elements of a head one thread takes: eight (even, odd) pairs, two 16-byte loads
constexpr int kThreads = 256;

struct RopeParams {
    const bf16 *qkv;         // [batch * t, (heads + 2 * kv_heads) * head_dim]
    const float *cos, *sin;  // [table_rows, head_dim / 2]
    const int64_t *pos;      // [t]
    bf16 *q_out;             // [batch * t, heads * head_dim]
    bf16 *k_cache, *v_cache; // [batch, kv_heads, max_seq, head_dim]
    int64_t total;           // threads with work
    int *status;             // of positions
    int t, heads, kv_heads, head_dim, table_rows, max_seq;
};

// Thread -> (row, head, part of the head), the part fastest: a warp reads one contiguous run of the row.
__global__ void __launch_bounds__(kThreads) rope_append_kernel(const __grid_constant__ RopeParams p) {
    grid_dependency_sync();
    // 32-bit quotients: a CTA's first row by one division, the rest from a small remainder
    const int parts = p.head_dim / kRopeVec, all = p.heads + 2 * p.kv_heads, row_threads = parts * all;
    const int64_t start = static_cast<int64_t>(blockIdx.x) * kThreads;
    const int row0 = static_cast<int>(start / row_threads), at0 = static_cast<int>(start - static_cast<int64_t>(row0) * row_threads) + static_cast<int>(threadIdx.x);
    const int64_t row = row0 + at0 / row_threads;
    const int at_row = at0 % row_threads, head = at_row / parts, part = at_row - head * parts;
    if (start + threadIdx.x >= p.total) return;
    const int b = static_cast<int>(row) / p.t;
    const uint4 *src = reinterpret_cast<const uint4 *>(p.qkv + (row * all + head) * p.head_dim + part * kRopeVec);
    const uint4 in0 = ld_stream(src), in1 = ld_stream(src + 1);
    const Place place = place_of(p.pos[static_cast<int>(row) % p.t], p.max_seq, p.table_rows);
    const int kv = head - p.heads, half = p.head_dim / 2, first = part * (kRopeVec / 2);
    if (!place.valid) {
        *p.status = 1;
        if (kv >= 0) return;
        bf16 *q = p.q_out + (row * p.heads + head) * p.head_dim;
        *reinterpret_cast<uint4 *>(q + first) = *reinterpret_cast<uint4 *>(q + half + first) = make_uint4(kNan2, kNan2, kNan2, kNan2);
        return;
    }
    const int64_t at = place.at, angle = place.angle;
    if (kv >= p.kv_heads) {      // v: as it is
        uint4 *dst = reinterpret_cast<uint4 *>(p.v_cache + ((static_cast<int64_t>(b) * p.kv_heads + kv - p.kv_heads) * p.max_seq + at) * p.head_dim + part * kRopeVec);
        dst[0] = in0;
        dst[1] = in1;
        return;
    }
    float c[8], s[8];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const float4 cv = __ldg(reinterpret_cast<const float4 *>(p.cos + angle * half + first) + i);
        const float4 sv = __ldg(reinterpret_cast<const float4 *>(p.sin + angle * half + first) + i);
        c[4 * i] = cv.x, c[4 * i + 1] = cv.y, c[4 * i + 2] = cv.z, c[4 * i + 3] = cv.w;
        s[4 * i] = sv.x, s[4 * i + 1] = sv.y, s[4 * i + 2] = sv.z, s[4 * i + 3] = sv.w;
    }
    const uint32_t w[8] = {in0.x, in0.y, in0.z, in0.w, in1.x, in1.y, in1.z, in1.w};
    float lo[8], hi[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float x1 = __uint_as_float(w[i] << 16), x2 = __uint_as_float(w[i] & 0xffff0000u);
        rotate(x1, x2, c[i], s[i], lo[i], hi[i]);
    }
    bf16 *dst = kv < 0 ? p.q_out + (row * p.heads + head) * p.head_dim
                       : p.k_cache + ((static_cast<int64_t>(b) * p.kv_heads + kv) * p.max_seq + at) * p.head_dim;
    *reinterpret_cast<uint4 *>(dst + first) = Elem<bf16>::pack(lo);
    *reinterpret_cast<uint4 *>(dst + half + first) = Elem<bf16>::pack(hi);
}

// in [rows, 2 * f]: w1's channels, then w3's.  A CTA takes V * kThreads 16-byte vectors of one row of the output.
template <int V>
__global__ void __launch_bounds__(kThreads) silu_mul_kernel(const uint4 *in, uint4 *out, int row_vecs, int chunks) {
    grid_dependency_sync();
    const int row = blockIdx.x / chunks, v0 = (blockIdx.x - row * chunks) * (V * kThreads) + threadIdx.x;
    const uint4 *src = in + static_cast<int64_t>(row) * 2 * row_vecs;
    uint4 a[V], b[V];
#pragma unroll
    for (int i = 0; i < V; ++i) {
        const int v = v0 + i * kThreads;
        if (v < row_vecs) a[i] = ld_stream(src + v), b[i] = ld_stream(src + row_vecs + v);
    }
#pragma unroll
    for (int i = 0; i < V; ++i) {
        const int v = v0 + i * kThreads;
        if (v >= row_vecs) break;
        float f[8];
        Elem<bf16>::unpack(a[i], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = silu(f[e]);
        out[static_cast<int64_t>(row) * row_vecs + v] = Elem<bf16>::mul(Elem<bf16>::pack(f), b[i]);
    }
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace
}  // namespace gpuk

using namespace gpuk;

extern "C" int gpuk_rope_append(const void *qkv, const float *cos, const float *sin, const int64_t *pos, void *q_out, void *k_cache, void *v_cache,
                                int batch, int t, int heads, int kv_heads, int head_dim, int table_rows, int max_seq, void *stream) {
    if (batch < 0 || t < 0 || heads <= 0 || kv_heads <= 0 || table_rows <= 0 || max_seq <= 0)
        return set_last_error(GPUK_ERR_INVALID_ARGUMENT, "rope_append: bad sizes");
    if (head_dim <= 0 || head_dim % kRopeVec) return set_last_error(GPUK_ERR_UNSUPPORTED, "rope_append: head_dim %d is not a multiple of %d", head_dim, kRopeVec);
    if (static_cast<int64_t>(batch) * t > 0x7fffffffll || (heads + 2ll * kv_heads) * (head_dim / kRopeVec) > 0x7fffffffll)
        return set_last_error(GPUK_ERR_UNSUPPORTED, "rope_append: too many rows or heads");
    if (batch == 0 || t == 0) return GPUK_OK;
    if (!qkv || !cos || !sin || !pos || !q_out || !k_cache || !v_cache) return set_last_error(GPUK_ERR_INVALID_ARGUMENT, "rope_append: null pointer");
    if (!aligned16(qkv) || !aligned16(cos) || !aligned16(sin) || !aligned16(q_out) || !aligned16(k_cache) || !aligned16(v_cache))
        return set_last_error(GPUK_ERR_INVALID_ARGUMENT, "rope_append: pointers must be 16-byte aligned");
    const DecodeDevice *d = nullptr;
    const int rc = decode_device(&d);
    if (rc != GPUK_OK) return rc;
    RopeParams p = {static_cast<const bf16 *>(qkv), cos, sin, pos, static_cast<bf16 *>(q_out), static_cast<bf16 *>(k_cache), static_cast<bf16 *>(v_cache),
                    static_cast<int64_t>(batch) * t * (heads + 2 * kv_heads) * (head_dim / kRopeVec), d->status + kStatusPosition, t, heads, kv_heads, head_dim, table_rows, max_seq};
    const int64_t grid = (p.total + kThreads - 1) / kThreads;
    if (grid > 0x7fffffffll) return set_last_error(GPUK_ERR_UNSUPPORTED, "rope_append: too many rows");
    void *args[] = {&p};
    cudaError_t e = launch_kernel(reinterpret_cast<const void *>(&rope_append_kernel), static_cast<int>(grid), kThreads, 1, false, args, static_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) return set_last_error(GPUK_ERR_CUDA, "rope_append: launch failed: %s", cudaGetErrorString(e));
    return GPUK_OK;
}

extern "C" int gpuk_silu_mul(const void *in, void *out, int64_t rows, int f, void *stream) {
    if (rows < 0 || f <= 0) return set_last_error(GPUK_ERR_INVALID_ARGUMENT, "silu_mul: bad sizes");
    if (f % 8) return set_last_error(GPUK_ERR_UNSUPPORTED, "silu_mul: %d channels are not a multiple of 8", f);
    if (rows > 0x7fffffffll) return set_last_error(GPUK_ERR_UNSUPPORTED, "silu_mul: too many rows");
    if (rows == 0) return GPUK_OK;
    if (!in || !out || !aligned16(in) || !aligned16(out)) return set_last_error(GPUK_ERR_INVALID_ARGUMENT, "silu_mul: pointers must be 16-byte aligned and not null");
    // two vectors a thread keep enough loads in flight; a batch of a few tokens is better spread over more CTAs (1184: eight for each of 148 SMs)
    int row_vecs = f / 8;
    const int v = rows * ((row_vecs + 2 * kThreads - 1) / (2 * kThreads)) >= 1184 ? 2 : 1;
    int chunks = (row_vecs + v * kThreads - 1) / (v * kThreads);
    const int64_t grid = rows * chunks;
    if (grid > 0x7fffffffll) return set_last_error(GPUK_ERR_UNSUPPORTED, "silu_mul: too many rows");
    void *args[] = {&in, &out, &row_vecs, &chunks};
    const void *fn = v == 2 ? reinterpret_cast<const void *>(&silu_mul_kernel<2>) : reinterpret_cast<const void *>(&silu_mul_kernel<1>);
    cudaError_t e = launch_kernel(fn, static_cast<int>(grid), kThreads, 1, false, args, static_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) return set_last_error(GPUK_ERR_CUDA, "silu_mul: launch failed: %s", cudaGetErrorString(e));
    return GPUK_OK;
}
