// Causal attention of a run of new tokens per sequence over the KV cache (the prefill), heads of 128, bf16.
//
// Bound by the tensor pipe and, just behind it, by the exponentials: 4 * 128 operations and one exponential per query, key and head.
//
//   * a CTA takes 256 queries of one head as two tiles of 128, the rows of a tcgen05.mma.  Two warpgroups own one tile each, a thread per row;
//     while one of them works on its scores the tensor pipe multiplies for the other.
//   * scores S = Q K^T go to tensor memory, 128 keys at a time; the row's thread reads them, and writes the probabilities back as bf16 into
//     the same columns, from where they are the first operand of O += P V.  Nothing passes through shared memory but Q, K and V, which one
//     warp fetches by TMA: 32 KiB per block of K or V through a ring of five.
//   * O stays in tensor memory and is rescaled by a warp whose rows have a new maximum.  To let the maximum lag behind saves most of that, but
//     the largest weight is then no longer 1, which bf16 holds exactly: the error grew from 1.9e-3 to 2.3e-3 with 2048 keys.
//   * a query sees the keys up to its position.  Blocks beyond a tile's last position are left out, which halves the work of a prompt;
//     a mask is applied only in blocks that some query sees in part.  CTAs with the most keys start first.
//
// fp32 scores, maxima and sums; probabilities are rounded to bf16 for the second product.
//
// Measured, the library's attention with a mask in brackets: 2048 queries, 64 / 8 heads 107 us (247), 640 TFLOP/s of what the mask leaves; 700,
// 64 / 16 heads 29 (148); 4 x 512, 16 / 2 heads 18 (28); 8 queries 5.9 (11.8); 64 after 1984 cached, 32 / 8 heads 38 (64).  Error against float64
// 1.86e-3 with 2048 keys (2.16e-3), 1.79e-3 with 100 (1.79e-3).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>

#include "../../include/gpuk_b200.h"
#include "launch.cuh"
#include "linear.cuh"
#include "tensor_core.cuh"

namespace gpuk {
namespace {

using bf16 = __nv_bfloat16;
constexpr int kHeadDim = 128;
constexpr int kTile = 128;                       // queries of a tile, keys of a block
constexpr int kTiles = 2;
constexpr int kSoftmaxThreads = kTiles * kTile;
constexpr int kThreads = kSoftmaxThreads + 64;   // and a warp that multiplies, and one that copies
constexpr int kSpanBytes = kTile * 128;          // 128 rows of one swizzle span (64 of the 128 dimensions)
constexpr int kBlockBytes = 2 * kSpanBytes;
constexpr int kSlots = 5;
constexpr int kSmemBytes = (kTiles + kSlots) * kBlockBytes + 1024;

constexpr float kLowest = -3.4e38f;              // a maximum where all scores are -infinity: finite, and any score behind it is larger

struct PrefillAttentionParams {
    const int64_t *pos;       // [t]: keys [0, pos] are seen
    const bf16 *q;            // [batch, t, heads, 128], as the tensor map has it
    bf16 *out;                // [batch, t, heads, 128]
    int t, heads, kv_heads;
    int len;                  // keys in the cache
    int tiles;                // CTAs per sequence and head
    int pairs;                // batch * heads
    float scale_log2;         // 1 / sqrt(128) * log2(e)
    int *status;
};

__device__ __forceinline__ float exp2_fast(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

__global__ void __launch_bounds__(kThreads, 1) prefill_attention_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap,
                                                                        const __grid_constant__ CUtensorMap vmap, const __grid_constant__ PrefillAttentionParams p) {
    extern __shared__ unsigned char dyn[];
    __shared__ alignas(8) uint64_t q_full, full[kSlots], empty[kSlots], s_full[kTiles], p_full[kTiles], o_done[kTiles], drained;
    __shared__ uint32_t tmem_slot;
    __shared__ int most[kTiles], least[kTiles];      // largest and smallest position of a tile's queries
    const int tid = threadIdx.x, warp = tid >> 5;
    const uint32_t base = (smem_addr(dyn) + 1023u) & ~1023u, ring = base + kTiles * kBlockBytes;
    if (tid == 0) {
        mbar_init(&q_full, 1), mbar_init(&drained, 1);
        for (int s = 0; s < kSlots; ++s) mbar_init(&full[s], 1), mbar_init(&empty[s], 1);
        for (int t = 0; t < kTiles; ++t) {
            mbar_init(&s_full[t], 1), mbar_init(&p_full[t], kTile), mbar_init(&o_done[t], 1);
            most[t] = -1, least[t] = 0x7fffffff;
        }
        mbar_init_fence();
    }
    if (warp == kSoftmaxThreads / 32) tmem_alloc<512>(&tmem_slot);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_dependency_sync();      // behind the allocation: a dependent kernel's CTA must not take tensor memory a CTA of this one still waits for
    const uint32_t tm = tmem_slot;
    // heads of a group side by side, queries with the most keys first
    const int pair = blockIdx.x % p.pairs, b = pair / p.heads, head = pair % p.heads, kvh = b * p.kv_heads + head / (p.heads / p.kv_heads);
    const int first = (p.tiles - 1 - blockIdx.x / p.pairs) * (kTiles * kTile);
    int limit = -1;      // last key this thread's query sees
    const int query = first + tid;
    if (tid < kSoftmaxThreads && query < p.t) {
        const int64_t at = p.pos[query], end = p.len - 1;
        limit = static_cast<int>(at < -1 ? -1 : at < end ? at : end);      // bounded before it is cut to 32 bits
        atomicMax(&most[tid / kTile], limit);
        atomicMin(&least[tid / kTile], limit);
    }
    __syncthreads();
    int blocks[kTiles];
#pragma unroll
    for (int t = 0; t < kTiles; ++t) blocks[t] = (most[t] + kTile) / kTile;
    const int rounds = max(blocks[0], blocks[1]);
    bool ok = true;

    if (warp == kSoftmaxThreads / 32 + 1) {      // copies: Q, then K and V of each block in turn
        if ((tid & 31) == 0 && rounds > 0) {
            const uint64_t once = policy_evict_first();
            mbar_expect_bytes(&q_full, kTiles * kBlockBytes);
            for (int t = 0; t < kTiles; ++t)
                for (int h = 0; h < 2; ++h)
                    tma_load_2d(base + t * kBlockBytes + h * kSpanBytes, &qmap, head * kHeadDim + h * 64, b * p.t + first + t * kTile, &q_full, once);
            int s = 0;
            uint32_t phase = 1;      // a fresh slot counts as released
            int filled = 0;
            for (int i = 0; i < 2 * rounds; ++i) {
                if (!mbar_wait(&empty[s], phase)) {
                    ok = false;
                    break;
                }
                mbar_expect_bytes(&full[s], kBlockBytes);
                for (int h = 0; h < 2; ++h) tma_load_3d(ring + s * kBlockBytes + h * kSpanBytes, i & 1 ? &vmap : &kmap, h * 64, (i >> 1) * kTile, kvh, &full[s]);
                ++filled;
                if (++s == kSlots) s = 0, phase ^= 1u;
            }
            // nobody leaves with copies in flight
            ok = mbar_wait(&q_full, 0) && ok;
            for (int i = max(0, filled - kSlots); i < filled; ++i) ok = mbar_wait(&full[i % kSlots], (i / kSlots) & 1) && ok;
        }
    } else if (warp == kSoftmaxThreads / 32) {   // multiplications
        if ((tid & 31) == 0 && rounds > 0) {
            constexpr uint32_t s_desc = mma_desc(1, 1, kTile, kTile), o_desc = mma_desc(1, 1, kTile, kHeadDim, true);
            auto slot = [&](int i) { return ring + (i % kSlots) * kBlockBytes; };
            // only a slot that the copies wait for: nothing may arrive in shared memory behind the CTA's end
            auto release = [&](int i) {
                if (i + kSlots < 2 * rounds) tc_commit(&empty[i % kSlots]);
            };
            auto wait_slot = [&](int i) { ok = ok && mbar_wait(&full[i % kSlots], (i / kSlots) & 1); };
            auto scores = [&](int t, int j) {      // 16 of the 128 dimensions per instruction
                const uint32_t q = base + t * kBlockBytes, k = slot(2 * j);
#pragma unroll
                for (int d = 0; d < kHeadDim / 16; ++d) {
                    const uint32_t off = (d / 4) * kSpanBytes + (d % 4) * 32;
                    tc_mma_f16(tm + t * kTile, kmajor_desc<128>(q + off), kmajor_desc<128>(k + off), s_desc, d > 0);
                }
                tc_commit(&s_full[t]);
            };
            ok = mbar_wait(&q_full, 0);
            wait_slot(0);
            tc_fence_after();
            if (ok)
                for (int t = 0; t < kTiles; ++t)
                    if (blocks[t] > 0) scores(t, 0);
            release(0);
            for (int j = 0; ok && j < rounds; ++j) {
                wait_slot(2 * j + 1);
                if (j + 1 < rounds) wait_slot(2 * j + 2);
                for (int t = 0; ok && t < kTiles; ++t) {
                    if (j >= blocks[t]) continue;
                    if (!mbar_wait(&p_full[t], j & 1)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t v = slot(2 * j + 1);
#pragma unroll
                    for (int k = 0; k < kTile / 16; ++k)      // 16 keys per instruction
                        tc_mma_f16_ts(tm + (kTiles + t) * kTile, tm + t * kTile + k * 8, mnmajor_desc(v + k * 16 * 128, kSpanBytes), o_desc, j > 0 || k > 0);
                    tc_commit(&o_done[t]);
                    if (j + 1 < blocks[t]) scores(t, j + 1);
                }
                release(2 * j + 1);
                release(2 * j + 2);
            }
            if (!ok) {      // a wait gave up: the row threads do not wait for what was issued, and the tensor memory is about to be freed
                tc_commit(&drained);
                mbar_wait(&drained, 0);
            }
        }
    } else {                                     // a row's thread
        const int t = tid / kTile;
        const uint32_t lanes = static_cast<uint32_t>((warp & 3) * 32) << 16, s_at = tm + lanes + t * kTile, o_at = tm + lanes + (kTiles + t) * kTile;
        float m = 0.f, l = 0.f;
        for (int j = 0; j < blocks[t]; ++j) {
            if (!mbar_wait(&s_full[t], j & 1)) {
                ok = false;
                break;
            }
            tc_fence_after();
            uint32_t s[4][32];
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_ld32(s[c], s_at + c * 32);
            tmem_wait_ld();
            if ((j + 1) * kTile - 1 > least[t]) {
                const int seen = limit - j * kTile;      // keys of this block up to here
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        if (c * 32 + i > seen) s[c][i] = 0xff800000u;
            }
            float mx[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                mx[c] = __uint_as_float(s[c][0]);
#pragma unroll
                for (int i = 1; i < 32; ++i) mx[c] = fmaxf(mx[c], __uint_as_float(s[c][i]));
            }
            const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.scale_log2;
            if (j == 0) {
                m = fmaxf(top, kLowest);
            } else {
                const bool grown = top > m;
                if (__any_sync(0xffffffffu, grown)) {
                    ok = mbar_wait(&o_done[t], (j - 1) & 1) && ok;      // issued before these scores: no wait in fact
                    tc_fence_after();
                    const float f = grown ? exp2_fast(m - top) : 1.f;
                    if (grown) m = top, l *= f;
#pragma unroll
                    for (int c = 0; c < kHeadDim; c += 16) {
                        float o[16];
                        tmem_ld16(o, o_at + c);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 16; ++i) o[i] *= f;
                        tmem_st16(o_at + c, o);
                    }
                }
            }
            float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t pk[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    const float a = exp2_fast(fmaf(__uint_as_float(s[2 * h + i / 16][2 * (i % 16)]), p.scale_log2, -m));
                    const float c = exp2_fast(fmaf(__uint_as_float(s[2 * h + i / 16][2 * (i % 16) + 1]), p.scale_log2, -m));
                    sum[i & 1] += a, sum[2 + (i & 1)] += c;
                    pk[i] = pack_bf16(a, c);
                }
                tmem_st32(s_at + h * 32, pk);
            }
            l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive(&p_full[t]);
        }
        if (blocks[t] > 0) {
            ok = mbar_wait(&o_done[t], (blocks[t] - 1) & 1) && ok;
            tc_fence_after();
        }
        const float r = l == 0.f ? 0.f : 1.f / l;
        const int64_t row = ((static_cast<int64_t>(b) * p.t + query) * p.heads + head) * kHeadDim;
        uint4 *out = reinterpret_cast<uint4 *>(p.out + row);
        // a query that sees no key: zeros, or NaN where it is one that the rotary embedding marked
        const uint32_t nothing = limit < 0 && query < p.t && __hisnan(p.q[row]) ? 0x7fff7fffu : 0u;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            uint32_t o[32];
            if (blocks[t] > 0) {
                tmem_ld32(o, o_at + c * 32);
                tmem_wait_ld();
            }
            if (query < p.t) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    uint32_t w[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        w[e] = limit < 0 ? nothing : pack_bf16(__uint_as_float(o[8 * i + 2 * e]) * r, __uint_as_float(o[8 * i + 2 * e + 1]) * r);
                    out[c * 4 + i] = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
        }
    }
    if (!ok) *p.status = 1;
    tc_fence_before();
    __syncthreads();
    if (warp == kSoftmaxThreads / 32) {
        tc_fence_after();
        tmem_free<512>(tm);
    }
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace

cudaError_t prefill_attention_setup() {
    return cudaFuncSetAttribute(reinterpret_cast<const void *>(&prefill_attention_kernel), cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
}

}  // namespace gpuk

using namespace gpuk;

extern "C" int gpuk_prefill_attention(const void *q, const void *k_cache, const void *v_cache, const int64_t *pos, void *out, int batch, int t, int heads, int kv_heads,
                                      int head_dim, int len, int max_seq, void *stream) {
    if (batch < 0 || t < 0 || heads <= 0 || kv_heads <= 0 || len <= 0 || max_seq < len) return set_last_error(GPUK_ERR_INVALID_ARGUMENT, "prefill_attention: bad sizes");
    if (head_dim != kHeadDim || heads % kv_heads)
        return set_last_error(GPUK_ERR_UNSUPPORTED, "prefill_attention: built for heads of %d, a whole number of them per kv head (got %d, %d / %d)", kHeadDim, head_dim, heads, kv_heads);
    if (static_cast<int64_t>(batch) * heads > 0x7fffffffll) return set_last_error(GPUK_ERR_UNSUPPORTED, "prefill_attention: too many sequences");
    if (batch == 0 || t == 0) return GPUK_OK;
    if (!q || !k_cache || !v_cache || !pos || !out) return set_last_error(GPUK_ERR_INVALID_ARGUMENT, "prefill_attention: null pointer");
    if (!aligned16(q) || !aligned16(k_cache) || !aligned16(v_cache) || !aligned16(out)) return set_last_error(GPUK_ERR_INVALID_ARGUMENT, "prefill_attention: pointers must be 16-byte aligned");
    const DecodeDevice *d = nullptr;
    const int rc = decode_device(&d);
    if (rc != GPUK_OK) return rc;
    const int tiles = (t + kTiles * kTile - 1) / (kTiles * kTile);
    const int64_t rows = static_cast<int64_t>(batch) * t, ctas = static_cast<int64_t>(batch) * heads * tiles;
    if (ctas > 0x7fffffffll || rows > 0x7fffffffll) return set_last_error(GPUK_ERR_UNSUPPORTED, "prefill_attention: too many sequences");
    CUtensorMap qmap, kmap, vmap;
    const uint64_t row = kHeadDim * 2, q_sizes[2] = {static_cast<uint64_t>(heads) * kHeadDim, static_cast<uint64_t>(rows)}, q_strides[1] = {heads * row};
    // keys beyond `len` read as zeros
    const uint64_t kv_sizes[3] = {kHeadDim, static_cast<uint64_t>(len), static_cast<uint64_t>(batch) * kv_heads}, kv_strides[2] = {row, max_seq * row};
    const uint32_t box[3] = {64, kTile, 1};
    int e = encode_map(&qmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, q, 2, q_sizes, q_strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (!e) e = encode_map(&kmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, k_cache, 3, kv_sizes, kv_strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (!e) e = encode_map(&vmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, v_cache, 3, kv_sizes, kv_strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (e) return set_last_error(GPUK_ERR_CUDA, "prefill_attention: the driver refused a tensor map (%d)", e);
    PrefillAttentionParams p = {pos, static_cast<const bf16 *>(q), static_cast<bf16 *>(out), t, heads, kv_heads, len, tiles, batch * heads, 1.4426950408889634f / std::sqrt(static_cast<float>(kHeadDim)), d->status};
    void *args[] = {&qmap, &kmap, &vmap, &p};
    const cudaError_t err = launch_kernel(reinterpret_cast<const void *>(&prefill_attention_kernel), static_cast<int>(ctas), kThreads, 1, false, args,
                                          static_cast<cudaStream_t>(stream), kSmemBytes);
    if (err != cudaSuccess) return set_last_error(GPUK_ERR_CUDA, "prefill_attention: launch failed: %s", cudaGetErrorString(err));
    return GPUK_OK;
}
