// Attention of one new token per sequence over the KV cache (the decode step).
//
// Bound by HBM: every cached key and value is read once and used for the `group` query heads that share it (4 to 16),
// a handful of operations a byte.  So the kernel is built around keeping loads in flight:
//
//   * one CTA works on one (sequence, kv head) and a range of its keys, for all query heads of the group at once -- the cache
//     is read once, not once per query head.  Where there are fewer such pairs than the GPU holds CTAs, the keys are split over a
//     thread-block cluster, whose CTAs combine their partial results through distributed shared memory: no workspace,
//     no second kernel.
//   * a warp owns every fourth block of 16 keys of the range and fetches it by cp.async into a ring of its own
//     (4 KiB of keys and 4 KiB of values per block), so no warp waits for another before the end.  Three blocks deep, two CTAs per SM; six deep
//     where all CTAs run at once with one per SM, so that an SM keeps 128 to 160 KiB in flight either way.  The first blocks are brought into L2
//     before griddepcontrol.wait.
//   * scores and outputs are mma.sync.m16n8k16 with the group's heads as the 16 rows (padded), keys / head dimension as columns:
//     the score fragment of a warp is, register for register, the operand of the second product.  A KV block of 16 keys
//     costs 32 mma and 16 ldmatrix against 8 KiB of loads; the tensor pipe is idle most of the time and does not matter.
//   * rows of 256 bytes would put the eight rows an ldmatrix reads into the same banks; 16-byte chunk c of row r lies at c ^ (r & 7).
//
// fp32 scores, running maximum and sums; probabilities are rounded to bf16 for the second product.
//
// Measured, 64 / 8 heads, the library's attention in brackets: 32 sequences x 2049 keys 42.5 us (49.7), 6.3 TB/s; 32 x 300 8.5 (10.7); 7 x 2049 of
// 32 / 8 heads 12.7 (13.4); 4 x 129 of 16 / 4 heads 3.2 (5.3).  Behind it: 7 x 1000 9.2 (8.6), 12 x 1000 12.2 (11.0), 1 x 8192 14.0 (12.0), 1 x 8192 of 8 / 1 heads 12.2 (8.6); its
// call takes 25 us more on the host.  Error against float64 1.65e-3 to 1.79e-3 (1.73e-3 to 1.89e-3).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>

#include "../../include/gpuk_b200.h"
#include "launch.cuh"
#include "linear.cuh"

namespace gpuk {
namespace {

using bf16 = __nv_bfloat16;
constexpr int kHeadDim = 128;
constexpr int kMaxGroup = 16;              // query heads per kv head: the rows of one mma
constexpr int kWarps = 4;
constexpr int kThreads = kWarps * 32;
constexpr int kBlockKeys = 16;             // keys a warp takes at a time
constexpr int kStages = 3, kDeepStages = 6;    // ... and blocks of them in its ring: two CTAs per SM, or one
constexpr int kRowBytes = kHeadDim * 2;
constexpr int kTileBytes = kBlockKeys * kRowBytes;           // keys or values of one block
constexpr int ring_bytes(int stages) { return kWarps * stages * 2 * kTileBytes; }      // 96 or 192 KiB
constexpr int kOutPitch = kHeadDim + 4;                      // floats per head in the partial outputs
static_assert((kWarps + 1) * kMaxGroup * kOutPitch * 4 <= ring_bytes(kStages), "the partial outputs reuse the ring");

struct DecodeAttentionParams {
    const bf16 *q;            // [batch, heads, 128]
    const bf16 *k, *v;        // [batch, kv_heads, max_seq, 128]
    bf16 *out;                // [batch, heads, 128]
    int kv_heads, group;      // heads = kv_heads * group
    int len, max_seq;         // keys [0, len) are attended to
    int splits;               // CTAs of the cluster that share a (sequence, kv head)
    float scale_log2;         // 1 / sqrt(128) * log2(e): scores in units of powers of two
    int *status;
};

struct PartialStats {
    float m[kWarps + 1][kMaxGroup], l[kWarps + 1][kMaxGroup];      // per warp, then of the CTA
    float w[kWarps][kMaxGroup];                                    // weight of a warp's partial output in the CTA's
};

__device__ __forceinline__ uint32_t swizzled(int row, int chunk) { return row * kRowBytes + ((chunk ^ (row & 7)) << 4); }

__device__ __forceinline__ void cp_async16_zfill(uint32_t smem, const void *gmem, bool valid) {
    const int bytes = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&r)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
// A maximum starts below every finite score and stays finite where all scores are -infinity, so that no difference of two is undefined: scores of
// -infinity weigh nothing beside others, and a part that saw no key, or only such, weighs nothing.
constexpr float kLowest = -3.4e38f;
__device__ __forceinline__ float weight_of(float m, float overall) { return exp2f(m - overall); }

__device__ __forceinline__ float ld_cluster(const float *local, int cta) {
    const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(local));
    uint32_t remote;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(a), "r"(cta));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
    return v;
}

__device__ __forceinline__ float4 ld_cluster4(const float *local, int cta) {
    const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(local));
    uint32_t remote;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(a), "r"(cta));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
    return v;
}

template <int STAGES>
__global__ void __launch_bounds__(kThreads, STAGES == kStages ? 2 : 1) decode_attention_kernel(const __grid_constant__ DecodeAttentionParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ PartialStats st;
    const int splits = cluster_size(), part = cluster_cta_rank();
    if (splits != p.splits) {      // the key ranges were cut for the planned cluster
        if (threadIdx.x == 0) *p.status = 1;
        return;
    }
    const int pair = blockIdx.x / splits, b = pair / p.kv_heads, kvh = pair % p.kv_heads;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int per = (p.len + splits - 1) / splits;
    const int lo = min(part * per, p.len), hi = min(lo + per, p.len);
    const int blocks = (hi - lo + kBlockKeys - 1) / kBlockKeys;
    const int mine = warp < blocks ? (blocks - warp + kWarps - 1) / kWarps : 0;      // this warp's blocks: warp, warp + 4, ...

    const bf16 *kbase = p.k + static_cast<int64_t>(pair) * p.max_seq * kHeadDim;
    const bf16 *vbase = p.v + static_cast<int64_t>(pair) * p.max_seq * kHeadDim;
    const uint32_t ring = static_cast<uint32_t>(__cvta_generic_to_shared(smem)) + warp * (STAGES * 2 * kTileBytes);

    // what the ring will take first comes into L2 while the kernel in front of this one ends: a hint, read only after the wait
    for (int i = 0; i < min(STAGES - 1, mine); ++i) {
        const int row = lo + (warp + i * kWarps) * kBlockKeys + (lane & 15);
        if (row < hi) {
            const bf16 *src = (lane < 16 ? kbase : vbase) + static_cast<int64_t>(row) * kHeadDim;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(src));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(src + kHeadDim / 2));
        }
    }
    grid_dependency_sync();

    // one block: 16 rows of 256 bytes each for keys and values; a warp-wide copy covers two rows
    auto issue = [&](int i) {
        if (i < mine) {
            const uint32_t slot = ring + (i % STAGES) * (2 * kTileBytes);
            const int row0 = lo + (warp + i * kWarps) * kBlockKeys;
#pragma unroll
            for (int j = 0; j < kBlockKeys / 2; ++j) {
                const int r = 2 * j + (lane >> 4), c = lane & 15, row = row0 + r;
                const bool valid = row < hi;
                const int64_t off = static_cast<int64_t>(valid ? row : lo) * kHeadDim + c * 8;
                cp_async16_zfill(slot + swizzled(r, c), kbase + off, valid);
                cp_async16_zfill(slot + kTileBytes + swizzled(r, c), vbase + off, valid);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");      // an empty group past the end keeps the count uniform
    };
#pragma unroll
    for (int i = 0; i < STAGES - 1; ++i) issue(i);

    // the group's query heads as the rows of the first operand, zero rows beyond them
    uint32_t qa[kHeadDim / 16][4];
    const bf16 *qbase = p.q + static_cast<int64_t>(pair) * p.group * kHeadDim;
#pragma unroll
    for (int s = 0; s < kHeadDim / 16; ++s)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int row = g + (r & 1) * 8, col = s * 16 + 2 * t + (r >> 1) * 8;
            qa[s][r] = row < p.group ? *reinterpret_cast<const uint32_t *>(qbase + row * kHeadDim + col) : 0u;
        }

    float o[kHeadDim / 8][4];
#pragma unroll
    for (int j = 0; j < kHeadDim / 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[j][e] = 0.f;
    float m[2] = {kLowest, kLowest}, l[2] = {0.f, 0.f};      // rows g and g + 8

    for (int i = 0; i < mine; ++i) {
        issue(i + STAGES - 1);
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 1) : "memory");
        __syncwarp();
        const uint32_t ks = ring + (i % STAGES) * (2 * kTileBytes), vs = ks + kTileBytes;
        float sc[2][4] = {};
        const int mi = lane >> 3, mr = lane & 7;      // which of the four 8x8 matrices this lane addresses, and its row
#pragma unroll
        for (int s = 0; s < kHeadDim / 16; ++s) {
            uint32_t kb[4];      // keys 0-7 | 8-15, dimensions 0-7 | 8-15 of this step
            ldmatrix4(kb, ks + swizzled((mi >> 1) * 8 + mr, 2 * s + (mi & 1)));
            mma_bf16(sc[0], qa[s], kb[0], kb[1]);
            mma_bf16(sc[1], qa[s], kb[2], kb[3]);
        }
        const int row0 = lo + (warp + i * kWarps) * kBlockKeys;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int key = row0 + h * 8 + 2 * t + (e & 1);
                sc[h][e] = key < hi ? sc[h][e] * p.scale_log2 : -INFINITY;
            }
        float mx[2], fade[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            mx[r] = fmaxf(fmaxf(sc[0][2 * r], sc[0][2 * r + 1]), fmaxf(sc[1][2 * r], sc[1][2 * r + 1]));
            mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
            mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
            mx[r] = fmaxf(mx[r], m[r]);
            fade[r] = exp2f(m[r] - mx[r]);         // 0 for the first block with a finite score
        }
        if (__any_sync(0xffffffffu, mx[0] != m[0] || mx[1] != m[1])) {
#pragma unroll
            for (int j = 0; j < kHeadDim / 8; ++j) {
                o[j][0] *= fade[0], o[j][1] *= fade[0];
                o[j][2] *= fade[1], o[j][3] *= fade[1];
            }
            l[0] *= fade[0], l[1] *= fade[1];
            m[0] = mx[0], m[1] = mx[1];
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int e = 0; e < 4; ++e) sc[h][e] = exp2f(sc[h][e] - m[e >> 1]);
        l[0] += (sc[0][0] + sc[0][1]) + (sc[1][0] + sc[1][1]);
        l[1] += (sc[0][2] + sc[0][3]) + (sc[1][2] + sc[1][3]);
        const uint32_t pa[4] = {pack_bf16(sc[0][0], sc[0][1]), pack_bf16(sc[0][2], sc[0][3]), pack_bf16(sc[1][0], sc[1][1]), pack_bf16(sc[1][2], sc[1][3])};
#pragma unroll
        for (int j = 0; j < kHeadDim / 16; ++j) {
            uint32_t vb[4];      // keys 0-7 | 8-15 of dimensions 0-7, then of dimensions 8-15
            ldmatrix4_trans(vb, vs + swizzled((mi & 1) * 8 + mr, 2 * j + (mi >> 1)));
            mma_bf16(o[2 * j], pa, vb[0], vb[1]);
            mma_bf16(o[2 * j + 1], pa, vb[2], vb[3]);
        }
        __syncwarp();      // the next issue refills the slot of the block before this one: every lane is past it
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
        if (t == 0) st.m[warp][g + 8 * r] = m[r], st.l[warp][g + 8 * r] = l[r];
    }
    __syncthreads();      // all warps are done with the ring: it takes the partial outputs, one [16][kOutPitch] tile per warp
    float *tiles = reinterpret_cast<float *>(smem);
#pragma unroll
    for (int j = 0; j < kHeadDim / 8; ++j)
#pragma unroll
        for (int r = 0; r < 2; ++r)
            if (g + 8 * r < p.group)
                *reinterpret_cast<float2 *>(tiles + (warp * kMaxGroup + g + 8 * r) * kOutPitch + j * 8 + 2 * t) = make_float2(o[j][2 * r], o[j][2 * r + 1]);
    if (threadIdx.x < kMaxGroup) {      // the CTA's maximum and sum of each head
        const int h = threadIdx.x;
        float mm = st.m[0][h], ll = 0.f;
#pragma unroll
        for (int w = 1; w < kWarps; ++w) mm = fmaxf(mm, st.m[w][h]);
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            st.w[w][h] = weight_of(st.m[w][h], mm);
            ll += st.l[w][h] * st.w[w][h];
        }
        st.m[kWarps][h] = mm, st.l[kWarps][h] = ll;
    }
    __syncthreads();
    // four outputs a thread: the CTA's own sum, in units of its maximum
    float *sum = tiles + kWarps * kMaxGroup * kOutPitch;
    constexpr int quads = kHeadDim / 4;
    bf16 *out = p.out + static_cast<int64_t>(pair) * p.group * kHeadDim;
    auto store = [&](int h, int d, float4 v, float total) {
        const float r = 1.f / total;
        *reinterpret_cast<uint2 *>(out + h * kHeadDim + d) = make_uint2(pack_bf16(v.x * r, v.y * r), pack_bf16(v.z * r, v.w * r));
    };
    for (int e = threadIdx.x; e < p.group * quads; e += kThreads) {
        const int h = e / quads, d = e % quads * 4;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const float4 t4 = *reinterpret_cast<const float4 *>(tiles + (w * kMaxGroup + h) * kOutPitch + d);
            const float f = st.w[w][h];
            acc.x += f * t4.x, acc.y += f * t4.y, acc.z += f * t4.z, acc.w += f * t4.w;
        }
        if (splits == 1) store(h, d, acc, st.l[kWarps][h]);
        else *reinterpret_cast<float4 *>(sum + h * kOutPitch + d) = acc;
    }
    if (splits == 1) return;
    cluster_barrier();
    // the group's outputs are dealt out over the cluster; parts are summed in order
    for (int e = part * kThreads + threadIdx.x; e < p.group * quads; e += splits * kThreads) {
        const int h = e / quads, d = e % quads * 4;
        float pm[8], pl[8];
        float4 ps[8];
#pragma unroll
        for (int s = 0; s < 8; ++s)
            if (s < splits) {
                pm[s] = ld_cluster(&st.m[kWarps][h], s);
                pl[s] = ld_cluster(&st.l[kWarps][h], s);
                ps[s] = ld_cluster4(sum + h * kOutPitch + d, s);
            }
        float mm = kLowest, total = 0.f;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int s = 0; s < 8; ++s)
            if (s < splits) mm = fmaxf(mm, pm[s]);
#pragma unroll
        for (int s = 0; s < 8; ++s)
            if (s < splits) {
                const float w = weight_of(pm[s], mm);
                acc.x += w * ps[s].x, acc.y += w * ps[s].y, acc.z += w * ps[s].z, acc.w += w * ps[s].w;
                total += w * pl[s];
            }
        store(h, d, acc, total);
    }
    cluster_barrier();      // nobody leaves while its partial results may still be read
}

const void *kernel_of(bool deep) {
    return deep ? reinterpret_cast<const void *>(&decode_attention_kernel<kDeepStages>) : reinterpret_cast<const void *>(&decode_attention_kernel<kStages>);
}
int stages_of(bool deep) { return deep ? kDeepStages : kStages; }

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace

cudaError_t decode_attention_setup(DecodeDevice *d) {
    cudaError_t e = cudaSuccess;
    for (int deep = 0; deep < 2 && e == cudaSuccess; ++deep) {
        e = cudaFuncSetAttribute(kernel_of(deep), cudaFuncAttributeMaxDynamicSharedMemorySize, ring_bytes(stages_of(deep)));
        for (int splits = 1; splits <= 8 && e == cudaSuccess; ++splits) {
            int64_t ctas = 0;
            e = resident_ctas(kernel_of(deep), kThreads, splits, d->sms, &ctas, ring_bytes(stages_of(deep)));
            d->attention_ctas[deep][splits] = static_cast<int>(ctas);
        }
    }
    return e;
}

}  // namespace gpuk

using namespace gpuk;

extern "C" int gpuk_decode_attention(const void *q, const void *k_cache, const void *v_cache, void *out, int batch, int heads, int kv_heads, int head_dim,
                                     int len, int max_seq, int splits, void *stream) {
    if (batch < 0 || heads <= 0 || kv_heads <= 0 || len <= 0 || max_seq < len) return set_last_error(GPUK_ERR_INVALID_ARGUMENT, "decode_attention: bad sizes");
    if (head_dim != kHeadDim || heads % kv_heads || heads / kv_heads > kMaxGroup)
        return set_last_error(GPUK_ERR_UNSUPPORTED, "decode_attention: built for heads of %d and at most %d query heads per kv head (got %d, %d / %d)", kHeadDim, kMaxGroup,
                              head_dim, heads, kv_heads);
    if (splits < 0 || splits > 8) return set_last_error(GPUK_ERR_INVALID_ARGUMENT, "decode_attention: splits must be 0 to 8");
    if (batch == 0) return GPUK_OK;
    if (!q || !k_cache || !v_cache || !out) return set_last_error(GPUK_ERR_INVALID_ARGUMENT, "decode_attention: null pointer");
    if (!aligned16(q) || !aligned16(k_cache) || !aligned16(v_cache) || (reinterpret_cast<uintptr_t>(out) & 7u)) return set_last_error(GPUK_ERR_INVALID_ARGUMENT, "decode_attention: pointers must be 16-byte aligned (out: 8)");
    const DecodeDevice *d = nullptr;
    const int rc = decode_device(&d);
    if (rc != GPUK_OK) return rc;
    const int64_t pairs = static_cast<int64_t>(batch) * kv_heads;
    // A cluster of parts costs about a microsecond and, from the second CTA an SM on, the overlap with the launch in front, so a part needs its keys: more than 160 in each half while
    // every CTA has an SM to itself (4 x 129 keys, 4 kv heads: 1 part 3.2 us, 2 3.6; 32 x 300, 1: 2 parts 4.8, 8 5.8), 384 beyond (7 x 300, 8: 1 part 5.0, 4 6.3; 7 x 1000: 2 parts
    // 10.2, 4 9.3), and all clusters have to run at once (2 x 2049, 8 kv heads, 8 parts: with the long ring, for which the
    // 16 clusters do not fit, 13.6 us, with the short one 8.4).
    if (splits == 0) {
        splits = 1;
        while (splits < 8 && len > (pairs * splits * 2 <= d->sms ? 160 : 384) * splits && pairs * splits * 2 <= d->attention_ctas[0][splits * 2]) splits *= 2;
    }
    if (pairs * splits > 0x7fffffffll) return set_last_error(GPUK_ERR_UNSUPPORTED, "decode_attention: too many sequences");
    DecodeAttentionParams p = {static_cast<const bf16 *>(q), static_cast<const bf16 *>(k_cache), static_cast<const bf16 *>(v_cache), static_cast<bf16 *>(out),
                               kv_heads, heads / kv_heads, len, max_seq, splits, 1.4426950408889634f / std::sqrt(static_cast<float>(kHeadDim)), d->status};
    void *args[] = {&p};
    const bool deep = pairs * splits <= d->attention_ctas[1][splits] && len > splits * kWarps * kBlockKeys * 2;
    const cudaError_t e = launch_kernel(kernel_of(deep), static_cast<int>(pairs) * splits, kThreads, splits, false, args, static_cast<cudaStream_t>(stream),
                                        ring_bytes(stages_of(deep)));
    if (e != cudaSuccess) return set_last_error(GPUK_ERR_CUDA, "decode_attention: launch failed: %s", cudaGetErrorString(e));
    return GPUK_OK;
}
