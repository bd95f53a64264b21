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
//     (kStages blocks of 4 KiB of keys and 4 KiB of values), so no warp waits for another before the end.  Two CTAs per SM keep
//     2 * 4 * (kStages - 1) * 8 KiB = 192 KiB in flight at most, several times what latency times bandwidth asks for.
//   * scores and outputs are mma.sync.m16n8k16 with the group's heads as the 16 rows (padded), keys / head dimension as columns:
//     the score fragment of a warp is, register for register, the operand of the second product.  A KV block of 16 keys
//     costs 32 mma and 16 ldmatrix against 8 KiB of loads; the tensor pipe is idle most of the time and does not matter.
//   * rows of 256 bytes would put the eight rows an ldmatrix reads into the same banks; 16-byte chunk c of row r lies at c ^ (r & 7).
//
// fp32 scores, running maximum and sums; probabilities are rounded to bf16 for the second product.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "../../include/gpuk_b200.h"
#include "launch.cuh"

namespace gpuk {
namespace {

using bf16 = __nv_bfloat16;
constexpr int kHeadDim = 128;
constexpr int kMaxGroup = 16;              // query heads per kv head: the rows of one mma
constexpr int kWarps = 4;
constexpr int kThreads = kWarps * 32;
constexpr int kBlockKeys = 16;             // keys a warp takes at a time
constexpr int kStages = 3;                 // ... and blocks of them in its ring
constexpr int kRowBytes = kHeadDim * 2;
constexpr int kTileBytes = kBlockKeys * kRowBytes;           // keys or values of one block
constexpr int kRingBytes = kWarps * kStages * 2 * kTileBytes;    // 96 KiB: two CTAs per SM
constexpr int kOutPitch = kHeadDim + 4;                      // floats per head in the partial outputs
static_assert((kWarps + 1) * kMaxGroup * kOutPitch * 4 <= kRingBytes, "the partial outputs reuse the ring");

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
// weight of a partial result whose maximum is m, relative to the overall maximum (0 where the part saw no key)
__device__ __forceinline__ float weight_of(float m, float overall) { return m == -INFINITY ? 0.f : exp2f(m - overall); }

__device__ __forceinline__ float ld_cluster(const float *local, int cta) {
    const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(local));
    uint32_t remote;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(a), "r"(cta));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
    return v;
}

__global__ void __launch_bounds__(kThreads, 2) decode_attention_kernel(const __grid_constant__ DecodeAttentionParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ PartialStats st;
    grid_dependency_sync();
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
    const uint32_t ring = static_cast<uint32_t>(__cvta_generic_to_shared(smem)) + warp * (kStages * 2 * kTileBytes);

    // one block: 16 rows of 256 bytes each for keys and values; a warp-wide copy covers two rows
    auto issue = [&](int i) {
        if (i < mine) {
            const uint32_t slot = ring + (i % kStages) * (2 * kTileBytes);
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
    for (int i = 0; i < kStages - 1; ++i) issue(i);

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
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};      // rows g and g + 8

    for (int i = 0; i < mine; ++i) {
        issue(i + kStages - 1);
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 1) : "memory");
        __syncwarp();
        const uint32_t ks = ring + (i % kStages) * (2 * kTileBytes), vs = ks + kTileBytes;
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
            mx[r] = fmaxf(mx[r], m[r]);            // finite: a block has at least one key
            fade[r] = exp2f(m[r] - mx[r]);         // 0 for the first block
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
        for (int w = 0; w < kWarps; ++w) ll += st.l[w][h] * weight_of(st.m[w][h], mm);
        st.m[kWarps][h] = mm, st.l[kWarps][h] = ll;
    }
    __syncthreads();
    float *sum = tiles + kWarps * kMaxGroup * kOutPitch;      // the CTA's own output, in units of its maximum
    for (int e = threadIdx.x; e < p.group * kHeadDim; e += kThreads) {
        const int h = e / kHeadDim, d = e % kHeadDim;
        float acc = 0.f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) acc += tiles[(w * kMaxGroup + h) * kOutPitch + d] * weight_of(st.m[w][h], st.m[kWarps][h]);
        sum[h * kOutPitch + d] = acc;
    }
    if (splits > 1) cluster_barrier();
    else __syncthreads();
    // each CTA of the cluster finishes an equal share of the group's outputs, parts taken in order
    bf16 *out = p.out + static_cast<int64_t>(pair) * p.group * kHeadDim;
    const int share = (p.group * kHeadDim + splits - 1) / splits, end = min((part + 1) * share, p.group * kHeadDim);
    for (int e = part * share + threadIdx.x; e < end; e += kThreads) {
        const int h = e / kHeadDim, d = e % kHeadDim;
        float acc, total;
        if (splits == 1) {
            acc = sum[h * kOutPitch + d], total = st.l[kWarps][h];
        } else {
            float pm[8], mm = -INFINITY;
            for (int s = 0; s < splits; ++s) mm = fmaxf(mm, pm[s] = ld_cluster(&st.m[kWarps][h], s));
            acc = total = 0.f;
            for (int s = 0; s < splits; ++s) {
                const float w = weight_of(pm[s], mm);
                acc += w * ld_cluster(sum + h * kOutPitch + d, s);
                total += w * ld_cluster(&st.l[kWarps][h], s);
            }
        }
        out[e] = __float2bfloat16_rn(acc / total);
    }
    if (splits > 1) cluster_barrier();      // nobody leaves while its partial results may still be read
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace
}  // namespace gpuk
