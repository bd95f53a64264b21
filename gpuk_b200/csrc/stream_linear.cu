// Linear layers of a decode batch (at most 32 tokens): y = x . w^T with the weights streamed once from HBM, in FP8 with
// row-wise scales (gpuk_fp8_linear_skinny) or in bf16 (gpuk_linear_skinny).
//
// Bound by the weights' bytes.  What the multiplication may cost beside the loads decides the design: warp-level FP8 mma has no
// native path on sm_100 (its conversions and HMMAs bound the kernel at 3 TB/s with 32 tokens), so the weights go straight
// from shared memory into tcgen05.mma, which one thread issues:
//
//   * a tile is 128 output channels = the 128 rows of one tcgen05.mma; the tokens are its 16 or 32 columns.  The accumulators
//     (below) take four times as many columns of tensor memory.
//   * a pipeline step is 128 bytes of k: 16 KiB of weights and 2 or 4 KiB of activations, fetched by one TMA copy each into a ring.
//     Two or three CTAs per SM with rings of four to six steps keep 160 to 192 KiB of weights in flight per SM, several times what latency
//     times bandwidth asks for, so that one CTA's start and end hide behind the other's stream.
//   * where there are fewer tiles than CTAs fit, k is split over a thread-block cluster whose CTAs sum their partial tiles through
//     distributed shared memory in CTA order (deterministic, no atomics, no workspace).
//   * the weights the ring takes first are brought into L2 before griddepcontrol.wait, while the kernel in front still runs (32 tokens,
//     57344 x 8192: 79.3 -> 76.0 us, 10240 x 8192: 18.0 -> 16.7 us, launches back to back).
//   * steps take turns with four accumulators, which the epilogue adds: shorter chains of rounded sums, so that a part of k that is four
//     times as long costs no precision (outputs that miss the nearest bf16, 32 tokens, 7168 x 8192: 8e-5; one accumulator 1e-4 to 2e-4).
//   * row-major weights arrive as rows of 128 bytes, swizzled over 128.  Weights in blocked order (gpuk_fp8_pack_weight: 16 rows x 64
//     bytes per KiB) are fetched as rows of 128 bytes too, i.e. two matrix rows at once -- half the requests of 64-byte rows, 79 instead of 82 us at
//     57344 x 8192.  Swizzled over 128 bytes they form the operand layout of 64-byte rows swizzled over 64, except that each
//     pair of rows in the second half of a band of 16 has changed places; the epilogue undoes that.  Either way
//     an instruction multiplies the same 32 bytes of k, so both layouts give the same bits.
//
// The elementwise step that follows a projection in a decoder layer can be its epilogue: a tile is then 64 channels of w1 and the same 64 of w3, or
// one head of q|k|v.  That saves two launches of 2.3 us a layer and the round trip of their inputs: decode step of four layers, 32 sequences, 1079 -> 1060
// us; of two small layers, 4 sequences, 121 -> 112 us.
//
// Measured, 32 tokens, FP8: 57344 x 8192 75 us (6.3 TB/s; the warp-level kernel 136, the library GEMM 89), 10240 x 8192 16.6 (39, 20.7), 7168 x 8192 13.2
// (21.7, 17.3), 4096 x 8192 10.1 (13.5, 15.8).  bf16, the library in brackets: 32 tokens, 8192 x 8192 22.7 us (24.8), 8192 x 28672 71.8 (71.2), 22528 x 4096 33.7
// (32.4), 1024 x 8192 9.3 (15.2), 3072 x 2048 7.1 (5.9); 4 tokens, 2048 x 4096 7.3 (12.9), 3072 x 2048 6.0 (7.5), 8192 x 2048 9.0 (8.2), 8192 x 3584 12.1 (11.4).  Below 30 MB
// what is left is a fixed 3 us of start and end; there the library is ahead by up to a microsecond and a half for 8192 channels, and for 17 tokens and more.  A
// call of it takes 4 us more on the host, and an epilogue here saves a launch.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "../../include/gpuk_b200.h"
#include "decoder_math.cuh"
#include "launch.cuh"
#include "linear.cuh"
#include "tensor_core.cuh"

namespace gpuk {
namespace {

using bf16 = __nv_bfloat16;
constexpr int kTileRows = 128;           // output channels per cluster: the rows of one tcgen05.mma
constexpr int kThreads = 128;            // warp 0 issues copies, warp 1 multiplications, all four finish the tile
constexpr int kStep = 128;               // bytes of k per pipeline step
constexpr int kWBytes = kTileRows * kStep;
constexpr int kAcc = 4;                  // accumulators the steps take turns with: shorter chains of rounded sums
constexpr int kRingMax = 6;              // steps of the deepest ring
constexpr int kPitch = kTileRows + 4;    // floats per token in the partial tile
constexpr int kMaxTokens = 32;

enum Weights { kFp8Blocked, kFp8Rows, kBf16Rows };

struct StreamParams {
    const float *x_scale, *w_scale;      // FP8: [m], [n]
    bf16 *out;                           // [m, n]
    int m, n;
    int steps;                           // pipeline steps of the whole k
    int stages;                          // depth of the ring
    int ks;                              // CTAs per cluster = parts the steps are split into (planned; checked in the kernel)
    int vec;                             // 1: out and w_scale are aligned for four channels at a time
    RopeCall rope;
    int *status;                         // set to 1 when a launch did not carry the planned cluster or a wait gave up; [kStatusPosition]: see place_of
};

template <int N>
__host__ __device__ constexpr int stage_bytes() { return kWBytes + N * kStep; }
constexpr int smem_bytes(int columns, int stages) { return stages * (kWBytes + columns * kStep) + 1024; }      // 1024: the ring starts on a swizzle boundary

__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t local, int cta) {
    uint32_t remote;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(cta));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
    return v;
}

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&v);
}
__device__ __forceinline__ float rounded(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

template <int W, int N, int EPI>
__global__ void __launch_bounds__(kThreads, 2) stream_linear_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap,
                                                                    const __grid_constant__ StreamParams p) {
    constexpr int kTmemCols = kAcc * N;
    extern __shared__ unsigned char dyn[];
    __shared__ alignas(8) uint64_t full[kRingMax], empty[kRingMax], done;
    __shared__ uint32_t tmem_slot;
    const int ks = cluster_size(), part = cluster_cta_rank();
    if (ks != p.ks) {
        if (threadIdx.x == 0) *p.status = 1;
        return;
    }
    const int tid = threadIdx.x, warp = tid >> 5, tile = blockIdx.x / ks;
    const uint32_t ring = (smem_addr(dyn) + 1023u) & ~1023u;
    if (tid == 0) {
        prefetch_map(&wmap);
        prefetch_map(&xmap);
        for (int s = 0; s < p.stages; ++s) mbar_init(&full[s], 1), mbar_init(&empty[s], 1);
        mbar_init(&done, 1);
        mbar_init_fence();
    }
    if (warp == 1) tmem_alloc<kTmemCols>(&tmem_slot);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t acc = tmem_slot;
    // this CTA's share of the steps: contiguous, the first `extra` parts take one more
    const int base = p.steps / ks, extra = p.steps % ks;
    const int begin = part * base + min(part, extra), nsteps = base + (part < extra ? 1 : 0);
    bool ok = true;
    if (tid == 0) {
        const uint64_t once = policy_evict_first(), keep = policy_evict_last();
        auto load_w = [&](int i, int s) {
            const uint32_t w = ring + s * stage_bytes<N>();
            mbar_expect_bytes(&full[s], stage_bytes<N>());
            if (W == kFp8Blocked) tma_load_4d(w, &wmap, 0, 0, tile * (kTileRows / 16), (begin + i) * 2, &full[s], once);
            else if (EPI == kSwiGlu) {      // 64 channels of either half
                for (int h = 0; h < 2; ++h)
                    tma_load_2d(w + h * (kWBytes / 2), &wmap, (begin + i) * (W == kBf16Rows ? kStep / 2 : kStep), h * (p.n / 2) + tile * (kTileRows / 2), &full[s], once);
            } else tma_load_2d(w, &wmap, (begin + i) * (W == kBf16Rows ? kStep / 2 : kStep), tile * kTileRows, &full[s], once);
        };
        auto load_x = [&](int i, int s) {
            tma_load_2d(ring + s * stage_bytes<N>() + kWBytes, &xmap, (begin + i) * (W == kBf16Rows ? kStep / 2 : kStep), 0, &full[s], keep);
        };
        // what the ring will take first comes into L2 while the kernel in front of this one ends; it is read only after the wait
        const int fill = min(p.stages, nsteps);
        for (int i = 0; i < fill; ++i) {
            if (W == kFp8Blocked) tma_prefetch_4d(&wmap, 0, 0, tile * (kTileRows / 16), (begin + i) * 2);
            else if (EPI == kSwiGlu) {
                for (int h = 0; h < 2; ++h)
                    tma_prefetch_2d(&wmap, (begin + i) * (W == kBf16Rows ? kStep / 2 : kStep), h * (p.n / 2) + tile * (kTileRows / 2));
            } else tma_prefetch_2d(&wmap, (begin + i) * (W == kBf16Rows ? kStep / 2 : kStep), tile * kTileRows);
        }
        grid_dependency_sync();
        for (int i = 0; i < fill; ++i) load_w(i, i), load_x(i, i);
        int s = 0;
        uint32_t phase = 0;
        for (int i = fill; i < nsteps; ++i) {
            if (!mbar_wait(&empty[s], phase)) {
                ok = false;
                break;
            }
            load_w(i, s);
            load_x(i, s);
            if (++s == p.stages) s = 0, phase ^= 1u;
        }
        if (!ok) {      // nobody leaves with copies in flight: slot s and those after it were filled a round earlier than those before it
            for (int j = 0; j < p.stages; ++j) mbar_wait(&full[j], j < s ? phase ^ 1u : phase);
        }
    } else {
        grid_dependency_sync();
        if (tid == 32) {
            constexpr uint32_t idesc = W == kBf16Rows ? mma_desc(1, 1, kTileRows, N) : mma_desc(0, 0, kTileRows, N);
            int s = 0;
            uint32_t phase = 0;
            for (int i = 0; i < nsteps; ++i) {
                if (!mbar_wait(&full[s], phase)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t w = ring + s * stage_bytes<N>(), x = w + kWBytes, d = acc + (i % kAcc) * N;
#pragma unroll
                for (int j = 0; j < kStep / 32; ++j) {      // 32 bytes of k per instruction
                    const uint64_t a = W == kFp8Blocked ? kmajor_desc<64>(w + (j / 2) * (kWBytes / 2) + (j % 2) * 32) : kmajor_desc<128>(w + j * 32);
                    const uint64_t b = kmajor_desc<128>(x + j * 32);
                    if (W == kBf16Rows) tc_mma_f16(d, a, b, idesc, i >= kAcc || j > 0);
                    else tc_mma_f8(d, a, b, idesc, i >= kAcc || j > 0);
                }
                // only a slot that the copies wait for: `done` stands for the rest, and nothing arrives in shared memory behind it
                if (i + p.stages < nsteps) tc_commit(&empty[s]);
                if (++s == p.stages) s = 0, phase ^= 1u;
            }
            tc_commit(&done);      // an arrival at once where there was nothing to multiply
        }
    }
    __syncwarp();
    ok = mbar_wait(&done, 0) && ok;
    if (!ok) *p.status = 1;
    tc_fence_after();
    // the partial tile, token-major fp32, over the ring: every copy has been multiplied
    const uint32_t partial = ring;
    const int channel = W == kFp8Blocked ? tid ^ ((tid >> 3) & 1) : tid;
    float r[N];
#pragma unroll
    for (int j = 0; j < N; ++j) r[j] = 0.f;
    for (int c = 0; c < min(kAcc, nsteps); ++c) {
        float v[N];
#pragma unroll
        for (int j = 0; j < N; j += 16) tmem_ld16(v + j, acc + (static_cast<uint32_t>(warp * 32) << 16) + c * N + j);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < N; ++j) r[j] += v[j];
    }
#pragma unroll
    for (int j = 0; j < N; ++j) asm volatile("st.shared.f32 [%0], %1;" ::"r"(partial + (j * kPitch + channel) * 4), "f"(r[j]) : "memory");
    tc_fence_before();
    if (ks > 1) cluster_arrive();
    // Before the wait for the cluster: a CTA that waits for its peers holds no tensor memory, for which a peer may still be waiting on another SM, behind
    // CTAs that in their turn wait for theirs.  Allocation has no time limit, and neither shared memory nor registers keep short parts of k at four CTAs an SM.
    // Only the warp that frees waits for the others' reads of it.
    if (warp == 1) {
        asm volatile("barrier.cta.sync 1, %0;" ::"n"(kThreads) : "memory");
        tc_fence_after();
        tmem_free<kTmemCols>(acc);
        __syncwarp();
    } else {
        asm volatile("barrier.cta.arrive 1, %0;" ::"n"(kThreads) : "memory");
    }
    if (ks > 1) cluster_wait();
    else __syncthreads();
    // the tile's outputs, four channels at a time, dealt out over the cluster; the sum over the cluster in CTA order
    auto sum = [&](int tok, int ch, int n) {      // channels ch.. of the tile, n.. of the weights
        const uint32_t at = partial + (tok * kPitch + ch) * 4;
        float4 v = ld_cluster_f32x4(at, 0);
#pragma unroll 8
        for (int c = 1; c < ks; ++c) {
            const float4 o = ld_cluster_f32x4(at, c);
            v.x += o.x, v.y += o.y, v.z += o.z, v.w += o.w;
        }
        if (W != kBf16Rows) {
            const float xs = p.x_scale[tok];
            const float *ws = p.w_scale + n;
            const float4 f = p.vec ? *reinterpret_cast<const float4 *>(ws) : make_float4(ws[0], ws[1], ws[2], ws[3]);
            v.x = v.x * xs * f.x, v.y = v.y * xs * f.y, v.z = v.z * xs * f.z, v.w = v.w * xs * f.w;
        }
        return v;
    };
    constexpr int quads = (EPI == kSwiGlu ? kTileRows / 2 : kTileRows) / 4;
    for (int e = part * kThreads + tid; e < quads * p.m; e += ks * kThreads) {
        const int ch = (e % quads) * 4, tok = e / quads, n = tile * quads * 4 + ch;
        const float4 v = sum(tok, ch, n);
        if constexpr (EPI == kPlain) {
            bf16 *out = p.out + static_cast<size_t>(tok) * p.n + n;
            const uint2 o = make_uint2(pack2(v.x, v.y), pack2(v.z, v.w));
            if (p.vec) *reinterpret_cast<uint2 *>(out) = o;
            else
                for (int i = 0; i < 4; ++i) out[i] = reinterpret_cast<const bf16 *>(&o)[i];
        } else if constexpr (EPI == kSwiGlu) {
            const float4 u = sum(tok, kTileRows / 2 + ch, p.n / 2 + n);
            const float g[4] = {rounded(silu(rounded(v.x))), rounded(silu(rounded(v.y))), rounded(silu(rounded(v.z))), rounded(silu(rounded(v.w)))};
            *reinterpret_cast<uint2 *>(p.out + static_cast<size_t>(tok) * (p.n / 2) + n) =
                make_uint2(pack2(g[0] * rounded(u.x), g[1] * rounded(u.y)), pack2(g[2] * rounded(u.z), g[3] * rounded(u.w)));
        } else {      // a tile is a head: rope_append_kernel's arithmetic
            const RopeCall &r = p.rope;
            const int b = tok / r.t, kv = tile - r.heads;
            const Place place = place_of(r.pos[tok % r.t], r.max_seq, r.table_rows);
            const int64_t at = place.at;
            if (!place.valid) {
                p.status[kStatusPosition] = 1;
                if (kv < 0) *reinterpret_cast<uint2 *>(p.out + (static_cast<size_t>(tok) * r.heads + tile) * kTileRows + ch) = make_uint2(kNan2, kNan2);
                continue;
            }
            if (kv >= r.kv_heads) {
                *reinterpret_cast<uint2 *>(static_cast<bf16 *>(r.v_cache) + ((static_cast<int64_t>(b) * r.kv_heads + kv - r.kv_heads) * r.max_seq + at) * kTileRows + ch) =
                    make_uint2(pack2(v.x, v.y), pack2(v.z, v.w));
                continue;
            }
            const int64_t row = place.angle * (kTileRows / 2) + ch / 2;
            const float2 c = *reinterpret_cast<const float2 *>(r.cos + row), s = *reinterpret_cast<const float2 *>(r.sin + row);
            float lo[2], hi[2];
            rotate(rounded(v.x), rounded(v.y), c.x, s.x, lo[0], hi[0]);
            rotate(rounded(v.z), rounded(v.w), c.y, s.y, lo[1], hi[1]);
            bf16 *dst = kv < 0 ? p.out + (static_cast<size_t>(tok) * r.heads + tile) * kTileRows
                               : static_cast<bf16 *>(r.k_cache) + ((static_cast<int64_t>(b) * r.kv_heads + kv) * r.max_seq + at) * kTileRows;
            *reinterpret_cast<uint32_t *>(dst + ch / 2) = pack2(lo[0], lo[1]);
            *reinterpret_cast<uint32_t *>(dst + kTileRows / 2 + ch / 2) = pack2(hi[0], hi[1]);
        }
    }
    if (ks > 1) cluster_barrier();      // nobody leaves while its partial tile may still be read
}


// Never launched: asked how many CTAs of the streaming kernel's size run at once, since the answer for a kernel with tensor memory is one per SM.
__global__ void __launch_bounds__(kThreads) yardstick_kernel() {}

// Steps in the ring of a CTA.  Where k is not split six keep more in flight; four leave room for a third CTA and for the next kernel's (1280 x 8192: 6.8 / 7.3 us with
// 4 / 8, and 22528 x 4096 in two parts of k, 16 tokens: 30.1 us, where rings of six, for which there is no third CTA, took 36.5).
int ring_stages(int columns, bool split, int tiles, int sms) { return columns == 32 ? 5 : split || tiles <= sms ? 4 : kRingMax; }

template <int W, int EPI>
const void *kernel_for(int columns) {
    return columns == 16 ? reinterpret_cast<const void *>(&stream_linear_kernel<W, 16, EPI>) : reinterpret_cast<const void *>(&stream_linear_kernel<W, 32, EPI>);
}
// blocked weights only with the plain epilogue
const void *kernel_of(int w, int epilogue, int columns) {
    if (w == kFp8Blocked) return kernel_for<kFp8Blocked, kPlain>(columns);
    if (epilogue == kSwiGlu) return w == kFp8Rows ? kernel_for<kFp8Rows, kSwiGlu>(columns) : kernel_for<kBf16Rows, kSwiGlu>(columns);
    if (epilogue == kRopeAppend) return w == kFp8Rows ? kernel_for<kFp8Rows, kRopeAppend>(columns) : kernel_for<kBf16Rows, kRopeAppend>(columns);
    return w == kFp8Rows ? kernel_for<kFp8Rows, kPlain>(columns) : kernel_for<kBf16Rows, kPlain>(columns);
}

}  // namespace

cudaError_t stream_linear_setup(DecodeDevice *d) {
    for (int columns = 16; columns <= kMaxTokens; columns += 16) {
        const int smem = smem_bytes(columns, ring_stages(columns, true, 0, d->sms)) + 256;      // barriers and such
        const void *fn = reinterpret_cast<const void *>(&yardstick_kernel);
        cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        for (int ks = 1; ks <= 8 && e == cudaSuccess; ++ks) {
            int64_t ctas = 0;
            e = resident_ctas(fn, kThreads, ks, d->sms, &ctas, smem);
            d->stream_ctas[columns / 32][ks] = static_cast<int>(ctas);
        }
        if (e != cudaSuccess) return e;
    }
    for (int columns = 16; columns <= kMaxTokens; columns += 16)
        for (int w : {kFp8Blocked, kFp8Rows, kBf16Rows})
            for (int epilogue : {kPlain, kSwiGlu, kRopeAppend}) {
                const cudaError_t e = cudaFuncSetAttribute(kernel_of(w, epilogue, columns), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                           smem_bytes(columns, kRingMax));
                if (e != cudaSuccess) return e;
            }
    return cudaSuccess;
}

int stream_linear(const StreamLinearCall &c, const DecodeDevice &d, cudaStream_t stream) {
    const int columns = c.m <= 16 ? 16 : 32, es = c.x_scale ? 1 : 2;
    CUtensorMap wmap, xmap;
    const CUtensorMapDataType type = es == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const uint64_t k = c.k, row = k * es, n = c.n;
    int rc;
    if (c.blocked) {
        const uint64_t sizes[4] = {128, 8, n / 16, k / 64}, strides[3] = {128, k * 16, 1024};
        const uint32_t box[4] = {128, 8, kTileRows / 16, kStep / 64};
        rc = encode_map(&wmap, type, c.w, 4, sizes, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
    } else {
        const uint64_t sizes[2] = {k, n}, strides[1] = {row};
        const uint32_t box[2] = {static_cast<uint32_t>(kStep / es), static_cast<uint32_t>(c.epilogue == kSwiGlu ? kTileRows / 2 : kTileRows)};
        rc = encode_map(&wmap, type, c.w, 2, sizes, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
    }
    if (!rc) {
        const uint64_t sizes[2] = {k, static_cast<uint64_t>(c.m)}, strides[1] = {row};
        const uint32_t box[2] = {static_cast<uint32_t>(kStep / es), static_cast<uint32_t>(columns)};
        rc = encode_map(&xmap, type, c.x, 2, sizes, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
    }
    if (rc) return set_last_error(GPUK_ERR_CUDA, "linear: the driver refused the tensor map (%d)", rc);
    const int tiles = c.n / kTileRows, steps = static_cast<int>((row + kStep - 1) / kStep);
    // Parts of k: as many as run at once in clusters of that size (6144 x 8192, 24 tokens: 6 parts, whose 48 clusters do not all fit, 26.6 us, 5 18.7, 4 19.7), 5 and 7 only
    // where they leave a tenth of the places free (7168 x 4096: 5 14.4, 4 13.5), as long as a part keeps enough steps to pay for its start: 8 tokens, 2048 x 2048 in 16
    // steps: 1 part 6.9 us, 2 5.3, 4 4.2, 8 4.7; 64 steps: 1280 x 8192 1 20.9, 4 8.2, 8 6.6, 10240 x 8192 with 32 tokens 1 24.0, 2 18.5, 3 17.2, 4 24.2.
    int ks = c.ks;
    if (ks == 0) {
        const int most = steps >= 32 ? 8 : steps < 8 ? 1 : tiles * 4 <= d.sms * 7 / 5 ? 4 : 2, *fit = d.stream_ctas[columns / 32];
        for (ks = most; ks > 1 && tiles * ks > (ks == 5 || ks == 7 ? fit[ks] * 9 / 10 : fit[ks]); --ks) {}
    }
    const int part_steps = (steps + ks - 1) / ks;
    const int stages = std::max(1, std::min(ring_stages(columns, ks > 1, tiles, d.sms), part_steps));
    const int smem = std::max(smem_bytes(columns, stages), 1024 + columns * kPitch * 4);
    const bool vec = ((reinterpret_cast<uintptr_t>(c.out) & 7u) | (reinterpret_cast<uintptr_t>(c.w_scale) & 15u)) == 0;
    StreamParams p = {c.x_scale, c.w_scale, static_cast<bf16 *>(c.out), c.m, c.n, steps, stages, ks, vec, c.rope, d.status};
    const void *fn = kernel_of(es == 2 ? kBf16Rows : c.blocked ? kFp8Blocked : kFp8Rows, c.epilogue, columns);
    void *args[] = {&wmap, &xmap, &p};
    const cudaError_t e = launch_kernel(fn, tiles * ks, kThreads, ks, false, args, stream, smem);
    if (e != cudaSuccess) return set_last_error(GPUK_ERR_CUDA, "linear: launch failed: %s", cudaGetErrorString(e));
    return GPUK_OK;
}

}  // namespace gpuk

using namespace gpuk;

// The checks every entry point makes; `what` names it.
static int run_skinny(const char *what, StreamLinearCall c, void *stream) {
    const int es = c.x_scale ? 1 : 2;
    if (c.m < 0 || c.n <= 0 || c.k <= 0) return set_last_error(GPUK_ERR_INVALID_ARGUMENT, "%s: bad shape %d x %d x %d", what, c.m, c.n, c.k);
    if (c.m > kMaxTokens) return set_last_error(GPUK_ERR_UNSUPPORTED, "%s: %d tokens; this kernel is built for at most %d", what, c.m, kMaxTokens);
    if (c.n % kTileRows || static_cast<int64_t>(c.k) * es % 16)
        return set_last_error(GPUK_ERR_UNSUPPORTED, "%s: n must be a multiple of %d and k of %d (got %d, %d)", what, kTileRows, 16 / es, c.n, c.k);
    if (c.ks < 0 || c.ks > 8) return set_last_error(GPUK_ERR_INVALID_ARGUMENT, "%s: k_split must be 0 to 8", what);
    if (c.m == 0) return GPUK_OK;
    if (!c.x || !c.w || !c.out || !c.x_scale != !c.w_scale) return set_last_error(GPUK_ERR_INVALID_ARGUMENT, "%s: null pointer", what);
    if ((reinterpret_cast<uintptr_t>(c.x) | reinterpret_cast<uintptr_t>(c.w)) & 15u) return set_last_error(GPUK_ERR_INVALID_ARGUMENT, "%s: operands must be 16-byte aligned", what);
    const DecodeDevice *d = nullptr;
    const int rc = decode_device(&d);
    return rc != GPUK_OK ? rc : stream_linear(c, *d, static_cast<cudaStream_t>(stream));
}

extern "C" int gpuk_linear_skinny(const void *x_bf16, const void *w_bf16, void *out_bf16, int m, int n, int k, int k_split, void *stream) {
    return run_skinny("linear", {x_bf16, nullptr, nullptr, w_bf16, out_bf16, m, n, k, false, kPlain, {}, k_split}, stream);
}

extern "C" int gpuk_swiglu_skinny(const void *x, const float *x_scale, const void *w, const float *w_scale, void *out_bf16, int m, int n, int k, int k_split, void *stream) {
    if ((reinterpret_cast<uintptr_t>(out_bf16) & 7u) | (reinterpret_cast<uintptr_t>(w_scale) & 15u))
        return set_last_error(GPUK_ERR_INVALID_ARGUMENT, "swiglu: scales must be 16-byte aligned, results 8-byte");
    return run_skinny("swiglu", {x, x_scale, w_scale, w, out_bf16, m, n, k, false, kSwiGlu, {}, k_split}, stream);
}

extern "C" int gpuk_qkv_rope_skinny(const void *x, const float *x_scale, const void *w, const float *w_scale, const float *cos, const float *sin, const int64_t *pos,
                                    void *q_out, void *k_cache, void *v_cache, int batch, int t, int heads, int kv_heads, int k, int table_rows, int max_seq,
                                    int k_split, void *stream) {
    if (batch < 0 || t <= 0 || heads <= 0 || kv_heads <= 0 || table_rows <= 0 || max_seq <= 0 || batch > kMaxTokens || t > kMaxTokens || heads > (1 << 20) || kv_heads > (1 << 20))
        return set_last_error(GPUK_ERR_INVALID_ARGUMENT, "qkv_rope: bad sizes");
    if (!cos || !sin || !pos || !k_cache || !v_cache) return set_last_error(GPUK_ERR_INVALID_ARGUMENT, "qkv_rope: null pointer");
    if ((reinterpret_cast<uintptr_t>(q_out) | reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache) | reinterpret_cast<uintptr_t>(cos) |
         reinterpret_cast<uintptr_t>(sin) | reinterpret_cast<uintptr_t>(w_scale)) & 15u)
        return set_last_error(GPUK_ERR_INVALID_ARGUMENT, "qkv_rope: pointers must be 16-byte aligned");
    return run_skinny("qkv_rope", {x, x_scale, w_scale, w, q_out, batch * t, (heads + 2 * kv_heads) * kTileRows, k, false, kRopeAppend,
                                   {cos, sin, pos, k_cache, v_cache, t, heads, kv_heads, table_rows, max_seq}, k_split}, stream);
}
