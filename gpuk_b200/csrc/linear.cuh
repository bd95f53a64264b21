// What the kernels of a decode step share: their set-up per device, and the call of the streaming linear layer.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace gpuk {

// What the streaming kernel does with its sums before it stores them.
enum LinearEpilogue { kPlain, kSwiGlu, kRopeAppend };
struct RopeCall {
    const float *cos, *sin;                 // [table_rows, 64]
    const int64_t *pos;                     // [t]
    void *k_cache, *v_cache;                // bf16 [batch, kv_heads, max_seq, 128]
    int t, heads, kv_heads, table_rows, max_seq;
};

struct StreamLinearCall {
    const void *x;                          // [m, k]
    const float *x_scale, *w_scale;         // [m], [n]; nullptr: bf16 operands
    const void *w;                          // [n, k] row-major, or blocked
    void *out;                              // bf16 [m, n]
    int m, n, k;                            // m <= 32, n a multiple of 128, rows of k a multiple of 16 bytes
    bool blocked;                           // FP8 weights in the order of gpuk_fp8_pack_weight
    LinearEpilogue epilogue;                // kSwiGlu: out [m, n / 2] = silu(first half) * second half; kRopeAppend: out [m, heads * 128], keys and values to the caches
    RopeCall rope;
    int ks;                                 // CTAs that share a tile (0: chosen from the shape)
};
// A device as the kernels of a decode step plan for it.
struct DecodeDevice {
    int sms;
    // The status words that the kernels set (gpuk_fp8_linear_status): the first where a launch went wrong, the one at kStatusPosition where a position pointed
    // outside the cache or the table of angles.
    int *status;
    // CTAs that run at once in clusters of a given size: fewer than SMs times CTAs per SM, by what does not divide the groups of SMs that clusters stay in
    int stream_ctas[2][9];                  // streaming linear layer with 16 and 32 columns, k split
    int attention_ctas[2][9];               // decode attention with the short and the long ring
};
cudaError_t stream_linear_setup(DecodeDevice *d);          // once per device
cudaError_t decode_attention_setup(DecodeDevice *d);
cudaError_t prefill_attention_setup();
constexpr int kStatusPosition = 1, kDecodeStatusWords = 2;
// The current device; the first call on it opts the kernels in to their shared memory, so that no later call has set-up left to do.
int decode_device(const DecodeDevice **device);
int stream_linear(const StreamLinearCall &c, const DecodeDevice &d, cudaStream_t stream);

}  // namespace gpuk
