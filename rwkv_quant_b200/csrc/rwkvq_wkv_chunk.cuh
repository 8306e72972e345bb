// Time-mix core of long sequences (rwkvq_wkv_chunk.cu): interface for the one-call forward.
#pragma once
#include "rwkvq_common.cuh"

namespace rwkvq {

struct WkvChunkArgs {
    const float *r, *k, *v, *yw, *ya, *yv, *v_first, *g;      // [B, T, H * 64]; yv / v_first null on layer 0
    const float *w0, *a0, *v0, *k_k, *k_a, *r_k, *ln_w, *ln_b;  // [H * 64]
    const float* h_in;                                        // [B, H, 64, 64] or null (zeros)
    float* h_out;                                             // [B, H, 64, 64]
    // the output: where wkv_chunked_f16(B, H), fp16 rows under a power of two each, else fp32
    __half* og16;                                             // [B * T, og_pitch]
    float* og_scale;                                          // [B * T]
    long long og_pitch;
    float* og;                                                // [B, T, H * 64]
    float* ops;                                               // scratch: wkv_chunk_floats(B, T, H)
    float* dp;                                                // scratch: [B, T, H]
    float* y;                                                 // scratch: [B, T, H * 64]
    int* status;                                              // receives RWKVQ_E_TIMEOUT if a bounded wait ran out
    int B, T, H;
    bool spread;                                              // other kernels run beside the scan: keep its CTAs apart
};
constexpr int kChunkSplitPairs = 148;                         // heads of all sequences up to which a head's rows are split over CTAs
inline bool wkv_chunked_f16(int B, int H) { return static_cast<long long>(B) * H <= kChunkSplitPairs; }
size_t wkv_chunk_floats(int B, int T, int H);
// decay, gates, key normalisation, the scan and the tail (group norm + bonus + gate); 16-byte aligned arrays
int launch_wkv_chunked(const WkvChunkArgs& a, cudaStream_t s);

}  // namespace rwkvq
