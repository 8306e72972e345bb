// Time-mix core of short sequences in one kernel (rwkvq_tmix_seq.cu): interface for the one-call forward.
#pragma once
#include "rwkvq_common.cuh"

namespace rwkvq {

struct TmixSeqArgs {
    const float *r, *k, *v, *yw, *ya, *yv, *v_first, *g;        // [B, T, H * 64]; yv / v_first null on layer 0
    const float *w0, *a0, *v0, *k_k, *k_a, *r_k, *ln_w, *ln_b;  // [H * 64]
    const float* h_in;                                          // [B, H, 64, 64] or null (zeros)
    float* h_out;                                               // [B, H, 64, 64]; may be h_in
    float* og;                                                  // [B, T, H * 64]
    float* og_amax;                                             // optional [B, T]: max|og| of every row is merged into it
    int B, T, H;
};
int launch_tmix_seq(const TmixSeqArgs& p, cudaStream_t s);

}  // namespace rwkvq
