// Launchers of the sequence-path glue kernels (rwkvq_seq.cu, rwkvq_wkv.cu) for the one-call forward.
#pragma once
#include "rwkvq_gemm_sb.cuh"

namespace rwkvq {

// Forms a mix row can be written in (bits of SeqPrepArgs::mode)
constexpr int kPrepScaled = 1;      // scaled fp16 copy + scale, the operand of the fp16 GEMM
constexpr int kPrepSplit = 2;       // fp16 pair [hi | lo]
constexpr int kPrepF32 = 4;
constexpr int kPrepAmax = 8;        // max|row| into scale[m] (beside kPrepF32: what the small-batch linears read)

constexpr int kPrepPair = 16;       // scaled fp16 pair with block sums into pair[m]: what launch_gemm_sb reads

struct SeqPrepArgs {
    const float *x, *ln_w, *ln_b, *shift_in, *mix;
    float* shift_out;
    __half* x16[6];        // [N, D + 64]
    float* scale[6];       // [N]
    __half* split[6];      // [N, 2 D]
    float* f32[6];         // [N, D]
    SbRows pair[6];
    int mode[6];
    int T, D, n_mix;
    float* n2;             // optional [N]: squared norm of mix row 0 (unscaled)
    float *zero_a, *zero_b;    // optional [N]: cleared
};
// mix == NULL: no shift and no lerp, the normalised row itself (n_mix = 1; shift_in, shift_out NULL).  shift_out may equal
// shift_in where T = 1 (kPrepPair: seq_prep_in_place_ok).  kPrepPair needs D % 256 == 0.
int launch_seq_prep(const SeqPrepArgs& a, long long n_tokens, cudaStream_t s);
inline bool seq_prep_in_place_ok(int D) { return D % 256 == 0 && D <= 4096; }

}  // namespace rwkvq
