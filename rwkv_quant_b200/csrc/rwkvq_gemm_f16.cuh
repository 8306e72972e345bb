// fp16 tensor-core GEMM over operands that lie in HBM / L2 as plain fp16 matrices, and the kernels
// that bring packed weights into that form.  Interface of rwkvq_gemm_f16.cu for the launch code of
// the sequence path and of the rwkvq_gemm entry points.
#pragma once
#include "rwkvq_common.cuh"

namespace rwkvq {

constexpr int kHgMaxProbs = 4;      // problems one launch can carry (r / k / v; the LoRA branches)

// What the epilogue makes of an accumulator row (y = sum over K, already divided by the token's scale):
enum HgOut {
    HG_F32 = 0,        // y32[tok, row] = epi(y)                        (epi: RWKVQ_EPI_*)
    HG_RELU2_F16,      // y16[tok, row] = fp16(relu(y)^2 * s_tok), out_scale[tok] = s_tok (see HgProb::bound)
    HG_SPLIT           // act(y) as the fp16 pair y16[tok, row] = hi, y16[tok, lo_off + row] = lo
};

// One product y[tok, row] = sum_k W[row, k] x[tok, k].
struct HgProb {
    const __half* w;            // [rows, k] K-major, row pitch w_pitch (halves, multiple of 8)
    const __half* x;            // [M, terms * k], row pitch x_pitch; terms = 2: [hi | lo], W is used for both
    long long w_pitch, x_pitch;
    int rows, k, terms;         // k: multiple of 64
    int w_rows;                 // rows W has in memory (0: `rows`); the rest of `rows` counts as zero
    const float* row_scale;     // [M] powers of two x was multiplied with, or null
    int out, epilogue, act;
    float* y32;
    const float* resid;         // [M, ldy] (RWKVQ_EPI_ADD)
    __half* y16;
    long long ldy;              // row pitch of y32 / resid or of y16
    int lo_off;
    // HG_RELU2_F16: |y| <= sqrt(bound_n2[0..n_bound) summed) * sqrt(x_n2[tok]) gives the power of two
    // s_tok with relu(y)^2 * s_tok inside the fp16 range before any y is known
    const float* w_n2;          // [n_w_n2] per 256 columns: the largest squared norm over the rows of W
    int n_w_n2;
    const float* x_n2;          // [M] squared norm of the unscaled token row
    float* out_scale;           // [M]
};

// status: device word that receives RWKVQ_E_TIMEOUT if a bounded wait ran out
int launch_gemm_f16(const HgProb* probs, int n_probs, int M, int* status, cudaStream_t s);

// fp32 rows -> x16 = fp16(x * scale) with the power of two scale[tok] that brings max|x| below 2^14;
// status (optional) is cleared
int launch_row_scale(const float* x, long long ldx, int cols, int M, float* scale, __half* x16, long long pitch, int* status, cudaStream_t s);

// Packed sb6 / sym rows [row0, row0 + rows) -> fp16(q * s + m) [rows, cols] (pitch cols).
// n2 (optional, [cols / 256], zeroed by the caller): merged with the largest squared norm of a row's
// 256-column pieces.
// per_sm: CTAs an SM where other kernels of the same call run beside this one (0: none do)
int launch_dequant_f16(const rwkvq_qtensor& t, int row0, int rows, __half* out, float* n2, cudaStream_t s, int per_sm = 0);

// Up to 8 matrices stored [in, out] -> fp16 transposed [out, in_pad] (in_pad = in rounded up to 64, the
// padding zero), in the loader's precision fp16(bf16(w)).
struct TransposeJob { const rwkvq_qtensor* t; __half* out; };
int launch_dequant_f16_t(const TransposeJob* jobs, int n, cudaStream_t s);

}  // namespace rwkvq
