// fp32-grade linear for small batches on tcgen05 (rwkvq_gemm_sb.cu): interface for the launch code and for the
// kernels that write activation rows in the form it reads.
#pragma once
#include <cuda.h>

#include "rwkvq_common.cuh"

namespace rwkvq {

// N activation rows as fp16 pairs scaled per row by a power of two, |x 2^s| <= 2^9.
struct SbRows {
    __half *hi, *lo;          // [N, pitch]: fp16(x 2^s), fp16(x 2^s - hi); 16-byte aligned, pitch a multiple of 8
    __half* sums;             // [K / 256][2][N][8]: sums of x 2^s over the 32-column blocks, high then low halves
    float* unscale;           // [N] 2^-s
    long long pitch;
};
inline size_t sb_pitch(int cols) { return static_cast<size_t>(cols) + 64; }      // rows of a TMA box spread over the L2 slices
// halves of storage for N rows of `cols` columns (hi, lo, sums)
inline size_t sb_halves(int N, int cols) { return 2 * static_cast<size_t>(N) * sb_pitch(cols) + static_cast<size_t>(N) * (cols / 256) * 16; }
inline SbRows sb_rows(__half* base, float* unscale, int N, int cols) {
    SbRows r;
    r.pitch = static_cast<long long>(sb_pitch(cols));
    r.hi = base; r.lo = base + static_cast<size_t>(N) * r.pitch; r.sums = r.lo + static_cast<size_t>(N) * r.pitch; r.unscale = unscale;
    return r;
}

// Power of two with |x| 2^s <= 2^9 for max|x| = m, and its inverse; rows without a finite maximum keep 1 and propagate.
__device__ __forceinline__ void sb_scale(float m, float& s1, float& u1) {
    s1 = u1 = 1.f;
    if (m > 0.f && m < INFINITY) {
        int e = 0;
        frexpf(m, &e);
        e = max(-100, e);
        s1 = ldexpf(1.f, 9 - e);
        u1 = ldexpf(1.f, e - 9);
    }
}

// Columns 8 i .. 8 i + 7 of row n (already scaled) as a pair; the four lanes of an aligned quad hold one 32-column
// block (consecutive i), whose sum the first of them stores.
__device__ __forceinline__ void sb_store_pair(const SbRows& o, int n, int N, int i, const float (&v)[8]) {
    uint32_t hw[4], lw[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const __half2 hh = __floats2half2_rn(v[2 * j], v[2 * j + 1]);
        const float2 hf = __half22float2(hh);
        const __half2 ll = __floats2half2_rn(v[2 * j] - hf.x, v[2 * j + 1] - hf.y);
        hw[j] = *reinterpret_cast<const uint32_t*>(&hh);
        lw[j] = *reinterpret_cast<const uint32_t*>(&ll);
    }
    *reinterpret_cast<uint4*>(o.hi + static_cast<size_t>(n) * o.pitch + 8 * i) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
    *reinterpret_cast<uint4*>(o.lo + static_cast<size_t>(n) * o.pitch + 8 * i) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
    float bs = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
    bs += __shfl_xor_sync(0xFFFFFFFFu, bs, 1);
    bs += __shfl_xor_sync(0xFFFFFFFFu, bs, 2);
    if ((i & 3) == 0) {
        const __half sh = __float2half_rn(bs);
        __half* s = o.sums + (static_cast<size_t>(i >> 5) * 2 * N + n) * 8 + ((i >> 2) & 7);
        s[0] = sh;
        s[static_cast<size_t>(N) * 8] = __float2half_rn(bs - __half2float(sh));
    }
}

// max|x| of each row, then the pairs; status (optional) is cleared.  cols: a multiple of 256
int launch_split_rows(const float* x, long long ldx, int cols, int N, const SbRows& o, int* status, cudaStream_t s);
// y[k] = epi(W_k x_k) for tensors gemm_sb_ok accepts, one shape and layout; rows[k]: the pairs of x_k;
// amax_outs (optional, per matrix): [N] slots merged with max|y| per token
int launch_gemm_sb(const rwkvq_qtensor* ts, int n_mats, const SbRows* rows, int N, float* const* ys, long long ldy, int epilogue,
                   const float* const* resids, float* const* amax_outs, int* status, int force_ks, cudaStream_t s, const Ahead* ahead = nullptr);
bool gemm_sb_ok(const rwkvq_qtensor& t);                  // sb6 / sym with the relayouted records and planes, 16-byte aligned streams
bool gemm_sb_pays(const rwkvq_qtensor& t, int N);
// tensor map of an fp16 matrix: boxes of 64 columns x box_rows, 128-byte swizzle, zero fill (rwkvq_gemm_f16.cu)
int make_half_map(CUtensorMap* map, const __half* base, long long rows, long long cols, long long pitch, int box_rows);
// tensor map of packed rows of row_bytes (a multiple of 16): boxes of 16, 32, 64 or 128 bytes x box_rows, swizzled by their width
// (16: not), zero fill
int make_byte_map(CUtensorMap* map, const void* base, long long rows, long long row_bytes, int box_bytes, int box_rows);

}  // namespace rwkvq
