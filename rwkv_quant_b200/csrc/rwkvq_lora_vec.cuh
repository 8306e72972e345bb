// The LoRA branches of the time-mix block for ONE stream, without launches of their own:
//   down   y-slices of the r / k / v GEMV's grid (rwkvq_gemv_mma.cu): both products read rows the same LayerNorm wrote;
//   up     the head of the time-mix core (rwkvq_decode.cu): a head's CTA needs its own 64 columns of the four W2 only.
// The layer's chain loses two dependent launches and the fork and join of a side stream, behind which no kernel starts
// programmatically (its weight loads then wait for the join).  2048 wide: 18.5 us of chain in four launches -> 14 in three.
#pragma once
#include <type_traits>

#include "rwkvq_decode_parts.cuh"

namespace rwkvq {

constexpr int kLvCols = 8;               // rank columns of a down CTA: half the sectors of a row's 16 bytes, and 64 CTAs at rank 512
constexpr int kLvMaxSmem = 100 * 1024;   // of the time-mix core: two CTAs per SM
constexpr int kLvMaxD = 4096;            // rows of W1: 16 per thread, 64 registers of weights

struct LoraVecArgs {
    QView t[4];              // W1 [D, r] (down) or W2 [r, D] (up)
    const float* x[4];       // down: [D] fp32 per branch
    int act[4];              // down: 1 tanh, 2 sigmoid, 0 none
    int first[5];            // ranks of the branches before; first[n_br] = all ranks
    float* h;                // [first[n_br]] activated rank space
    int n_br, D;
};

// shared memory of the up projection: weights, h, the warps' partial sums
inline size_t lora_vec_smem(int ranks) { return static_cast<size_t>(ranks) * (64 * sizeof(__half) + sizeof(float)) + 8 * 256 * sizeof(float); }

// Whether one stream's LoRA branches run inside their neighbours: codes in whole bytes and 16-byte rows, ranks in
// multiples of 16, and room for a head's columns of all W2 twice per SM.
bool lora_vec_ok(const rwkvq_qtensor* const* t1, const rwkvq_qtensor* const* t2, int n_br, int D);
// The three projections of one stream (fp32 rows x_each) and the LoRA down projections in one launch.
int launch_gemv_mma_lora(int layout, const rwkvq_qtensor* ts, int n_mats, const void* const* x_each, float* y, long long ldy,
                         const LoraVecArgs& lora, const Ahead& ahead, cudaStream_t s);

// h[8 columns] = act(x @ W1): thread i owns rows 4 (i + 256 k) + e.  The weights are in registers as fp16 (exact, the
// loader's precision) before x is awaited; behind it there is one L2 round trip, 64 multiply-adds and one reduction.
template <int PER>                       // groups of 4 rows per thread
__device__ __forceinline__ void lora_down_vec(const LoraVecArgs& a, int cta) {
    __shared__ float red[8][kLvCols];
    const int col = cta * kLvCols, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int br = 0;
    while (col >= a.first[br + 1]) ++br;
    const QView& t = a.t[br];
    const int c = col - a.first[br], mode = lora_mode(t), n4 = a.D >> 2;
    const int nb = mode == 0 ? (t.cols + t.gs - 1) / t.gs : 0;
    __half2 w[PER][4][kLvCols / 2];
    auto rows = [&](auto m) {
        constexpr int MODE = decltype(m)::value;
        const int b0 = MODE == 0 ? c / t.gs : 0, b1 = MODE == 0 ? (c + 4) / t.gs : 0;
#pragma unroll
        for (int k = 0; k < PER; ++k)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = tid + 256 * k;
                float v0[4] = {0.f, 0.f, 0.f, 0.f}, v1[4] = {0.f, 0.f, 0.f, 0.f};
                if (i < n4) {
                    lora_w4<MODE>(t, 4 * i + e, c, nb, b0, v0);
                    lora_w4<MODE>(t, 4 * i + e, c + 4, nb, b1, v1);
                }
                w[k][e][0] = __floats2half2_rn(v0[0], v0[1]); w[k][e][1] = __floats2half2_rn(v0[2], v0[3]);
                w[k][e][2] = __floats2half2_rn(v1[0], v1[1]); w[k][e][3] = __floats2half2_rn(v1[2], v1[3]);
            }
    };
    if (mode == 0) rows(std::integral_constant<int, 0>{});
    else rows(std::integral_constant<int, 1>{});
    pdl_wait();
    float acc[kLvCols];
#pragma unroll
    for (int j = 0; j < kLvCols; ++j) acc[j] = 0.f;
    float4 xv[PER];
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int i = tid + 256 * k;
        xv[k] = i < n4 ? __ldcg(reinterpret_cast<const float4*>(a.x[br]) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int k = 0; k < PER; ++k)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float x = e == 0 ? xv[k].x : e == 1 ? xv[k].y : e == 2 ? xv[k].z : xv[k].w;
#pragma unroll
            for (int j = 0; j < kLvCols / 2; ++j) {
                const float2 f = __half22float2(w[k][e][j]);
                acc[2 * j] = fmaf(x, f.x, acc[2 * j]);
                acc[2 * j + 1] = fmaf(x, f.y, acc[2 * j + 1]);
            }
        }
    // 8 sums over 32 lanes: halve the values while halving the lanes (lane bits 4, 3, 2 pick the column), then two steps more
#pragma unroll
    for (int s = 16, n = kLvCols / 2; s >= 4; s >>= 1, n >>= 1) {
        const bool up = lane & s;
#pragma unroll
        for (int j = 0; j < n; ++j) {
            const float mine = up ? acc[n + j] : acc[j], other = up ? acc[j] : acc[n + j];
            acc[j] = mine + __shfl_xor_sync(0xFFFFFFFFu, other, s);
        }
    }
    acc[0] += __shfl_xor_sync(0xFFFFFFFFu, acc[0], 2);
    acc[0] += __shfl_xor_sync(0xFFFFFFFFu, acc[0], 1);
    if ((lane & 3) == 0) red[warp][lane >> 2] = acc[0];
    __syncthreads();
    if (tid < kLvCols) {
        float v = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) v += red[k][tid];
        if (a.act[br] == 1) v = tanhf(v);
        else if (a.act[br] == 2) v = sigmoidf_(v);
        a.h[col + tid] = v;
    }
}

// columns [c0, c0 + 64) of all W2 as fp16 [ranks][64] in shared memory (before h is awaited)
__device__ __forceinline__ void lora_up_stage(const LoraVecArgs& a, int c0, __half* w) {
    for (int br = 0; br < a.n_br; ++br) {
        const QView& t = a.t[br];
        const int n = t.rows * 4, nb = lora_mode(t) == 0 ? (t.cols + t.gs - 1) / t.gs : 0;
        __half* dst = w + a.first[br] * 64;
        auto rows = [&](auto m) {
            constexpr int MODE = decltype(m)::value;
#pragma unroll 4
            for (int item = threadIdx.x; item < n; item += 256) {        // 16 columns of a row: one 16-byte load
                const int r = item >> 2, c = c0 + (item & 3) * 16;
                const uint4 q = __ldg(reinterpret_cast<const uint4*>(t.codes + static_cast<size_t>(r) * t.cols + c));
                uint32_t out[8];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t b = k == 0 ? q.x : k == 1 ? q.y : k == 2 ? q.z : q.w;
                    float s, mn = 0.f, v[4];
                    if (MODE == 0) {
                        const size_t blk = static_cast<size_t>(r) * nb + (c + 4 * k) / t.gs;
                        s = __ldg(static_cast<const float*>(t.scale) + blk);
                        mn = __ldg(t.mn + blk);
                    } else {
                        s = __half2float(__ldg(static_cast<const __half*>(t.scale) + r));
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const uint32_t byte = (b >> (8 * e)) & 0xFFu;
                        v[e] = dense_param_rounding(MODE == 0 ? __fadd_rn(__fmul_rn(static_cast<float>(byte), s), mn)
                                                              : __fmul_rn(static_cast<float>(static_cast<int8_t>(byte)), s));
                    }
                    const __half2 lo = __floats2half2_rn(v[0], v[1]), hi = __floats2half2_rn(v[2], v[3]);
                    out[2 * k] = *reinterpret_cast<const uint32_t*>(&lo);
                    out[2 * k + 1] = *reinterpret_cast<const uint32_t*>(&hi);
                }
                uint4* d = reinterpret_cast<uint4*>(dst + r * 64 + (item & 3) * 16);
                d[0] = make_uint4(out[0], out[1], out[2], out[3]);
                d[1] = make_uint4(out[4], out[5], out[6], out[7]);
            }
        };
        if (lora_mode(t) == 0) rows(std::integral_constant<int, 0>{});
        else rows(std::integral_constant<int, 1>{});
    }
}

// y[br][64] += h @ W2 of the staged columns: warp w takes every 8th chunk of 16 ranks, a lane two columns; the warps'
// sums of branch br and column c go to part[w][br * 64 + c]
__device__ __forceinline__ void lora_up_vec(const LoraVecArgs& a, const __half* w, const float* h, float* part) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, chunks = a.first[a.n_br] >> 4;
    float acc[4][2];
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[b][0] = acc[b][1] = 0.f;
    for (int ch = warp; ch < chunks; ch += 8) {
        float s0 = 0.f, s1 = 0.f;
        const __half2* row = reinterpret_cast<const __half2*>(w + ch * 16 * 64) + lane;
#pragma unroll
        for (int k = 0; k < 16; k += 4) {
            const float4 hv = *reinterpret_cast<const float4*>(h + ch * 16 + k);
            const float hk[4] = {hv.x, hv.y, hv.z, hv.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = __half22float2(row[(k + e) * 32]);
                s0 = fmaf(hk[e], f.x, s0);
                s1 = fmaf(hk[e], f.y, s1);
            }
        }
#pragma unroll
        for (int b = 0; b < 4; ++b)
            if (b < a.n_br && ch * 16 >= a.first[b] && ch * 16 < a.first[b + 1]) { acc[b][0] += s0; acc[b][1] += s1; }
    }
#pragma unroll
    for (int b = 0; b < 4; ++b) *reinterpret_cast<float2*>(part + warp * 256 + b * 64 + 2 * lane) = make_float2(acc[b][0], acc[b][1]);
}

}  // namespace rwkvq
