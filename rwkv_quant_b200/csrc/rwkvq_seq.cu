// Glue kernels of the sequence (prefill) path, T > 1: what the decode step does inside
// ln_shift_mix_kernel / tmix_core_kernel for one token, for all B*T tokens of a call.
//
//   seq_ln_shift_mix   xn = LN(x[b,t]);  prev = xn[b,t-1] (t = 0: the carried shift state, zeros
//                      for a fresh stream);  out[m][b,t] = xn + (prev - xn) * mix[m];
//                      new shift state = xn[b,T-1]            (quant_model.py:281-301, 648-651)
//   seq_tmix_pre       decay w = exp(-0.606531 sigmoid(yw + w0)), gate a = sigmoid(ya + a0),
//                      kk = l2norm_head(k * k_k), k' = k (1 + (a - 1) k_a),
//                      v' = v + (v_first - v) sigmoid(yv + v0) (layers > 0); emits w, k', v',
//                      -kk and kk*a, the operands of the WKV-7 scan       (quant_model.py:700-712)
#include "rwkvq_seq.cuh"

#include <algorithm>

#include "rwkvq_decode_parts.cuh"

namespace rwkvq {

constexpr int kSeqThreads = 256;
constexpr int kSeqPer = 16;          // D <= 4096

// One CTA per token.  The previous token's normalised row is recomputed here (same code,
// same bits as the CTA that owns it), so tokens do not depend on one another.
template <int NMIX>
__global__ void __launch_bounds__(kSeqThreads) seq_ln_shift_mix_kernel(const float* __restrict__ x,
                                                                       const float* __restrict__ ln_w,
                                                                       const float* __restrict__ ln_b,
                                                                       const float* __restrict__ shift_in,
                                                                       const float* __restrict__ mix,
                                                                       float* __restrict__ out,
                                                                       float* __restrict__ shift_out, int T, int D,
                                                                       long long n_tokens) {
    __shared__ float red[kSeqThreads / 32];
    const long long tok = blockIdx.x;
    const int b = static_cast<int>(tok / T), t = static_cast<int>(tok % T);
    const float* row = x + tok * D;
    float v[kSeqPer], pv[kSeqPer], lw[kSeqPer], lb[kSeqPer];
#pragma unroll
    for (int i = 0; i < kSeqPer; ++i) {
        const int d = threadIdx.x + i * kSeqThreads;
        const bool ok = d < D;
        v[i] = ok ? row[d] : 0.f;
        pv[i] = !ok ? 0.f : (t > 0 ? row[d - D] : (shift_in ? shift_in[static_cast<size_t>(b) * D + d] : 0.f));
        lw[i] = ok ? ln_w[d] : 0.f;
        lb[i] = ok ? ln_b[d] : 0.f;
    }
    auto normalise = [&](float (&y)[kSeqPer]) {
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < kSeqPer; ++i) s += y[i];
        const float mean = block_sum(s, red) / D;
        float s2 = 0.f;
#pragma unroll
        for (int i = 0; i < kSeqPer; ++i) {
            const float c = (threadIdx.x + i * kSeqThreads < D) ? y[i] - mean : 0.f;
            s2 += c * c;
        }
        const float inv = 1.0f / sqrtf(block_sum(s2, red) / D + 1e-5f);
#pragma unroll
        for (int i = 0; i < kSeqPer; ++i) y[i] = (y[i] - mean) * inv * lw[i] + lb[i];
    };
    normalise(v);
    if (t > 0) normalise(pv);               // t == 0: pv already is a normalised row (or zeros)
#pragma unroll
    for (int i = 0; i < kSeqPer; ++i) {
        const int d = threadIdx.x + i * kSeqThreads;
        if (d >= D) continue;
        const float xx = pv[i] - v[i];
        if (t == T - 1) shift_out[static_cast<size_t>(b) * D + d] = v[i];
#pragma unroll
        for (int m = 0; m < NMIX; ++m)
            out[(static_cast<size_t>(m) * n_tokens + tok) * D + d] = v[i] + xx * __ldg(mix + m * D + d);
    }
}

// ---- the same, emitting what the consumers of each mix read ---------------------------------
// A mix row feeds either the fp16 GEMM (which reads a per-token power-of-two-scaled
// fp16 copy, pitch D + 64 halves, plus the scale) or the LoRA GEMM (which reads the fp16 hi/lo
// split [hi | lo]), or both; writing those forms here saves the fp32 round trip through HBM and
// one launch per consumer.  The conversions are those of the GEMM's own pre-pass (scale =
// 2^(14 - exponent of the row maximum)) and of split_fp16_kernel.
__device__ __forceinline__ float block_max(float v, float* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float m = red[0];
    for (int w = 1; w < (blockDim.x >> 5); ++w) m = fmaxf(m, red[w]);
    return m;
}

// One CTA per token; thread t owns the column pairs 2 (t + 256 i), i < 8 (D <= 4096, D even).
__global__ void __launch_bounds__(kSeqThreads, 3) seq_ln_shift_mix_prep_kernel(const SeqPrepArgs a) {
    __shared__ float red[kSeqThreads / 32];
    constexpr int kPairs = kSeqPer / 2;
    const long long tok = blockIdx.x;
    const int D = a.D, b = static_cast<int>(tok / a.T), t = static_cast<int>(tok % a.T);
    const float* row = a.x + tok * D;
    pdl_launch_dependents();
    pdl_wait();
    if (threadIdx.x == 0) {
        if (a.zero_a != nullptr) a.zero_a[tok] = 0.f;
        if (a.zero_b != nullptr) a.zero_b[tok] = 0.f;
    }
    float2 v[kPairs], pv[kPairs];
    const float2 zero = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < kPairs; ++i) {
        const int d = 2 * (threadIdx.x + i * kSeqThreads);
        const bool ok = d < D;
        v[i] = ok ? *reinterpret_cast<const float2*>(row + d) : zero;
        pv[i] = !ok ? zero
                    : (t > 0 ? *reinterpret_cast<const float2*>(row + d - D)
                             : (a.shift_in ? *reinterpret_cast<const float2*>(a.shift_in + static_cast<size_t>(b) * D + d) : zero));
    }
    // LayerNorm of the token's row and of its predecessor's at once: the two means, then the two
    // variances, each pair in one block reduction (one barrier each)
    __shared__ float2 red_mean[kSeqThreads / 32], red_var[kSeqThreads / 32];
    auto block_sum2 = [&](float2 q, float2* buf) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            q.x += __shfl_xor_sync(0xFFFFFFFFu, q.x, o);
            q.y += __shfl_xor_sync(0xFFFFFFFFu, q.y, o);
        }
        if ((threadIdx.x & 31) == 0) buf[threadIdx.x >> 5] = q;
        __syncthreads();
        float2 tot = buf[0];
#pragma unroll
        for (int w = 1; w < kSeqThreads / 32; ++w) { tot.x += buf[w].x; tot.y += buf[w].y; }
        return tot;
    };
    float2 sum = zero;
#pragma unroll
    for (int i = 0; i < kPairs; ++i) { sum.x += v[i].x + v[i].y; sum.y += pv[i].x + pv[i].y; }
    sum = block_sum2(sum, red_mean);
    const float mean = sum.x / D, pmean = sum.y / D;
    float2 sq = zero;
#pragma unroll
    for (int i = 0; i < kPairs; ++i) {
        if (2 * (threadIdx.x + i * kSeqThreads) < D) {
            const float c0 = v[i].x - mean, c1 = v[i].y - mean, p0 = pv[i].x - pmean, p1 = pv[i].y - pmean;
            sq.x += c0 * c0 + c1 * c1;
            sq.y += p0 * p0 + p1 * p1;
        }
    }
    sq = block_sum2(sq, red_var);
    const float inv = 1.0f / sqrtf(sq.x / D + 1e-5f), pinv = 1.0f / sqrtf(sq.y / D + 1e-5f);
#pragma unroll
    for (int i = 0; i < kPairs; ++i) {
        const int d = 2 * (threadIdx.x + i * kSeqThreads);
        if (d >= D) continue;
        const float2 lw = __ldg(reinterpret_cast<const float2*>(a.ln_w + d)), lb = __ldg(reinterpret_cast<const float2*>(a.ln_b + d));
        v[i].x = (v[i].x - mean) * inv * lw.x + lb.x;
        v[i].y = (v[i].y - mean) * inv * lw.y + lb.y;
        if (t > 0) {                    // t == 0: pv already is a normalised row (or zeros)
            pv[i].x = (pv[i].x - pmean) * pinv * lw.x + lb.x;
            pv[i].y = (pv[i].y - pmean) * pinv * lw.y + lb.y;
        }
    }
#pragma unroll
    for (int i = 0; i < kPairs; ++i) {
        const int d = 2 * (threadIdx.x + i * kSeqThreads);
        if (d < D && t == a.T - 1) *reinterpret_cast<float2*>(a.shift_out + static_cast<size_t>(b) * D + d) = v[i];
        pv[i].x -= v[i].x;                     // xx = prev - cur
        pv[i].y -= v[i].y;
    }
    for (int m = 0; m < a.n_mix; ++m) {
        float2 val[kPairs];
        float amax = 0.f;
#pragma unroll
        for (int i = 0; i < kPairs; ++i) {
            const int d = 2 * (threadIdx.x + i * kSeqThreads);
            val[i] = zero;
            if (d < D) {
                const float2 mx = __ldg(reinterpret_cast<const float2*>(a.mix + static_cast<size_t>(m) * D + d));
                val[i].x = v[i].x + pv[i].x * mx.x;
                val[i].y = v[i].y + pv[i].y * mx.y;
                amax = fmaxf(amax, fmaxf(fabsf(val[i].x), fabsf(val[i].y)));
            }
        }
        const int mode = a.mode[m];
        float sc = 1.f;
        if (m == 0 && a.n2 != nullptr) {
            float q = 0.f;
#pragma unroll
            for (int i = 0; i < kPairs; ++i) q += val[i].x * val[i].x + val[i].y * val[i].y;
            q = block_sum(q, red);
            if (threadIdx.x == 0) a.n2[tok] = q;
        }
        if (mode & kPrepAmax) {
            amax = block_max(amax, red);
            if (threadIdx.x == 0) a.scale[m][tok] = amax;
        }
        if (mode & kPrepScaled) {
            amax = block_max(amax, red);
            int e = 0;
            if (amax > 0.f && amax < INFINITY) frexpf(amax, &e);
            sc = ldexpf(1.f, 14 - e);
            if (threadIdx.x == 0) a.scale[m][tok] = sc;
        }
#pragma unroll
        for (int i = 0; i < kPairs; ++i) {
            const int d = 2 * (threadIdx.x + i * kSeqThreads);
            if (d >= D) continue;
            if (mode & kPrepScaled)
                *reinterpret_cast<__half2*>(a.x16[m] + tok * (D + 64) + d) = __floats2half2_rn(val[i].x * sc, val[i].y * sc);
            if (mode & kPrepSplit) {
                const __half2 hi = __floats2half2_rn(val[i].x, val[i].y);
                const float2 hf = __half22float2(hi);
                __half* o = a.split[m] + tok * 2 * D + d;
                *reinterpret_cast<__half2*>(o) = hi;
                *reinterpret_cast<__half2*>(o + D) = __floats2half2_rn(val[i].x - hf.x, val[i].y - hf.y);
            }
            if (mode & kPrepF32) *reinterpret_cast<float2*>(a.f32[m] + tok * D + d) = val[i];
        }
    }
}

// The same for few tokens and D a multiple of 256: a CTA per token (or run of tokens) and mix, so that the
// mixes run side by side; D / 8 threads own 8 consecutive columns each (16-byte stores of the fp16 forms),
// parameters and lerp vector loaded before the launch wait.  Bound: the latency of the two sums.
constexpr int kSeqVecWarps = 16;
__device__ __forceinline__ void prep_load8(const float* p, float (&o)[8]) {
    const float4 x = *reinterpret_cast<const float4*>(p), y = *reinterpret_cast<const float4*>(p + 4);
    o[0] = x.x; o[1] = x.y; o[2] = x.z; o[3] = x.w; o[4] = y.x; o[5] = y.y; o[6] = y.z; o[7] = y.w;
}
__device__ __forceinline__ void prep_load8cg(const float* p, float (&o)[8]) {
    const float4 x = __ldcg(reinterpret_cast<const float4*>(p)), y = __ldcg(reinterpret_cast<const float4*>(p) + 1);
    o[0] = x.x; o[1] = x.y; o[2] = x.z; o[3] = x.w; o[4] = y.x; o[5] = y.y; o[6] = y.z; o[7] = y.w;
}
__device__ __forceinline__ void prep_store8(float* p, const float (&v)[8]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ uint4 prep_pack8(const float (&v)[8]) {
    uint4 r;
    __half2 h;
    h = __floats2half2_rn(v[0], v[1]); r.x = *reinterpret_cast<uint32_t*>(&h);
    h = __floats2half2_rn(v[2], v[3]); r.y = *reinterpret_cast<uint32_t*>(&h);
    h = __floats2half2_rn(v[4], v[5]); r.z = *reinterpret_cast<uint32_t*>(&h);
    h = __floats2half2_rn(v[6], v[7]); r.w = *reinterpret_cast<uint32_t*>(&h);
    return r;
}
__device__ __forceinline__ float warp_add(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}
// power of two with |x| * 2^s <= 2^14 for max|x| = amax
__device__ __forceinline__ float prep_scale(float amax) {
    int e = 0;
    if (amax > 0.f && amax < INFINITY) frexpf(amax, &e);
    return ldexpf(1.f, 14 - e);
}
// 8 columns of mix row m of token tok in the forms `mode` selects
__device__ __forceinline__ void prep_emit8(const SeqPrepArgs& a, int m, int mode, long long tok, int d0, float (&o)[8], float sc) {
    const int D = a.D;
    if (mode & kPrepF32) prep_store8(a.f32[m] + tok * D + d0, o);
    if (mode & kPrepSplit) {
        float lo[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) lo[i] = o[i] - __half2float(__float2half_rn(o[i]));
        __half* p = a.split[m] + tok * 2 * D + d0;
        *reinterpret_cast<uint4*>(p) = prep_pack8(o);
        *reinterpret_cast<uint4*>(p + D) = prep_pack8(lo);
    }
    if (mode & kPrepScaled) {
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] *= sc;
        *reinterpret_cast<uint4*>(a.x16[m] + tok * (D + 64) + d0) = prep_pack8(o);
    }
}

// CLUSTER: the CTAs of a token's mixes form a cluster, so that the shift state can be updated in place: it is
// written once all of them have read it.
template <bool CLUSTER>
__global__ void __launch_bounds__(kSeqVecWarps * 32) seq_prep_vec_kernel(const SeqPrepArgs a, long long n_tokens, int run) {
    __shared__ float red_s[kSeqVecWarps], red_q[kSeqVecWarps];
    __shared__ float2 red_m[kSeqVecWarps];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
    const int D = a.D, d0 = tid * 8, m = blockIdx.y, mode = a.mode[m];
    const long long tok0 = static_cast<long long>(blockIdx.x) * run, tok1 = min(tok0 + run, n_tokens);
    float lw[8], lb[8], mx[8];
    prep_load8(a.ln_w + d0, lw);
    prep_load8(a.ln_b + d0, lb);
    if (a.mix != nullptr) prep_load8(a.mix + static_cast<size_t>(m) * D + d0, mx);
    else {
#pragma unroll
        for (int i = 0; i < 8; ++i) mx[i] = 0.f;
    }
    const bool want_n2 = a.n2 != nullptr && m == 0, want_max = (mode & (kPrepScaled | kPrepAmax | kPrepPair)) != 0;
    pdl_launch_dependents();
    pdl_wait();
    if (m == 0)
        for (long long t = tok0 + tid; t < tok1; t += blockDim.x) {
            if (a.zero_a != nullptr) a.zero_a[t] = 0.f;
            if (a.zero_b != nullptr) a.zero_b[t] = 0.f;
        }
    // two-pass LayerNorm; the barriers of the two sums also separate the uses of each buffer
    auto normalise = [&](float (&y)[8]) {
        float s = warp_add(((y[0] + y[1]) + (y[2] + y[3])) + ((y[4] + y[5]) + (y[6] + y[7])));
        if (lane == 0) red_s[warp] = s;
        __syncthreads();
        s = 0.f;
        for (int w = 0; w < nw; ++w) s += red_s[w];
        const float mean = s / D;
        float q = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) { const float c = y[i] - mean; q = fmaf(c, c, q); }
        q = warp_add(q);
        if (lane == 0) red_q[warp] = q;
        __syncthreads();
        q = 0.f;
        for (int w = 0; w < nw; ++w) q += red_q[w];
        const float inv = 1.0f / sqrtf(q / D + 1e-5f);
#pragma unroll
        for (int i = 0; i < 8; ++i) y[i] = (y[i] - mean) * inv * lw[i] + lb[i];
    };
    float nx[8], pv[8];
    prep_load8cg(a.x + tok0 * D + d0, nx);
    int t = static_cast<int>(tok0 % a.T), b = static_cast<int>(tok0 / a.T);
    if (t > 0) {
        prep_load8cg(a.x + (tok0 - 1) * D + d0, pv);
        normalise(pv);
    }
    for (long long tok = tok0; tok < tok1; ++tok) {
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = nx[i];
        if (tok + 1 < tok1) prep_load8cg(a.x + (tok + 1) * D + d0, nx);
        if (t == 0) {
            if (a.shift_in) prep_load8cg(a.shift_in + static_cast<size_t>(b) * D + d0, pv);
            else {
#pragma unroll
                for (int i = 0; i < 8; ++i) pv[i] = 0.f;
            }
        }
        if (CLUSTER) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        normalise(v);
        if (CLUSTER) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (t == a.T - 1 && m == 0 && a.shift_out != nullptr) prep_store8(a.shift_out + static_cast<size_t>(b) * D + d0, v);
        float o[8], am = 0.f, n2 = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            o[i] = v[i] + (pv[i] - v[i]) * mx[i];
            am = fmaxf(am, fabsf(o[i]));
            n2 = fmaf(o[i], o[i], n2);
            pv[i] = v[i];
        }
        float sc = 1.f;
        if (want_max || want_n2) {
#pragma unroll
            for (int q = 16; q > 0; q >>= 1) {
                am = fmaxf(am, __shfl_xor_sync(0xFFFFFFFFu, am, q));
                n2 += __shfl_xor_sync(0xFFFFFFFFu, n2, q);
            }
            if (lane == 0) red_m[warp] = make_float2(am, n2);
            __syncthreads();
            n2 = 0.f;
            for (int w = 0; w < nw; ++w) { am = fmaxf(am, red_m[w].x); n2 += red_m[w].y; }
            sc = prep_scale(am);
            if (tid == 0) {
                if (want_n2) a.n2[tok] = n2;
                if (mode & (kPrepScaled | kPrepAmax)) a.scale[m][tok] = (mode & kPrepScaled) ? sc : am;
            }
        }
        if (mode & kPrepPair) {                          // the mode goes alone or with kPrepF32
            float s1, u1, q[8];
            sb_scale(am, s1, u1);
            if (tid == 0) a.pair[m].unscale[tok] = u1;
#pragma unroll
            for (int i = 0; i < 8; ++i) q[i] = o[i] * s1;
            sb_store_pair(a.pair[m], static_cast<int>(tok), static_cast<int>(n_tokens), tid, q);
        }
        prep_emit8(a, m, mode, tok, d0, o, sc);
        if (++t == a.T) { t = 0; ++b; }
    }
}

// One token of each stream, the shift state in place: all mixes of a token in one CTA, which holds the row and the state it
// replaces.  Bound: the latency of three block reductions (two sums, the maxima of all mixes together) and of a thread's 6 x 8 columns
// out; the form of many streams, see the dispatch.
__global__ void __launch_bounds__(kSeqVecWarps * 32) seq_prep_step_kernel(const SeqPrepArgs a) {
    constexpr int M = 6;
    __shared__ float red_s[kSeqVecWarps], red_q[kSeqVecWarps], red_n[kSeqVecWarps], red_m[kSeqVecWarps][M];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
    const int D = a.D, d0 = tid * 8;
    const long long tok = blockIdx.x;
    float lw[8], lb[8], mx[M][8];
    prep_load8(a.ln_w + d0, lw);
    prep_load8(a.ln_b + d0, lb);
#pragma unroll
    for (int m = 0; m < M; ++m)
        if (m < a.n_mix) prep_load8(a.mix + static_cast<size_t>(m) * D + d0, mx[m]);
    pdl_launch_dependents();
    pdl_wait();
    if (tid == 0) {
        if (a.zero_a != nullptr) a.zero_a[tok] = 0.f;
        if (a.zero_b != nullptr) a.zero_b[tok] = 0.f;
    }
    float v[8], pv[8];
    prep_load8cg(a.x + tok * D + d0, v);
    prep_load8cg(a.shift_in + tok * D + d0, pv);
    float r = warp_add(((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7])));
    if (lane == 0) red_s[warp] = r;
    __syncthreads();
    r = 0.f;
    for (int w = 0; w < nw; ++w) r += red_s[w];
    const float mean = r / D;
    r = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) { const float c = v[i] - mean; r = fmaf(c, c, r); }
    r = warp_add(r);
    if (lane == 0) red_q[warp] = r;
    __syncthreads();
    r = 0.f;
    for (int w = 0; w < nw; ++w) r += red_q[w];
    const float inv = 1.0f / sqrtf(r / D + 1e-5f);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        v[i] = (v[i] - mean) * inv * lw[i] + lb[i];
        pv[i] -= v[i];                                   // xx = prev - cur
    }
    prep_store8(a.shift_out + tok * D + d0, v);
    float am[M], n2 = 0.f;
#pragma unroll
    for (int m = 0; m < M; ++m) {
        am[m] = 0.f;
        if (m >= a.n_mix) continue;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float o = v[i] + pv[i] * mx[m][i];
            am[m] = fmaxf(am[m], fabsf(o));
            if (m == 0) n2 = fmaf(o, o, n2);
        }
    }
#pragma unroll
    for (int m = 0; m < M; ++m) {
#pragma unroll
        for (int q = 16; q > 0; q >>= 1) am[m] = fmaxf(am[m], __shfl_xor_sync(0xFFFFFFFFu, am[m], q));
        if (lane == 0) red_m[warp][m] = am[m];
    }
    n2 = warp_add(n2);
    if (lane == 0) red_n[warp] = n2;
    __syncthreads();
    if (a.n2 != nullptr && tid == 0) {
        n2 = 0.f;
        for (int w = 0; w < nw; ++w) n2 += red_n[w];
        a.n2[tok] = n2;
    }
#pragma unroll
    for (int m = 0; m < M; ++m) {
        if (m >= a.n_mix) break;
        const int mode = a.mode[m];
        float o[8], sc = 1.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = v[i] + pv[i] * mx[m][i];
        if (mode & (kPrepScaled | kPrepAmax | kPrepPair)) {
            float top = 0.f;
            for (int w = 0; w < nw; ++w) top = fmaxf(top, red_m[w][m]);
            sc = prep_scale(top);
            if (tid == 0 && (mode & (kPrepScaled | kPrepAmax))) a.scale[m][tok] = (mode & kPrepScaled) ? sc : top;
            if (mode & kPrepPair) {                      // the mode goes alone or with kPrepF32
                float s1, u1, q[8];
                sb_scale(top, s1, u1);
                if (tid == 0) a.pair[m].unscale[tok] = u1;
#pragma unroll
                for (int i = 0; i < 8; ++i) q[i] = o[i] * s1;
                sb_store_pair(a.pair[m], static_cast<int>(tok), static_cast<int>(gridDim.x), tid, q);
            }
        }
        prep_emit8(a, m, mode, tok, d0, o, sc);
    }
}

// Many tokens, D a multiple of 512: 64 threads per token (a barrier of two warps, not of a CTA, behind
// every sum), four tokens side by side in a CTA that share the parameters and lerp vectors in shared
// memory; a group walks a run of consecutive tokens and keeps the normalised row for its successor.
// Bound: HBM writes of the six rows.
constexpr int kPrepGroup = 64, kPrepGroups = 4;
template <int CH>      // chunks of 512 columns
__global__ void __launch_bounds__(kPrepGroup * kPrepGroups, 2) seq_prep_group_kernel(const SeqPrepArgs a, long long n_tokens, int run) {
    extern __shared__ __align__(16) float params[];      // [2 + n_mix][D]
    __shared__ float red_s[kPrepGroups][2], red_q[kPrepGroups][2];
    __shared__ float red_m[kPrepGroups][2][8];
    constexpr int D = CH * 512;
    const int grp = threadIdx.x / kPrepGroup, tid = threadIdx.x % kPrepGroup, wp = tid >> 5, lane = tid & 31, n_mix = a.n_mix;
    for (int i = threadIdx.x; i < D / 4; i += kPrepGroup * kPrepGroups) {
        reinterpret_cast<float4*>(params)[i] = __ldg(reinterpret_cast<const float4*>(a.ln_w) + i);
        reinterpret_cast<float4*>(params + D)[i] = __ldg(reinterpret_cast<const float4*>(a.ln_b) + i);
        for (int m = 0; m < n_mix; ++m)
            reinterpret_cast<float4*>(params + (2 + m) * D)[i] = __ldg(reinterpret_cast<const float4*>(a.mix + static_cast<size_t>(m) * D) + i);
    }
    bool any_max = a.n2 != nullptr;
    for (int m = 0; m < n_mix; ++m) any_max |= (a.mode[m] & (kPrepScaled | kPrepAmax)) != 0;
    pdl_launch_dependents();
    __syncthreads();
    pdl_wait();
    auto group_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "n"(kPrepGroup) : "memory"); };
    const long long tok0 = (static_cast<long long>(blockIdx.x) * kPrepGroups + grp) * run, tok1 = min(tok0 + run, n_tokens);
    if (tok0 >= tok1) return;
    for (long long t = tok0 + tid; t < tok1; t += kPrepGroup) {
        if (a.zero_a != nullptr) a.zero_a[t] = 0.f;
        if (a.zero_b != nullptr) a.zero_b[t] = 0.f;
    }
    auto load_row = [&](const float* row, float (&y)[CH][8]) {
#pragma unroll
        for (int c = 0; c < CH; ++c) prep_load8cg(row + 8 * (tid + kPrepGroup * c), y[c]);
    };
    auto normalise = [&](float (&y)[CH][8]) {
        float s = 0.f;
#pragma unroll
        for (int c = 0; c < CH; ++c)
#pragma unroll
            for (int i = 0; i < 8; ++i) s += y[c][i];
        s = warp_add(s);
        if (lane == 0) red_s[grp][wp] = s;
        group_sync();
        const float mean = (red_s[grp][0] + red_s[grp][1]) / D;
        float q = 0.f;
#pragma unroll
        for (int c = 0; c < CH; ++c)
#pragma unroll
            for (int i = 0; i < 8; ++i) { const float e = y[c][i] - mean; q = fmaf(e, e, q); }
        q = warp_add(q);
        if (lane == 0) red_q[grp][wp] = q;
        group_sync();
        const float inv = 1.0f / sqrtf((red_q[grp][0] + red_q[grp][1]) / D + 1e-5f);
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            float w[8], b[8];
            prep_load8(params + 8 * (tid + kPrepGroup * c), w);
            prep_load8(params + D + 8 * (tid + kPrepGroup * c), b);
#pragma unroll
            for (int i = 0; i < 8; ++i) y[c][i] = (y[c][i] - mean) * inv * w[i] + b[i];
        }
    };
    float v[CH][8], pv[CH][8];
    int t = static_cast<int>(tok0 % a.T), b = static_cast<int>(tok0 / a.T);
    if (t > 0) load_row(a.x + (tok0 - 1) * D, pv);
    load_row(a.x + tok0 * D, v);
    if (t > 0) normalise(pv);
    for (long long tok = tok0;;) {
        if (t == 0) {
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                if (a.shift_in) prep_load8(a.shift_in + static_cast<size_t>(b) * D + 8 * (tid + kPrepGroup * c), pv[c]);
                else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) pv[c][i] = 0.f;
                }
            }
        }
        normalise(v);
        if (t == a.T - 1) {
#pragma unroll
            for (int c = 0; c < CH; ++c) prep_store8(a.shift_out + static_cast<size_t>(b) * D + 8 * (tid + kPrepGroup * c), v[c]);
        }
#pragma unroll
        for (int c = 0; c < CH; ++c)
#pragma unroll
            for (int i = 0; i < 8; ++i) pv[c][i] -= v[c][i];     // xx = prev - cur
        if (any_max) {
            float n2 = 0.f;
            for (int m = 0; m < n_mix; ++m) {
                float x = 0.f;
#pragma unroll
                for (int c = 0; c < CH; ++c) {
                    float mx[8];
                    prep_load8(params + (2 + m) * D + 8 * (tid + kPrepGroup * c), mx);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float o = v[c][i] + pv[c][i] * mx[i];
                        x = fmaxf(x, fabsf(o));
                        if (m == 0) n2 = fmaf(o, o, n2);
                    }
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xFFFFFFFFu, x, o));
                if (lane == 0) red_m[grp][wp][m] = x;
            }
            n2 = warp_add(n2);
            if (lane == 0) red_m[grp][wp][6] = n2;
            group_sync();
            if (a.n2 != nullptr && tid == 0) a.n2[tok] = red_m[grp][0][6] + red_m[grp][1][6];
        }
        for (int m = 0; m < n_mix; ++m) {
            const int mode = a.mode[m];
            float sc = 1.f;
            if (mode & (kPrepScaled | kPrepAmax)) {
                const float am = fmaxf(red_m[grp][0][m], red_m[grp][1][m]);
                sc = prep_scale(am);
                if (tid == 0) a.scale[m][tok] = (mode & kPrepScaled) ? sc : am;
            }
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                const int d0 = 8 * (tid + kPrepGroup * c);
                float mx[8], o[8];
                prep_load8(params + (2 + m) * D + d0, mx);
#pragma unroll
                for (int i = 0; i < 8; ++i) o[i] = v[c][i] + pv[c][i] * mx[i];
                prep_emit8(a, m, mode, tok, d0, o, sc);
            }
        }
        if (++tok == tok1) break;
#pragma unroll
        for (int c = 0; c < CH; ++c)
#pragma unroll
            for (int i = 0; i < 8; ++i) pv[c][i] = v[c][i];
        load_row(a.x + tok * D, v);
        if (++t == a.T) { t = 0; ++b; }
    }
}

template <int CH>
static cudaError_t launch_prep_group(const SeqPrepArgs& a, long long n_tokens, cudaStream_t s) {
    const size_t smem = sizeof(float) * (2 + a.n_mix) * CH * 512;
    cudaError_t e = cudaFuncSetAttribute(seq_prep_group_kernel<CH>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(8 * sizeof(float) * CH * 512));
    if (e != cudaSuccess) return e;
    const long long wave = 148 * 2 * kPrepGroups;                // groups resident at once
    const int run = static_cast<int>((n_tokens + wave - 1) / wave);
    const long long groups = (n_tokens + run - 1) / run;
    return launch_pdl(seq_prep_group_kernel<CH>, dim3(static_cast<unsigned>((groups + kPrepGroups - 1) / kPrepGroups)),
                      dim3(kPrepGroup * kPrepGroups), smem, s, a, n_tokens, run);
}

int launch_seq_prep(const SeqPrepArgs& a, long long n_tokens, cudaStream_t s) {
    cudaError_t e;
    // rows on 16-byte boundaries throughout, as the vector forms read and write them
    bool vec = a.D % 256 == 0 && a.D <= kSeqVecWarps * 256 && aligned(a.x, 16) && aligned(a.ln_w, 16) && aligned(a.ln_b, 16) &&
               aligned(a.mix, 16) && aligned(a.shift_in, 16) && aligned(a.shift_out, 16);
    for (int m = 0; m < a.n_mix; ++m) vec = vec && aligned(a.x16[m], 16) && aligned(a.split[m], 16) && aligned(a.f32[m], 16);
    bool pair = a.mix == nullptr;
    for (int m = 0; m < a.n_mix; ++m) pair = pair || (a.mode[m] & kPrepPair) != 0;
    const bool in_place = a.shift_out != nullptr && a.shift_in == a.shift_out;
    RWKVQ_REQUIRE(vec || !pair, RWKVQ_E_ALIGN, "seq_ln_shift_mix_prep: D %d, rows on 16-byte boundaries", a.D);
    RWKVQ_REQUIRE(aligned(a.x, 8) && aligned(a.ln_w, 8) && aligned(a.ln_b, 8) && aligned(a.mix, 8) && aligned(a.shift_in, 8) && aligned(a.shift_out, 8),
                  RWKVQ_E_ALIGN, "seq_ln_shift_mix_prep: 8-byte aligned rows required");       // the scalar form reads pairs
    RWKVQ_REQUIRE(!in_place || a.T == 1, RWKVQ_E_SHAPE, "seq_ln_shift_mix_prep: the shift state in place needs T = 1");
    // (in place: the scalar and the step form have a token's mixes in one CTA, the vector form in one cluster)
    // Which form (us, scalar / vector / groups, six mixes and one):
    //   few      the vector form while its CTAs, one per token and mix, are one wave: two an SM up to 2048 columns, one above (six
    //            mixes: still ahead at two a slot).  2048 columns, 49 tokens: 7.6 / 4.1, one mix 296: 4.8 / 4.2; 2304, 231: 4.9 / 7.1
    //   many     groups where D is a multiple of 512 up to 3072 (above, two rows a thread no longer fit its registers: 4096 columns,
    //            8192 tokens 245 / 711 / 319), from where one wave of the scalar form (3 CTAs an SM) ends.  8192 tokens, six
    //            mixes: 1536 163 / 240 / 74, 2048 174 / 276 / 102, 2560 186 / 542 / 132; 512 tokens: 16.7 / 23.7 / 12.1, 17.9 / 26.8 / 13.1,
    //            19.4 / 49 / 18.9, one mix 7.4 / 6.7 / 6.4, 8.0 / 7.7 / 7.2, 8.5 / 13.8 / 9.7
    //   other widths: the vector form where it is narrow (768: 139 / 91, one mix 60 / 20; 1280, one mix 63 / 41), else the scalar one
    //            (2304, 8192 tokens: 177 / 521; 1792: 166 / 260)
    const int wave = a.n_mix == 1 && a.D > 2048 ? 148 : 2 * 148;
    const bool few = n_tokens * a.n_mix <= wave || pair || in_place;
    const long long groups_from = a.D <= 1536 ? 0 : a.D > 2048 ? 1024 : a.n_mix > 1 ? 200 : 445;
    if (vec && !few && a.D % 512 == 0 && a.D <= 3072 && n_tokens >= groups_from) {
        switch (a.D / 512) {
            case 1: e = launch_prep_group<1>(a, n_tokens, s); break;
            case 2: e = launch_prep_group<2>(a, n_tokens, s); break;
            case 3: e = launch_prep_group<3>(a, n_tokens, s); break;
            case 4: e = launch_prep_group<4>(a, n_tokens, s); break;
            case 5: e = launch_prep_group<5>(a, n_tokens, s); break;
            default: e = launch_prep_group<6>(a, n_tokens, s); break;
        }
    } else if (vec && in_place && a.n_mix > 1 && a.mix != nullptr && 2 * n_tokens * a.n_mix > 3 * 148 * std::max(1, 65536 / (112 * a.D / 8))) {
        // A CTA per token instead of a cluster of one per mix, which normalises the row six times, from where the clusters are one
        // and a half waves (by registers two CTAs an SM up to 2304 columns, one above: from 75 streams on at 2048 and 2304, from 38 at
        // 2560).  us a step, cluster / this: 1.5B 16 streams 1760 / 1855, 64 2447 / 2485, 100 3369 / 3315, 200 5049 / 4810; 2.9B 32 streams
        // 3418 / 3453, 64 4492 / 4281, 128 7074 / 6565
        e = launch_pdl(seq_prep_step_kernel, dim3(static_cast<unsigned>(n_tokens)), dim3(a.D / 8), 0, s, a);
    } else if (vec && in_place && a.n_mix > 1) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(static_cast<unsigned>(n_tokens), a.n_mix);
        cfg.blockDim = dim3(a.D / 8);
        cfg.stream = s;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = a.n_mix; attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = pdl_enabled() ? 2 : 1;
        e = cudaLaunchKernelEx(&cfg, seq_prep_vec_kernel<true>, a, n_tokens, 1);
    } else if (vec && (few || a.D <= (a.n_mix == 1 ? 1280 : 1024))) {
        long long run = in_place ? 1 : n_tokens * a.n_mix / (148 * 8);
        run = run < 1 ? 1 : run > 16 ? 16 : run;
        e = launch_pdl(seq_prep_vec_kernel<false>, dim3(static_cast<unsigned>((n_tokens + run - 1) / run), a.n_mix), dim3(a.D / 8), 0, s, a, n_tokens,
                       static_cast<int>(run));
    } else {
        e = launch_pdl(seq_ln_shift_mix_prep_kernel, dim3(static_cast<unsigned>(n_tokens)), dim3(kSeqThreads), 0, s, a);
    }
    if (e != cudaSuccess) return fail(RWKVQ_E_LAUNCH, "seq_ln_shift_mix_prep: %s", cudaGetErrorString(e));
    return RWKVQ_OK;
}

struct TmixPreArgs {
    const float *k, *v, *yw, *ya, *yv, *v_first;     // [N, D]; yv / v_first null on layer 0
    const float *w0, *a0, *v0, *k_k, *k_a;           // [D]
    float *w, *k2, *v2, *na, *nb;                     // [N, D]: decay, k', v', -kk, kk * a
    long long n_pairs;                                // N * H
    int H;
};

// One warp per (token, head): lane owns the channel pair 2 lane, 2 lane + 1 of the head (64-bit
// loads and stores).
__global__ void __launch_bounds__(256) seq_tmix_pre_kernel(const TmixPreArgs p) {
    const long long pair = blockIdx.x * 8ll + (threadIdx.x >> 5);
    pdl_launch_dependents();
    pdl_wait();
    if (pair >= p.n_pairs) return;
    const int lane = threadIdx.x & 31, hd = static_cast<int>(pair % p.H);
    const size_t i = static_cast<size_t>(pair) * 64 + 2 * lane;
    const int c = hd * 64 + 2 * lane;
    auto ld2 = [](const float* q, size_t at) { return *reinterpret_cast<const float2*>(q + at); };
    auto st2 = [](float* q, size_t at, float x, float y) { *reinterpret_cast<float2*>(q + at) = make_float2(x, y); };
    const float2 k = ld2(p.k, i), yw = ld2(p.yw, i), ya = ld2(p.ya, i);
    float2 v = ld2(p.v, i);
    const float2 w0 = ld2(p.w0, c), a0 = ld2(p.a0, c), kk_w = ld2(p.k_k, c), ka_w = ld2(p.k_a, c);
    if (p.yv) {
        const float2 yv = ld2(p.yv, i), vf = ld2(p.v_first, i), v0 = ld2(p.v0, c);
        v.x = v.x + (vf.x - v.x) * sigmoidf_(yv.x + v0.x);
        v.y = v.y + (vf.y - v.y) * sigmoidf_(yv.y + v0.y);
    }
    st2(p.w, i, expf(-0.606531f * sigmoidf_(yw.x + w0.x)), expf(-0.606531f * sigmoidf_(yw.y + w0.y)));
    const float ax = sigmoidf_(ya.x + a0.x), ay = sigmoidf_(ya.y + a0.y);
    const float kx = k.x * kk_w.x, ky = k.y * kk_w.y;
    float n2 = kx * kx + ky * ky;
    st2(p.k2, i, k.x * (1.0f + (ax - 1.0f) * ka_w.x), k.y * (1.0f + (ay - 1.0f) * ka_w.y));
    st2(p.v2, i, v.x, v.y);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n2 += __shfl_xor_sync(0xFFFFFFFFu, n2, o);
    const float inv = 1.0f / sqrtf(n2 + 1e-12f);
    st2(p.na, i, -(kx * inv), -(ky * inv));
    st2(p.nb, i, kx * inv * ax, ky * inv * ay);
}

// x fp32 [rows, cols] -> out fp16 [rows, 2 * cols] = [hi | lo] with hi = fp16(x), lo = fp16(x - hi):
// a product of [hi | lo] with a matrix stacked twice equals x @ W to ~2^-22 relative while running
// on the fp16 tensor cores.  One pass over x.
__global__ void __launch_bounds__(256) split_fp16_kernel(const float* __restrict__ x, __half* __restrict__ out,
                                                         long long n_pairs, int cols) {
    const int half_cols = cols >> 1;
    for (long long i = blockIdx.x * 256ll + threadIdx.x; i < n_pairs; i += gridDim.x * 256ll) {
        const long long r = i / half_cols;
        const int c = static_cast<int>(i % half_cols) * 2;
        const float2 v = *reinterpret_cast<const float2*>(x + r * cols + c);
        const __half2 hi = __floats2half2_rn(v.x, v.y);
        const float2 hf = __half22float2(hi);
        const __half2 lo = __floats2half2_rn(v.x - hf.x, v.y - hf.y);
        __half* o = out + r * 2 * cols + c;
        *reinterpret_cast<__half2*>(o) = hi;
        *reinterpret_cast<__half2*>(o + cols) = lo;
    }
}

}  // namespace rwkvq

using namespace rwkvq;

extern "C" {

int rwkvq_seq_ln_shift_mix(const float* x, const float* ln_w, const float* ln_b, const float* shift_in,
                           const float* mix, int n_mix, float* out, float* shift_out, int B, int T, int D,
                           void* stream) {
    RWKVQ_REQUIRE(x && ln_w && ln_b && out && shift_out, RWKVQ_E_NULL, "rwkvq_seq_ln_shift_mix: null pointer");
    RWKVQ_REQUIRE(B >= 1 && T >= 1 && D >= 1 && D <= kSeqThreads * kSeqPer, RWKVQ_E_LIMIT,
                  "rwkvq_seq_ln_shift_mix: B=%d T=%d D=%d (D at most %d)", B, T, D, kSeqThreads * kSeqPer);
    RWKVQ_REQUIRE((n_mix == 1 || n_mix == 6) && mix, RWKVQ_E_SHAPE, "rwkvq_seq_ln_shift_mix: n_mix %d (1 or 6)", n_mix);
    const long long n = static_cast<long long>(B) * T;
    RWKVQ_REQUIRE(n < (1ll << 31), RWKVQ_E_LIMIT, "rwkvq_seq_ln_shift_mix: %lld tokens", n);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (n_mix == 6)
        seq_ln_shift_mix_kernel<6><<<static_cast<unsigned>(n), kSeqThreads, 0, s>>>(x, ln_w, ln_b, shift_in, mix, out, shift_out, T, D, n);
    else
        seq_ln_shift_mix_kernel<1><<<static_cast<unsigned>(n), kSeqThreads, 0, s>>>(x, ln_w, ln_b, shift_in, mix, out, shift_out, T, D, n);
    return check_launch("rwkvq_seq_ln_shift_mix");
}

int rwkvq_seq_ln_shift_mix_prep(const float* x, const float* ln_w, const float* ln_b, const float* shift_in,
                                const float* mix, int n_mix, const int* modes, void* const* out_x16,
                                float* const* out_scale, void* const* out_split, float* const* out_f32,
                                float* shift_out, int B, int T, int D, void* stream) {
    RWKVQ_REQUIRE(x && ln_w && ln_b && mix && modes && shift_out, RWKVQ_E_NULL, "rwkvq_seq_ln_shift_mix_prep: null pointer");
    RWKVQ_REQUIRE(B >= 1 && T >= 1 && D >= 2 && D % 2 == 0 && D <= kSeqThreads * kSeqPer, RWKVQ_E_LIMIT,
                  "rwkvq_seq_ln_shift_mix_prep: B=%d T=%d D=%d (even, at most %d)", B, T, D, kSeqThreads * kSeqPer);
    RWKVQ_REQUIRE(n_mix >= 1 && n_mix <= 6, RWKVQ_E_SHAPE, "rwkvq_seq_ln_shift_mix_prep: n_mix %d (1..6)", n_mix);
    const long long n = static_cast<long long>(B) * T;
    RWKVQ_REQUIRE(n < (1ll << 31), RWKVQ_E_LIMIT, "rwkvq_seq_ln_shift_mix_prep: %lld tokens", n);
    RWKVQ_REQUIRE(aligned(x, 8) && aligned(ln_w, 8) && aligned(ln_b, 8) && aligned(mix, 8) && aligned(shift_in, 8) &&
                      aligned(shift_out, 8), RWKVQ_E_ALIGN, "rwkvq_seq_ln_shift_mix_prep: 8-byte aligned rows required");
    SeqPrepArgs a{};
    a.x = x; a.ln_w = ln_w; a.ln_b = ln_b; a.shift_in = shift_in; a.mix = mix; a.shift_out = shift_out;
    a.T = T; a.D = D; a.n_mix = n_mix;
    for (int m = 0; m < n_mix; ++m) {
        const int mode = modes[m];
        RWKVQ_REQUIRE(mode >= 1 && mode <= 7, RWKVQ_E_DTYPE, "rwkvq_seq_ln_shift_mix_prep: mode[%d] = %d", m, mode);
        a.mode[m] = mode;
        if (mode & kPrepScaled) {
            RWKVQ_REQUIRE(out_x16 && out_scale && out_x16[m] && out_scale[m] && aligned(out_x16[m], 16), RWKVQ_E_NULL,
                          "rwkvq_seq_ln_shift_mix_prep: scaled output %d missing or unaligned", m);
            a.x16[m] = static_cast<__half*>(out_x16[m]);
            a.scale[m] = out_scale[m];
        }
        if (mode & kPrepSplit) {
            RWKVQ_REQUIRE(out_split && out_split[m] && aligned(out_split[m], 4), RWKVQ_E_NULL,
                          "rwkvq_seq_ln_shift_mix_prep: split output %d missing or unaligned", m);
            a.split[m] = static_cast<__half*>(out_split[m]);
        }
        if (mode & kPrepF32) {
            RWKVQ_REQUIRE(out_f32 && out_f32[m] && aligned(out_f32[m], 8), RWKVQ_E_NULL,
                          "rwkvq_seq_ln_shift_mix_prep: fp32 output %d missing or unaligned", m);
            a.f32[m] = out_f32[m];
        }
    }
    int rc = launch_seq_prep(a, n, static_cast<cudaStream_t>(stream));
    return rc ? rc : check_launch("rwkvq_seq_ln_shift_mix_prep");
}

int rwkvq_seq_tmix_pre(const float* k, const float* v, const float* yw, const float* ya, const float* yv,
                       const float* v_first, const float* w0, const float* a0, const float* v0, const float* k_k,
                       const float* k_a, float* w, float* k2, float* v2, float* neg_kk, float* kk_a, int64_t n_tokens,
                       int H, void* stream) {
    RWKVQ_REQUIRE(k && v && yw && ya && w0 && a0 && k_k && k_a && w && k2 && v2 && neg_kk && kk_a, RWKVQ_E_NULL,
                  "rwkvq_seq_tmix_pre: null pointer");
    RWKVQ_REQUIRE((yv == nullptr) == (v_first == nullptr) && (yv == nullptr || v0 != nullptr), RWKVQ_E_NULL,
                  "rwkvq_seq_tmix_pre: yv, v_first and v0 go together");
    RWKVQ_REQUIRE(n_tokens >= 1 && H >= 1, RWKVQ_E_SHAPE, "rwkvq_seq_tmix_pre: n_tokens=%lld H=%d", (long long)n_tokens, H);
    for (const void* q : {(const void*)k, (const void*)v, (const void*)yw, (const void*)ya, (const void*)yv, (const void*)v_first,
                          (const void*)w0, (const void*)a0, (const void*)v0, (const void*)k_k, (const void*)k_a, (const void*)w,
                          (const void*)k2, (const void*)v2, (const void*)neg_kk, (const void*)kk_a})
        RWKVQ_REQUIRE(aligned(q, 8), RWKVQ_E_ALIGN, "rwkvq_seq_tmix_pre: 8-byte aligned arrays required");
    TmixPreArgs p{k, v, yw, ya, yv, v_first, w0, a0, v0, k_k, k_a, w, k2, v2, neg_kk, kk_a, n_tokens * H, H};
    const long long blocks = (p.n_pairs + 7) / 8;
    RWKVQ_REQUIRE(blocks < (1ll << 31), RWKVQ_E_LIMIT, "rwkvq_seq_tmix_pre: too many tokens");
    launch_pdl(seq_tmix_pre_kernel, dim3(static_cast<unsigned>(blocks)), dim3(256), 0, static_cast<cudaStream_t>(stream), p);
    return check_launch("rwkvq_seq_tmix_pre");
}

int rwkvq_split_fp16(const float* x, void* out_fp16, int64_t rows, int cols, void* stream) {
    RWKVQ_REQUIRE(x && out_fp16, RWKVQ_E_NULL, "rwkvq_split_fp16: null pointer");
    RWKVQ_REQUIRE(rows >= 1 && cols >= 2 && cols % 2 == 0, RWKVQ_E_SHAPE, "rwkvq_split_fp16: rows=%lld cols=%d (even)",
                  (long long)rows, cols);
    RWKVQ_REQUIRE(aligned(x, 8) && aligned(out_fp16, 4), RWKVQ_E_ALIGN, "rwkvq_split_fp16: x needs 8-byte, out 4-byte alignment");
    const long long n_pairs = rows * (cols / 2);
    long long blocks = (n_pairs + 255) / 256;
    if (blocks > 148 * 32) blocks = 148 * 32;
    split_fp16_kernel<<<static_cast<unsigned>(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        x, static_cast<__half*>(out_fp16), n_pairs, cols);
    return check_launch("rwkvq_split_fp16");
}

}  // extern "C"
