// Every kernel here may be launched programmatically (resident while its producer is
// still running), so values produced by earlier kernels are read with L2-coherent
// loads (__ldcg) after pdl_wait(); only weights and parameters use cached paths.
//
// Single-token decode step of a quantized RWKV-7 model: the glue kernels between
// the GEMVs and the host-side launch sequence (rwkvq_decode_step).
//
// Per layer (backends/metal/quant_model.py:638-728, 803-836):
//   ln_shift_mix   LN1 + token shift + the six lerps           -> xs[6][B][D]
//   linear x3      r, k, v projections (one fused launch; one stream: with the LoRA down projections)
//   lora pair      w1, a1, v1, g1, activation (tanh / - / - / sigmoid), w2, a2, v2, g2 (rwkvq_lora_mma.cu; the SIMT
//                  kernels of this file for odd shapes; one stream: inside its neighbours, rwkvq_lora_vec.cuh)
//   tmix_core      decay, gates, kk, k and v updates, WKV-7 step on the 64x64 state,
//                  group norm, bonus, gate                      -> og[B][D]
//   linear + add   output projection and residual
//   ln_shift_mix   LN2 + token shift + lerp                     -> xk[B][D]
//   linear + relu^2  ffn key;  linear + add  ffn value and residual
// Linears: one stream rwkvq_gemv_mma.cu, 2 to 8 rwkvq_gemv_batch.cu, from 9 on rwkvq_gemm_sb.cu (LayerNorms by
// rwkvq_seq.cu, rows as fp16 pairs).
#include <stdlib.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <utility>

#include "rwkvq_ahead.cuh"
#include "rwkvq_lora_vec.cuh"
#include "rwkvq_seq.cuh"

namespace rwkvq {

// LayerNorm of row b held as `per` values per thread (two-pass variance, eps 1e-5).
template <int PER>
__device__ __forceinline__ void layer_norm_row(float (&x)[PER], int D, const float* w, const float* b,
                                               float* red) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i) s += x[i];
    const float mean = block_sum(s, red) / D;
    float s2 = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int d = threadIdx.x + i * blockDim.x;
        const float c = (d < D) ? x[i] - mean : 0.f;
        s2 += c * c;
    }
    const float inv = 1.0f / sqrtf(block_sum(s2, red) / D + 1e-5f);
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int d = threadIdx.x + i * blockDim.x;
        if (d < D) x[i] = (x[i] - mean) * inv * w[d] + b[d];
    }
}

constexpr int kRowThreads = 256;
constexpr int kRowPer = 16;      // D <= 4096
constexpr int kLnVecThreads = 1024;      // a float4 of the row per thread

// Columns [32 g, 32 g + 32) of row R of an sb6 or sym table as exact fp32 values (the arithmetic of
// decode_element: separate multiply and add), with every load of the group issued before any use:
// 16 bytes of codes, the plane words, the scale record.  Requires 32 | cols and the natural alignment
// of the file buffers (rows of codes are multiples of 16 bytes).
__device__ __forceinline__ void decode_group32(const QView& t, size_t R, int g, float* out) {
    if (t.kind == RWKVQ_KIND_SB6) {
        const int nsb = t.cols >> 8, sbi = g >> 3, j = g & 7;
        const uint4 cw = *reinterpret_cast<const uint4*>(t.codes + R * (t.cols >> 1) + g * 16);
        const uint32_t h1 = t.qh ? *reinterpret_cast<const uint32_t*>(t.qh + R * (t.cols >> 3) + g * 4) : 0u;
        const uint32_t h2 = t.qh2 ? *reinterpret_cast<const uint32_t*>(t.qh2 + R * (t.cols >> 3) + g * 4) : 0u;
        const uint32_t* mp = reinterpret_cast<const uint32_t*>(t.qsqm + (R * nsb + sbi) * 12);
        const uint32_t m0 = mp[0], m1 = mp[1], m2 = mp[2];
        const float d = __half2float(t.d[R * nsb + sbi]), dm = __half2float(t.dm[R * nsb + sbi]);
        float sc, mn;
        sb6_scale_min(m0, m1, m2, j, d, dm, sc, mn);
        const uint32_t w[4] = {cw.x, cw.y, cw.z, cw.w};
#pragma unroll
        for (int k = 0; k < 16; ++k) {               // byte k: column k (low nibble), column k + 16 (high nibble)
            const uint32_t byte = (w[k >> 2] >> (8 * (k & 3))) & 0xFFu;
            const uint32_t lo = (byte & 0xFu) + 16u * ((h1 >> k) & 1u) + 32u * ((h2 >> k) & 1u);
            const uint32_t hi = (byte >> 4) + 16u * ((h1 >> (k + 16)) & 1u) + 32u * ((h2 >> (k + 16)) & 1u);
            out[k] = __fadd_rn(__fmul_rn(static_cast<float>(lo), sc), mn);
            out[k + 16] = __fadd_rn(__fmul_rn(static_cast<float>(hi), sc), mn);
        }
    } else {                                         // sym: two blocks of 16
        const int nb = t.cols >> 4, nsb = t.cols >> 8;
        const float d = __half2float(t.d[R * nsb + (g >> 3)]);
        const uint32_t qs2 = *reinterpret_cast<const unsigned short*>(t.qs + R * nb + 2 * g);
        float s[2];
#pragma unroll
        for (int b2 = 0; b2 < 2; ++b2)
            s[b2] = half_roundtrip(__fmul_rn(static_cast<float>(static_cast<int8_t>((qs2 >> (8 * b2)) & 0xFFu)), d));
        if (t.bits == 8) {
            const uint4* cp = reinterpret_cast<const uint4*>(t.codes + R * t.cols + g * 32);
            const uint4 c0 = cp[0], c1 = cp[1];
            const uint32_t w[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
            for (int k = 0; k < 32; ++k)
                out[k] = __fmul_rn(static_cast<float>(static_cast<int8_t>((w[k >> 2] >> (8 * (k & 3))) & 0xFFu)), s[k >> 4]);
        } else {
            const uint4 cw = *reinterpret_cast<const uint4*>(t.codes + R * (t.cols >> 1) + g * 16);
            const uint32_t h1 = t.qh ? *reinterpret_cast<const uint32_t*>(t.qh + R * (t.cols >> 3) + g * 4) : 0u;
            const uint32_t h2 = t.qh2 ? *reinterpret_cast<const uint32_t*>(t.qh2 + R * (t.cols >> 3) + g * 4) : 0u;
            const uint32_t w[4] = {cw.x, cw.y, cw.z, cw.w};
#pragma unroll
            for (int b2 = 0; b2 < 2; ++b2)
#pragma unroll
                for (int k = 0; k < 8; ++k) {        // block b2, byte k: column k (low nibble), column k + 8 (high nibble)
                    const uint32_t byte = (w[2 * b2 + (k >> 2)] >> (8 * (k & 3))) & 0xFFu;
                    const int c_lo = 16 * b2 + k, c_hi = c_lo + 8;
                    const int lo = static_cast<int>((byte & 0xFu) + 16u * ((h1 >> c_lo) & 1u) + 32u * ((h2 >> c_lo) & 1u)) - 32;
                    const int hi = static_cast<int>((byte >> 4) + 16u * ((h1 >> c_hi) & 1u) + 32u * ((h2 >> c_hi) & 1u)) - 32;
                    out[c_lo] = __fmul_rn(static_cast<float>(lo), s[b2]);
                    out[c_hi] = __fmul_rn(static_cast<float>(hi), s[b2]);
                }
        }
    }
}
__device__ __forceinline__ bool group32_ok(const QView& t) {
    if (t.cols % 256 != 0) return false;
    if (t.kind == RWKVQ_KIND_SB6) return t.gs == 32 && t.sb == 8;
    return t.kind == RWKVQ_KIND_SYM && t.gs == 16 && t.sb == 16;
}

// x[b] = LN0(fp16(bf16(dequant(emb[token[b]])))): one embedding row is decoded from the
// packed table (quant_model.py:853, 975-976; rounding policy :128-154).  sb6 / sym tables: one
// thread per 32 columns decodes its group with all loads in flight at once and hands the row over
// through shared memory; other layouts: element by element.
__global__ void __launch_bounds__(kRowThreads) embed_ln0_kernel(QView emb, const long long* tokens,
                                                               const float* ln_w, const float* ln_b,
                                                               float* x, int D) {
    __shared__ float red[kRowThreads / 32];
    __shared__ float srow[kRowThreads * kRowPer];
    const int b = blockIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    long long tok = __ldcg(tokens + b);
    tok = tok < 0 ? 0 : (tok >= emb.rows ? emb.rows - 1 : tok);
    float v[kRowPer];
    if (group32_ok(emb)) {
        for (int g = threadIdx.x; g < D / 32; g += kRowThreads) {
            float o[32];
            decode_group32(emb, static_cast<size_t>(tok), g, o);
#pragma unroll
            for (int k = 0; k < 32; ++k) srow[g * 32 + k] = dense_param_rounding(o[k]);
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kRowPer; ++i) {
            const int d = threadIdx.x + i * kRowThreads;
            v[i] = (d < D) ? srow[d] : 0.f;
        }
    } else {
#pragma unroll
        for (int i = 0; i < kRowPer; ++i) {
            const int d = threadIdx.x + i * kRowThreads;
            v[i] = (d < D) ? dense_param_rounding(decode_element(emb, static_cast<int>(tok), d)) : 0.f;
        }
    }
    layer_norm_row<kRowPer>(v, D, ln_w, ln_b, red);
#pragma unroll
    for (int i = 0; i < kRowPer; ++i) {
        const int d = threadIdx.x + i * kRowThreads;
        if (d < D) x[static_cast<size_t>(b) * D + d] = v[i];
    }
}

// xn = LN(x[b]); prev = shift[b] (zeros for a fresh stream); shift[b] = xn;
// out[m][b] = xn + (prev - xn) * mix[m]   for m < n_mix   (n_mix = 0: out[0][b] = xn)
// All loads are issued before the reductions so that their latencies overlap.  PER: elements per thread (16: D <= 4096).
// For rows the vector form below cannot read: odd widths, rows off a 16-byte boundary.
template <int NMIX, int PER>
__global__ void __launch_bounds__(kRowThreads) ln_shift_mix_kernel(const float* __restrict__ x,
                                                                  const float* __restrict__ ln_w,
                                                                  const float* __restrict__ ln_b,
                                                                  float* __restrict__ shift,
                                                                  const float* __restrict__ mix,
                                                                  float* __restrict__ out, int B, int D,
                                                                  __half* __restrict__ x16_out, float* __restrict__ unscale_out, int x16_mask,
                                                                  float* __restrict__ zero_a, float* __restrict__ zero_b) {
    // x16_out (optional) [max(NMIX, 1)][B][D] with unscale_out [max(NMIX, 1)][B]: the rows selected by
    // x16_mask also as fp16(out * 2^s), s chosen from the row's max so that no value leaves the fp16
    // range, and 2^-s: the form the single-term small-batch linear reads (half the bytes, no
    // conversion there).  With unscale_out alone, max|out| of the selected rows goes there instead (what the
    // two-term mma.sync linear wants beside the fp32 rows);
    // zero_a / zero_b (optional) [B]: slots later kernels of the layer merge their own row maxima
    // into, cleared here for stream b
    constexpr int NM = NMIX > 0 ? NMIX : 1;
    __shared__ float red[kRowThreads / 32];
    __shared__ float redm[kRowThreads / 32][NM];
    const int b = blockIdx.x;
    float v[PER], prev[PER], lw[PER], lb[PER];
    pdl_launch_dependents();
#pragma unroll
    for (int i = 0; i < PER; ++i) {          // parameters do not depend on the previous kernel
        const int d = threadIdx.x + i * kRowThreads;
        lw[i] = d < D ? ln_w[d] : 0.f;
        lb[i] = d < D ? ln_b[d] : 0.f;
    }
    pdl_wait();
    if (threadIdx.x == 0) {
        if (zero_a) zero_a[b] = 0.f;
        if (zero_b) zero_b[b] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int d = threadIdx.x + i * kRowThreads;
        const bool ok = d < D;
        const size_t bd = static_cast<size_t>(b) * D + d;
        v[i] = ok ? __ldcg(x + bd) : 0.f;
        prev[i] = (ok && NMIX > 0) ? __ldcg(shift + bd) : 0.f;
    }
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i) s += v[i];
    const float mean = block_sum(s, red) / D;
    float s2 = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const float c = (threadIdx.x + i * kRowThreads < D) ? v[i] - mean : 0.f;
        s2 += c * c;
    }
    const float inv = 1.0f / sqrtf(block_sum(s2, red) / D + 1e-5f);
    float mx[NM];
#pragma unroll
    for (int m = 0; m < NM; ++m) mx[m] = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int d = threadIdx.x + i * kRowThreads;
        if (d >= D) continue;
        const size_t bd = static_cast<size_t>(b) * D + d;
        const float xn = (v[i] - mean) * inv * lw[i] + lb[i];
        if (NMIX == 0) { out[bd] = xn; mx[0] = fmaxf(mx[0], fabsf(xn)); continue; }
        const float xx = prev[i] - xn;
        shift[bd] = xn;
#pragma unroll
        for (int m = 0; m < NMIX; ++m) {
            const float o = xn + xx * __ldg(mix + m * D + d);
            out[(static_cast<size_t>(m) * B) * D + bd] = o;
            mx[m < NM ? m : 0] = fmaxf(mx[m < NM ? m : 0], fabsf(o));
        }
    }
    if (unscale_out != nullptr) {
        __shared__ float sc_m[NM];
#pragma unroll
        for (int m = 0; m < NM; ++m) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mx[m] = fmaxf(mx[m], __shfl_xor_sync(0xFFFFFFFFu, mx[m], o));
            if ((threadIdx.x & 31) == 0) redm[threadIdx.x >> 5][m] = mx[m];
        }
        __syncthreads();
        if (threadIdx.x < NM) {
            float r = 0.f;
            for (int w = 0; w < kRowThreads / 32; ++w) r = fmaxf(r, redm[w][threadIdx.x]);
            if (x16_out == nullptr) {
                if ((x16_mask >> threadIdx.x) & 1) unscale_out[threadIdx.x * B + b] = r;
                return;
            }
            // |x| * 2^(14 - e) <= 2^14 with max|x| <= 2^e; a non-finite row keeps scale 1 and propagates
            float s1 = 1.f, u1 = 1.f;
            if (r > 0.f && r < INFINITY) {
                int e = 0;
                frexpf(r, &e);
                e = max(-100, e);
                s1 = ldexpf(1.f, 14 - e);
                u1 = ldexpf(1.f, e - 14);
            }
            sc_m[threadIdx.x] = s1;
            if ((x16_mask >> threadIdx.x) & 1) unscale_out[threadIdx.x * B + b] = u1;
        }
        if (x16_out == nullptr) return;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int d = threadIdx.x + i * kRowThreads;
            if (d >= D) continue;
            const size_t bd = static_cast<size_t>(b) * D + d;
            const float xn = (v[i] - mean) * inv * lw[i] + lb[i];
            auto emit = [&](int m, float sx) { x16_out[(static_cast<size_t>(m) * B) * D + bd] = __float2half_rn(sx); };
            if (NMIX == 0) { emit(0, xn * sc_m[0]); continue; }
            const float xx = prev[i] - xn;
#pragma unroll
            for (int m = 0; m < NMIX; ++m) {
                if (!((x16_mask >> m) & 1)) continue;
                const float o = xn + xx * __ldg(mix + m * D + d);
                emit(m, o * sc_m[m < NM ? m : 0]);
            }
        }
    }
}

// The same for rows of whole, aligned float4: a thread per float4, every parameter in registers before the wait.
// Bound: latency (one L2 round trip, two block sums, the stores); at 256 threads of 8 or 16 scalars each the loads and
// stores alone issue for a microsecond.  One stream: 2560 wide 8.7 -> 3.3 us, 2048 wide 3.9 -> 3.0 us.
template <int NMIX>
__global__ void __launch_bounds__(kLnVecThreads) ln_shift_mix_vec_kernel(const float* __restrict__ x, const float* __restrict__ ln_w,
                                                                         const float* __restrict__ ln_b, float* __restrict__ shift,
                                                                         const float* __restrict__ mix, float* __restrict__ out, int B, int D,
                                                                         __half* __restrict__ x16_out, float* __restrict__ unscale_out,
                                                                         int x16_mask, float* __restrict__ zero_a, float* __restrict__ zero_b) {
    constexpr int NM = NMIX > 0 ? NMIX : 1;
    __shared__ float red[2][32];
    __shared__ float redm[NM][32];
    const int b = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, warps = blockDim.x >> 5;
    const bool ok = 4 * tid < D;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const size_t at = static_cast<size_t>(b) * (D >> 2) + tid;         // in float4
    pdl_launch_dependents();
    const float4 lw = ok ? __ldg(reinterpret_cast<const float4*>(ln_w) + tid) : zero;
    const float4 lb = ok ? __ldg(reinterpret_cast<const float4*>(ln_b) + tid) : zero;
    float4 mx[NM];
#pragma unroll
    for (int m = 0; m < NMIX; ++m) mx[m] = ok ? __ldg(reinterpret_cast<const float4*>(mix + static_cast<size_t>(m) * D) + tid) : zero;
    pdl_wait();
    if (tid == 0) {
        if (zero_a) zero_a[b] = 0.f;
        if (zero_b) zero_b[b] = 0.f;
    }
    const float4 v = ok ? __ldcg(reinterpret_cast<const float4*>(x) + at) : zero;
    const float4 prev = ok && NMIX > 0 ? __ldcg(reinterpret_cast<const float4*>(shift) + at) : zero;
    auto sum = [&](float s, float* r) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
        if (lane == 0) r[warp] = s;
        __syncthreads();
        s = lane < warps ? r[lane] : 0.f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
        return s;
    };
    const float mean = sum((v.x + v.y) + (v.z + v.w), red[0]) / D;
    const float4 c = ok ? make_float4(v.x - mean, v.y - mean, v.z - mean, v.w - mean) : zero;
    const float inv = 1.0f / sqrtf(sum((c.x * c.x + c.y * c.y) + (c.z * c.z + c.w * c.w), red[1]) / D + 1e-5f);
    const float4 xn = make_float4(c.x * inv * lw.x + lb.x, c.y * inv * lw.y + lb.y, c.z * inv * lw.z + lb.z, c.w * inv * lw.w + lb.w);
    const float4 xx = make_float4(prev.x - xn.x, prev.y - xn.y, prev.z - xn.z, prev.w - xn.w);
    auto mixed = [&](int m) {
        return NMIX == 0 ? xn : make_float4(xn.x + xx.x * mx[m].x, xn.y + xx.y * mx[m].y, xn.z + xx.z * mx[m].z, xn.w + xx.w * mx[m].w);
    };
    const size_t stride = static_cast<size_t>(B) * (D >> 2);
#pragma unroll
    for (int m = 0; m < NM; ++m)
        if (ok) reinterpret_cast<float4*>(out)[m * stride + at] = mixed(m);
    if (ok && NMIX > 0) reinterpret_cast<float4*>(shift)[at] = xn;
    if (unscale_out == nullptr) return;
#pragma unroll
    for (int m = 0; m < NM; ++m) {
        const float4 o = mixed(m);
        float r = ok ? fmaxf(fmaxf(fabsf(o.x), fabsf(o.y)), fmaxf(fabsf(o.z), fabsf(o.w))) : 0.f;
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) r = fmaxf(r, __shfl_xor_sync(0xFFFFFFFFu, r, s));
        if (lane == 0) redm[m][warp] = r;
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < NM; ++m) {
        if (!((x16_mask >> m) & 1)) continue;
        float r = lane < warps ? redm[m][lane] : 0.f;
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) r = fmaxf(r, __shfl_xor_sync(0xFFFFFFFFu, r, s));
        if (x16_out == nullptr) {
            if (tid == 0) unscale_out[m * B + b] = r;
            continue;
        }
        float s1 = 1.f, u1 = 1.f;                                      // as in the scalar form
        if (r > 0.f && r < INFINITY) {
            int e = 0;
            frexpf(r, &e);
            e = max(-100, e);
            s1 = ldexpf(1.f, 14 - e);
            u1 = ldexpf(1.f, e - 14);
        }
        if (tid == 0) unscale_out[m * B + b] = u1;
        const float4 o = mixed(m);
        __half2 h[2] = {__floats2half2_rn(o.x * s1, o.y * s1), __floats2half2_rn(o.z * s1, o.w * s1)};
        if (ok) reinterpret_cast<uint2*>(x16_out)[m * stride + at] = *reinterpret_cast<uint2*>(h);
    }
}

template <int NMIX>
void launch_ln_shift_mix(int B, cudaStream_t s, const float* x, const float* ln_w, const float* ln_b, float* shift, const float* mix,
                         float* out, int D, __half* x16_out, float* unscale_out, int x16_mask, float* zero_a, float* zero_b) {
    if (D % 4 == 0 && D <= 4 * kLnVecThreads && aligned(x, 16) && aligned(ln_w, 16) && aligned(ln_b, 16) && aligned(out, 16) &&
        (NMIX == 0 || (aligned(shift, 16) && aligned(mix, 16)))) {
        launch_pdl(ln_shift_mix_vec_kernel<NMIX>, dim3(B), dim3((D / 4 + 31) / 32 * 32), 0, s, x, ln_w, ln_b, shift, mix, out, B, D, x16_out,
                   unscale_out, x16_mask, zero_a, zero_b);
    } else {
        launch_pdl(ln_shift_mix_kernel<NMIX, kRowPer>, dim3(B), dim3(kRowThreads), 0, s, x, ln_w, ln_b, shift, mix, out, B, D, x16_out,
                   unscale_out, x16_mask, zero_a, zero_b);
    }
}

// ---- batched LoRA products, tensors stored [in, out] (a warp reads 128 contiguous codes)
//
// down:  part[br][chunk][n][j] = sum_{i in chunk} x_br[n][i] * W1_br[i][j]     (j < rank)
//        grid (row chunks of 64, branches); the partial sums go to scratch in a fixed
//        layout and are added in chunk order by the consumer, so the result does not
//        depend on scheduling.
// up:    h[j] = act_br(sum_chunk part[br][chunk][n][j]);  y_br[n][c] = sum_j h[j] * W2_br[j][c]
//        grid (column tiles of 128, branches).
constexpr int kLmMaxN = 8;            // right-hand sides per launch
constexpr int kLdRows = 64;           // rows of W1 per CTA
constexpr int kLuCols = 128;          // columns of W2 per CTA
constexpr int kLmMaxRank = 512;

struct LoraDownArgs {
    QView t[4];
    const float* x[4];      // [n_cols, ldx]
    float* part;            // [4][n_chunks][n_stride][max_rank]
    long long ldx;
    int n_cols, n_chunks, max_rank;
    int n_stride;           // right-hand sides the scratch is laid out for (multiple of kLmMaxN)
    int rep;                // 64-row sub-chunks one CTA accumulates (more for large batches: fewer partial sums)
};
struct LoraUpArgs {
    QView t[4];
    const float* part;
    float* y[4];            // [n_cols, ldy]
    int act[4];
    long long ldy;
    int n_cols, n_chunks, max_rank, n_stride;
};

// 256 threads = 4 row groups x 64 column threads (4 columns each, 256 columns per pass)
// MULTI = false: one 64-row chunk per CTA (the batch-1 form, loops resolved at compile time)
template <int MODE, bool MULTI>
__device__ __forceinline__ void lora_down_body(const LoraDownArgs& a, const QView& t, const float* __restrict__ xall,
                                               float (&red)[4][kLmMaxN][256]) {
    const int chunk = blockIdx.x, br = blockIdx.y;
    const int n0 = blockIdx.z * kLmMaxN;                  // this CTA's group of right-hand sides
    const int nc = min(kLmMaxN, a.n_cols - n0);
    const float* x = xall + static_cast<size_t>(n0) * a.ldx;
    const int rg = threadIdx.x >> 6, ct = threadIdx.x & 63;
    const int nb = MODE == 0 ? (t.cols + t.gs - 1) / t.gs : 0;
    for (int c0 = 0; c0 < t.cols; c0 += 256) {
        const int c = c0 + ct * 4;
        const int blk = MODE == 0 ? c / t.gs : 0;
        float acc[kLmMaxN][4];
#pragma unroll
        for (int n = 0; n < kLmMaxN; ++n)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[n][k] = 0.f;
        const int rep = MULTI ? a.rep : 1;
#pragma unroll 1
        for (int sub = 0; sub < rep; ++sub) {
            const int row0 = (chunk * rep + sub) * kLdRows;
            if (c < t.cols && row0 < t.rows) {
                constexpr int RPT = kLdRows / 4;          // rows per thread, all loads issued together
                float w[RPT][4];
#pragma unroll
                for (int r = 0; r < RPT; ++r) lora_w4<MODE>(t, min(row0 + rg + 4 * r, t.rows - 1), c, nb, blk, w[r]);
                pdl_wait();              // the weights above are constants; x comes from the previous kernel
#pragma unroll
                for (int n = 0; n < kLmMaxN; ++n) {
                    if (n >= nc) break;
#pragma unroll
                    for (int r = 0; r < RPT; ++r) {
                        const int i = row0 + rg + 4 * r;
                        const float xv = i < t.rows ? __ldcg(x + n * a.ldx + i) : 0.f;
#pragma unroll
                        for (int k = 0; k < 4; ++k) acc[n][k] = fmaf(xv, w[r][k], acc[n][k]);
                    }
                }
            }
        }
        pdl_wait();
        __syncthreads();
#pragma unroll
        for (int n = 0; n < kLmMaxN; ++n) {
            if (n >= nc) break;
#pragma unroll
            for (int k = 0; k < 4; ++k) red[rg][n][ct * 4 + k] = acc[n][k];
        }
        __syncthreads();
        for (int idx = threadIdx.x; idx < nc * 256; idx += 256) {
            const int n = idx >> 8, cc = idx & 255;
            if (c0 + cc >= t.cols) continue;
            const float v = (red[0][n][cc] + red[1][n][cc]) + (red[2][n][cc] + red[3][n][cc]);
            a.part[((static_cast<size_t>(br) * a.n_chunks + chunk) * a.n_stride + n0 + n) * a.max_rank + c0 + cc] = v;
        }
    }
}

template <bool MULTI>
__global__ void __launch_bounds__(256) lora_down_kernel(const LoraDownArgs a) {
    __shared__ float red[4][kLmMaxN][256];
    const QView& t = a.t[blockIdx.y];
    const float* x = a.x[blockIdx.y];
    pdl_launch_dependents();
    switch (lora_mode(t)) {
        case 0: lora_down_body<0, MULTI>(a, t, x, red); break;
        case 1: lora_down_body<1, MULTI>(a, t, x, red); break;
        default: lora_down_body<2, MULTI>(a, t, x, red); break;
    }
}

// 256 threads = 8 row groups x 32 column threads (4 columns each)
template <int MODE>
__device__ __forceinline__ void lora_up_body(const LoraUpArgs& a, int n_cols, const QView& t,
                                             const float (&h)[kLmMaxN][kLmMaxRank], float (&acc)[kLmMaxN][4]) {
    const int rg = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = blockIdx.x * kLuCols + lane * 4;
    const int rank = t.rows;
    const int nb = MODE == 0 ? (t.cols + t.gs - 1) / t.gs : 0;
    const int blk = MODE == 0 ? c / t.gs : 0;
    if (c >= t.cols) return;
    for (int j0 = rg; j0 < rank; j0 += 64) {          // 8 rows of this thread per batch of loads
        float w[8][4];
#pragma unroll
        for (int r = 0; r < 8; ++r) lora_w4<MODE>(t, min(j0 + 8 * r, rank - 1), c, nb, blk, w[r]);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int j = j0 + 8 * r;
            if (j >= rank) break;
#pragma unroll
            for (int n = 0; n < kLmMaxN; ++n) {
                if (n >= n_cols) break;
                const float hv = h[n][j];
#pragma unroll
                for (int k = 0; k < 4; ++k) acc[n][k] = fmaf(hv, w[r][k], acc[n][k]);
            }
        }
    }
}

__global__ void __launch_bounds__(256) lora_up_kernel(const LoraUpArgs a) {
    __shared__ float h[kLmMaxN][kLmMaxRank];
    __shared__ float red[8][kLmMaxN][kLuCols];
    const int br = blockIdx.y;
    const QView& t = a.t[br];
    pdl_launch_dependents();
    pdl_wait();
    if (blockIdx.x * kLuCols >= t.cols) return;
    const int rank = t.rows;
    const int n0 = blockIdx.z * kLmMaxN;                      // this CTA's group of right-hand sides
    const int nc = min(kLmMaxN, a.n_cols - n0);
    for (int idx = threadIdx.x; idx < nc * rank; idx += 256) {
        const int n = idx / rank, j = idx % rank;
        const float* pp = a.part + ((static_cast<size_t>(br) * a.n_chunks) * a.n_stride + n0 + n) * a.max_rank + j;
        const size_t stride = static_cast<size_t>(a.n_stride) * a.max_rank;
        float v = 0.f;
        int ch = 0;
        for (; ch + 8 <= a.n_chunks; ch += 8) {       // 8 loads in flight, summed in chunk order
            float pv[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) pv[u] = __ldcg(pp + (ch + u) * stride);
#pragma unroll
            for (int u = 0; u < 8; ++u) v += pv[u];
        }
        for (; ch < a.n_chunks; ++ch) v += __ldcg(pp + ch * stride);
        if (a.act[br] == 1) v = tanhf(v);
        else if (a.act[br] == 2) v = sigmoidf_(v);
        h[n][j] = v;
    }
    __syncthreads();
    const int rg = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float acc[kLmMaxN][4];
#pragma unroll
    for (int n = 0; n < kLmMaxN; ++n)
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[n][k] = 0.f;
    switch (lora_mode(t)) {
        case 0: lora_up_body<0>(a, nc, t, h, acc); break;
        case 1: lora_up_body<1>(a, nc, t, h, acc); break;
        default: lora_up_body<2>(a, nc, t, h, acc); break;
    }
#pragma unroll
    for (int n = 0; n < kLmMaxN; ++n) {
        if (n >= nc) break;
#pragma unroll
        for (int k = 0; k < 4; ++k) red[rg][n][lane * 4 + k] = acc[n][k];
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < nc * kLuCols; idx += 256) {
        const int n = idx / kLuCols, cc = idx % kLuCols;
        const int col = blockIdx.x * kLuCols + cc;
        if (col >= t.cols) continue;
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) v += red[w][n][cc];
        a.y[br][static_cast<size_t>(n0 + n) * a.ldy + col] = v;
    }
}

// ---- time-mix core for one token: grid (H, B), 256 threads = (state row dv, quarter)
struct TmixCoreArgs {
    const float *r, *k, *v;            // [B, D] projections
    const float *yw, *ya, *yv, *g;     // [B, D] LoRA outputs (yv null on layer 0)
    const float *w0, *a0, *v0;         // [D]
    const float *k_k, *k_a, *r_k, *lnx_w, *lnx_b;
    float* v_first;                    // [B, D] written by layer 0, read by the others
    float* state;                      // [B, H, 64, 64] in place
    float* og;                         // [B, D]
    int D, H, layer0;
    float* og_amax;                    // optional [B]: max|og| per stream is merged into it (atomic max on the bits)
};

// sum over 64 shared-memory values, computed redundantly by every warp (two values per lane):
// no block-wide barrier beyond the one that published the values
__device__ __forceinline__ float warp_sum64(const float* v, int lane) {
    float s = v[lane] + v[lane + 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
    return s;
}

// One stream: the LoRA up projections of the head's 64 channels run here too, their weights staged before the wait.
__global__ void __launch_bounds__(256) tmix_core_up_kernel(const TmixCoreArgs p, const LoraVecArgs up) {
    extern __shared__ __align__(16) unsigned char up_smem[];         // [ranks][64] fp16, [ranks] h, [8][4][64] partial sums
    // per-column operands of the state update, written once by warps 0 and 1 and read as float4 by all:
    // sA = -kk / |kk|, sB = (kk / |kk|) * a_gate, sW decay, sK key, sR receptance
    __shared__ __align__(16) float sA[64], sB[64], sW[64], sK[64], sR[64];
    __shared__ float sV[64], sY[64], sG[64], sT[64];
    const int hi = blockIdx.x, b = blockIdx.y, tid = threadIdx.x, lane = tid & 31;
    const size_t row = static_cast<size_t>(b) * p.D + hi * 64;
    // the state slice of this thread is requested first: it is the largest load
    // thread (dv, part) owns columns 16 i + 4 part + e of state row dv (i, e < 4): every load
    // instruction of a quad covers 64 contiguous bytes
    const int dv = tid >> 2, part = tid & 3;
    float* hp = p.state + ((static_cast<size_t>(b) * p.H + hi) * 64 + dv) * 64 + part * 4;
    float h[16];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 v4 = __ldcs(reinterpret_cast<const float4*>(hp + 16 * i));
        h[4 * i] = v4.x; h[4 * i + 1] = v4.y; h[4 * i + 2] = v4.z; h[4 * i + 3] = v4.w;
    }
    pdl_launch_dependents();
    // per-channel parameters of warps 0 and 1 (channel hi * 64 + tid; r_k also for the partner channel of the
    // final dot product): nothing the kernels before this one write, so they are loaded before the wait
    float pw0 = 0.f, pa0 = 0.f, pka = 0.f, pkk = 0.f, pv0 = 0.f, prk0 = 0.f, prk1 = 0.f, plw = 0.f, plb = 0.f;
    if (tid < 64) {
        const int c = hi * 64 + tid;
        pw0 = __ldg(p.w0 + c); pa0 = __ldg(p.a0 + c); pka = __ldg(p.k_a + c); pkk = __ldg(p.k_k + c);
        if (!p.layer0) pv0 = __ldg(p.v0 + c);
        prk0 = __ldg(p.r_k + hi * 64 + lane); prk1 = __ldg(p.r_k + hi * 64 + lane + 32);
        plw = __ldg(p.lnx_w + c); plb = __ldg(p.lnx_b + c);
    }
    const int ranks = up.first[up.n_br];
    __half* wt = reinterpret_cast<__half*>(up_smem);
    float* hl = reinterpret_cast<float*>(wt + ranks * 64);
    float* part_up = hl + ranks;
    lora_up_stage(up, hi * 64, wt);
    pdl_wait();                // the state above was written a whole token ago
    for (int i = tid; i < ranks; i += 256) hl[i] = __ldcg(up.h + i);
    __syncthreads();
    lora_up_vec(up, wt, hl, part_up);
    __syncthreads();
    // LoRA output `br` (decay, rate, gate, value-residual) of the thread's channel
    auto lora = [&](int br) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) v += part_up[w * 256 + br * 64 + tid];
        return v;
    };
    if (tid < 64) {
        const float r = __ldcg(p.r + row + tid), k = __ldcg(p.k + row + tid);
        float v = __ldcg(p.v + row + tid);
        const float w = expf(-0.606531f * sigmoidf_(lora(0) + pw0));
        const float av = sigmoidf_(lora(1) + pa0);
        const float k2 = k * (1.0f + (av - 1.0f) * pka);
        if (p.layer0) p.v_first[row + tid] = v;
        else v = v + (__ldcg(p.v_first + row + tid) - v) * sigmoidf_(lora(3) + pv0);
        const float kk = k * pkk;
        sT[tid] = kk * kk;
        sW[tid] = w; sK[tid] = k2; sR[tid] = r; sV[tid] = v; sG[tid] = lora(2);
        asm volatile("bar.sync 1, 64;" ::: "memory");        // warps 0 and 1 only: sT is complete
        // both warps reduce the head-wide sum themselves; a = -kk / |kk|, b = -a * a_gate
        const float kn = kk * (1.0f / sqrtf(warp_sum64(sT, lane) + 1e-12f));
        sA[tid] = -kn;
        sB[tid] = kn * av;
    }
    __syncthreads();
    // one WKV-7 step on the thread's 16 state columns
    float sa = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 a4 = *reinterpret_cast<const float4*>(sA + 16 * i + 4 * part);
        sa = fmaf(h[4 * i], a4.x, sa); sa = fmaf(h[4 * i + 1], a4.y, sa);
        sa = fmaf(h[4 * i + 2], a4.z, sa); sa = fmaf(h[4 * i + 3], a4.w, sa);
    }
    sa += __shfl_xor_sync(0xFFFFFFFFu, sa, 1);
    sa += __shfl_xor_sync(0xFFFFFFFFu, sa, 2);
    const float vv = sV[dv];
    float y = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int dk = 16 * i + 4 * part;
        const float4 b4 = *reinterpret_cast<const float4*>(sB + dk), w4 = *reinterpret_cast<const float4*>(sW + dk);
        const float4 k4 = *reinterpret_cast<const float4*>(sK + dk), r4 = *reinterpret_cast<const float4*>(sR + dk);
        h[4 * i] = fmaf(w4.x, h[4 * i], fmaf(vv, k4.x, sa * b4.x));
        y = fmaf(h[4 * i], r4.x, y);
        h[4 * i + 1] = fmaf(w4.y, h[4 * i + 1], fmaf(vv, k4.y, sa * b4.y));
        y = fmaf(h[4 * i + 1], r4.y, y);
        h[4 * i + 2] = fmaf(w4.z, h[4 * i + 2], fmaf(vv, k4.z, sa * b4.z));
        y = fmaf(h[4 * i + 2], r4.z, y);
        h[4 * i + 3] = fmaf(w4.w, h[4 * i + 3], fmaf(vv, k4.w, sa * b4.w));
        y = fmaf(h[4 * i + 3], r4.w, y);
    }
    y += __shfl_xor_sync(0xFFFFFFFFu, y, 1);
    y += __shfl_xor_sync(0xFFFFFFFFu, y, 2);
#pragma unroll
    for (int i = 0; i < 4; ++i)
        *reinterpret_cast<float4*>(hp + 16 * i) = make_float4(h[4 * i], h[4 * i + 1], h[4 * i + 2], h[4 * i + 3]);
    if (part == 0) sY[dv] = y;
    __syncthreads();
    if (tid < 64) {            // warps 0 and 1: group norm over the head (two-pass), bonus, gate
        const float mean = warp_sum64(sY, lane) / 64.f;
        const float d0 = sY[lane] - mean, d1 = sY[lane + 32] - mean;
        float var = d0 * d0 + d1 * d1, dp = sR[lane] * sK[lane] * prk0 + sR[lane + 32] * sK[lane + 32] * prk1;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            var += __shfl_xor_sync(0xFFFFFFFFu, var, o);
            dp += __shfl_xor_sync(0xFFFFFFFFu, dp, o);
        }
        const float nrm = (sY[tid] - mean) * (1.0f / sqrtf(var / 64.f + 64e-5f));
        const float o = (nrm * plw + plb + dp * sV[tid]) * sG[tid];
        p.og[row + tid] = o;
        if (p.og_amax != nullptr) {          // warps 0 and 1 hold the 64 outputs
            float m = fabsf(o);
#pragma unroll
            for (int of = 16; of > 0; of >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, of));
            if ((tid & 31) == 0) atomicMax(reinterpret_cast<int*>(p.og_amax) + b, __float_as_int(m));
        }
    }
}

// Several streams: two warps a (head, stream) pair.  Bound: latency of the chain rows -> gates -> row sums -> update -> group norm up to
// some 20 streams, then the state (64 streams, 67 MB read and written: 20 -> 12 us a layer, 100 streams 35 -> 24).  A thread's tile is
// 8 state rows x 8 columns: the five vectors of a step cost it 10 shared-memory loads for 64 state values (20 for 16 with eight warps
// a pair, as above), the arithmetic goes in pairs, and a barrier waits for one other warp; a pair takes a quarter of the
// instructions and of an SM's threads.  Against eight warps a pair, ms a step: 1.5B 4 streams 1.64 / 1.64, 16 1.79 / 1.76, 20 1.95 / 1.82,
// 64 2.64 / 2.46, 100 3.63 / 3.39; 2.9B 2 streams 2.81 / 2.78, 16 3.08 / 2.95, 128 7.57 / 7.11.  Persistent CTAs of eight warps with the state and
// rows of the next pair in registers lost 1 to 2 % (64 streams 2.67).
__global__ void __launch_bounds__(64, 8) tmix_core_kernel(const TmixCoreArgs p) {
    __shared__ __align__(16) float sA[64], sB[64], sW[64], sK[64], sR[64], sV[64];
    __shared__ float sY[64], sT[64];
    const int hi = blockIdx.x, b = blockIdx.y, tid = threadIdx.x, lane = tid & 31;
    const size_t row = static_cast<size_t>(b) * p.D + hi * 64 + tid;
    const int c = tid & 7, dv0 = (tid >> 3) * 8;
    float* hp = p.state + ((static_cast<size_t>(b) * p.H + hi) * 64 + dv0) * 64 + 4 * c;     // columns 4 c .. and 32 + 4 c ..
    float2 h[8][4];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float4 lo = __ldcs(reinterpret_cast<const float4*>(hp + 64 * j)), hj = __ldcs(reinterpret_cast<const float4*>(hp + 64 * j + 32));
        h[j][0] = make_float2(lo.x, lo.y); h[j][1] = make_float2(lo.z, lo.w);
        h[j][2] = make_float2(hj.x, hj.y); h[j][3] = make_float2(hj.z, hj.w);
    }
    pdl_launch_dependents();
    const int ch = hi * 64 + tid;
    const float pw0 = __ldg(p.w0 + ch), pa0 = __ldg(p.a0 + ch), pka = __ldg(p.k_a + ch), pkk = __ldg(p.k_k + ch);
    const float pv0 = p.layer0 ? 0.f : __ldg(p.v0 + ch);
    const float prk0 = __ldg(p.r_k + hi * 64 + lane), prk1 = __ldg(p.r_k + hi * 64 + lane + 32), plw = __ldg(p.lnx_w + ch), plb = __ldg(p.lnx_b + ch);
    pdl_wait();                              // the state above was written a whole token ago
    const float r = __ldcg(p.r + row), k = __ldcg(p.k + row), yw = __ldcg(p.yw + row), ya = __ldcg(p.ya + row), g = __ldcg(p.g + row);
    float v = __ldcg(p.v + row);
    if (p.layer0) p.v_first[row] = v;
    else v = v + (__ldcg(p.v_first + row) - v) * sigmoidf_(__ldcg(p.yv + row) + pv0);
    const float w = expf(-0.606531f * sigmoidf_(yw + pw0)), av = sigmoidf_(ya + pa0), kk = k * pkk;
    sT[tid] = kk * kk;
    sW[tid] = w; sK[tid] = k * (1.0f + (av - 1.0f) * pka); sR[tid] = r; sV[tid] = v;
    __syncthreads();
    const float kn = kk * (1.0f / sqrtf(warp_sum64(sT, lane) + 1e-12f));
    sA[tid] = -kn;
    sB[tid] = kn * av;
    __syncthreads();
    float2 x[4];
    float sa[8], y[8];
    cols8(sA, c, x);
#pragma unroll
    for (int j = 0; j < 8; ++j) sa[j] = dot8(h[j], x);
    {
        float2 wc[4], kc[4];                 // decay and v k^T while the sums cross the lanes
        cols8(sW, c, wc);
        cols8(sK, c, kc);
        const float4 va = *reinterpret_cast<const float4*>(sV + dv0), vb = *reinterpret_cast<const float4*>(sV + dv0 + 4);
        const float vs[8] = {va.x, va.y, va.z, va.w, vb.x, vb.y, vb.z, vb.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float2 vj = make_float2(vs[j], vs[j]);
#pragma unroll
            for (int q = 0; q < 4; ++q) h[j][q] = __ffma2_rn(wc[q], h[j][q], __fmul2_rn(vj, kc[q]));
        }
    }
#pragma unroll
    for (int m = 1; m < 8; m <<= 1)
#pragma unroll
        for (int j = 0; j < 8; ++j) sa[j] += __shfl_xor_sync(0xFFFFFFFFu, sa[j], m);
    cols8(sB, c, x);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float2 s2 = make_float2(sa[j], sa[j]);
#pragma unroll
        for (int q = 0; q < 4; ++q) h[j][q] = __ffma2_rn(s2, x[q], h[j][q]);
        *reinterpret_cast<float4*>(hp + 64 * j) = make_float4(h[j][0].x, h[j][0].y, h[j][1].x, h[j][1].y);
        *reinterpret_cast<float4*>(hp + 64 * j + 32) = make_float4(h[j][2].x, h[j][2].y, h[j][3].x, h[j][3].y);
    }
    cols8(sR, c, x);
#pragma unroll
    for (int j = 0; j < 8; ++j) y[j] = dot8(h[j], x);
    // eight sums over eight lanes, half of them handed over at each of the three steps: lane bit 0 picks rows 0-3 or 4-7, bit 1 and 2 the row
#pragma unroll
    for (int n = 4, m = 1; n > 0; n >>= 1, m <<= 1)
#pragma unroll
        for (int j = 0; j < n; ++j) {
            const bool up = (c & m) != 0;
            const float keep = up ? y[j + n] : y[j], give = up ? y[j] : y[j + n];
            y[j] = keep + __shfl_xor_sync(0xFFFFFFFFu, give, m);
        }
    sY[dv0 + (c & 1) * 4 + (c & 2) + (c >> 2)] = y[0];
    __syncthreads();
    // group norm over the head (two-pass), bonus, gate
    const float mean = warp_sum64(sY, lane) / 64.f;
    const float d0 = sY[lane] - mean, d1 = sY[lane + 32] - mean;
    float var = d0 * d0 + d1 * d1, dp = sR[lane] * sK[lane] * prk0 + sR[lane + 32] * sK[lane + 32] * prk1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        var += __shfl_xor_sync(0xFFFFFFFFu, var, o);
        dp += __shfl_xor_sync(0xFFFFFFFFu, dp, o);
    }
    const float nrm = (sY[tid] - mean) * (1.0f / sqrtf(var / 64.f + 64e-5f));
    const float o = (nrm * plw + plb + dp * v) * g;
    p.og[row] = o;
    if (p.og_amax != nullptr) {
        float m = fabsf(o);
#pragma unroll
        for (int of = 16; of > 0; of >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, of));
        if (lane == 0) atomicMax(reinterpret_cast<int*>(p.og_amax) + b, __float_as_int(m));
    }
}

// greedy argmax in two stages (lowest index wins ties): 64 slices per row, then one CTA
constexpr int kArgSlices = 64;
__global__ void __launch_bounds__(256) argmax_partial_kernel(const float* logits, float* pv, int* pi, int V) {
    __shared__ float bv[8];
    __shared__ int bi[8];
    pdl_launch_dependents();
    pdl_wait();
    const float* row = logits + static_cast<size_t>(blockIdx.y) * V;
    const int per = (V + kArgSlices - 1) / kArgSlices;
    const int lo = blockIdx.x * per, hi = min(lo + per, V);
    float best = -INFINITY;
    int idx = V;
    for (int i = lo + threadIdx.x; i < hi; i += 256) argmax_combine(best, idx, __ldcg(row + i), i);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        argmax_combine(best, idx, __shfl_xor_sync(0xFFFFFFFFu, best, o), __shfl_xor_sync(0xFFFFFFFFu, idx, o));
    if ((threadIdx.x & 31) == 0) { bv[threadIdx.x >> 5] = best; bi[threadIdx.x >> 5] = idx; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) argmax_combine(best, idx, bv[w], bi[w]);
        pv[blockIdx.y * kArgSlices + blockIdx.x] = best;
        pi[blockIdx.y * kArgSlices + blockIdx.x] = idx;
    }
}
__global__ void __launch_bounds__(kArgSlices) argmax_final_kernel(const float* pv, const int* pi, long long* out, int V) {
    pdl_wait();
    float best = __ldcg(pv + blockIdx.x * kArgSlices + threadIdx.x);
    int idx = __ldcg(pi + blockIdx.x * kArgSlices + threadIdx.x);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        argmax_combine(best, idx, __shfl_xor_sync(0xFFFFFFFFu, best, o), __shfl_xor_sync(0xFFFFFFFFu, idx, o));
    __shared__ float bv[2];
    __shared__ int bi[2];
    if ((threadIdx.x & 31) == 0) { bv[threadIdx.x >> 5] = best; bi[threadIdx.x >> 5] = idx; }
    __syncthreads();
    if (threadIdx.x == 0) {
        argmax_combine(best, idx, bv[1], bi[1]);
        out[blockIdx.x] = idx < V ? idx : 0;
    }
}

// The LoRA branches depend on the normalised row only, not on r/k/v: the two run on two streams between a fork after LN1
// and a join before the time mix, in a captured graph as parallel branches.  One side stream and two events per (device,
// caller stream), created on the first call that uses that stream (not during its capture: such a call goes without):
// sequences issued on different streams, from one or several host threads, never share an event.  Calls on the SAME
// stream must come from one thread at a time, as for any stream-ordered API.
// RWKVQ_FORK=0 keeps everything on the caller's stream.
SideLane* side_lane(cudaStream_t caller) {
    static const bool enabled = [] { const char* e = getenv("RWKVQ_FORK"); return !(e && e[0] == '0'); }();
    if (!enabled || caller == cudaStreamPerThread) return nullptr;      // one handle for a stream of every thread: their forks would mix
    static std::mutex mu;
    static std::map<std::pair<int, cudaStream_t>, SideLane> lanes;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    SideLane& l = lanes[std::make_pair(dev, caller)];
    if (!l.stream) {
        cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(caller, &capturing) != cudaSuccess) { cudaGetLastError(); return nullptr; }
        if (capturing != cudaStreamCaptureStatusNone) return nullptr;
        SideLane n;
        if (cudaStreamCreateWithFlags(&n.stream, cudaStreamNonBlocking) != cudaSuccess ||
            cudaEventCreateWithFlags(&n.fork, cudaEventDisableTiming) != cudaSuccess ||
            cudaEventCreateWithFlags(&n.join, cudaEventDisableTiming) != cudaSuccess) {
            if (n.fork) cudaEventDestroy(n.fork);
            if (n.stream) cudaStreamDestroy(n.stream);
            return nullptr;
        }
        l = n;
    }
    return &l;
}
int SideLane::start(cudaStream_t caller) const {
    if (cudaEventRecord(fork, caller) != cudaSuccess || cudaStreamWaitEvent(stream, fork, 0) != cudaSuccess)
        return fail(RWKVQ_E_LAUNCH, "fork onto the side stream failed");
    return RWKVQ_OK;
}
int SideLane::mark() const {
    return cudaEventRecord(join, stream) == cudaSuccess ? RWKVQ_OK : fail(RWKVQ_E_LAUNCH, "join of the side stream failed");
}
int SideLane::wait(cudaStream_t caller) const {
    return cudaStreamWaitEvent(caller, join, 0) == cudaSuccess ? RWKVQ_OK : fail(RWKVQ_E_LAUNCH, "join of the side stream failed");
}

}  // namespace rwkvq

using namespace rwkvq;

namespace {

constexpr int kBatchMax = 256;     // streams up to which the small-batch kernel serves the linears of a step
// (two streams: 1.60 ms per step of the 1.5B model against 1.82 on one single-vector launch per stream, 2.9B 2.79 / 3.81)
// with single-term operands from three on: two streams keep the single-vector kernels' precision in every mode
inline bool batch_path(int B) { return B > (batch_fast() ? 2 : 1) && B <= kBatchMax; }
// Single-term operands (RWKVQ_BATCH_FAST=1): the tcgen05 form wins over the mma.sync one from 33 streams on (1.5B, whole
// step, 64 streams: 3.77 against 4.43 ms) and loses below (32: 2.87 / 2.68 ms, 8: 2.42 / 2.01): its pass (dependent weight
// loads -> conversion -> MMA) is longer than a warp-iteration.  The default precision is faster from 20 streams on, with sym tensors
// from 9 (ms, default / this: 1.5B sb6 8 streams 1.67 / 1.49, 16 1.77 / 1.66, 20 1.82 / 1.99, 64 2.44 / 3.11; sym 8 1.70 / 1.59, 9 1.65 / 1.74,
// 64 2.43 / 3.37).
inline bool tcb_pays(int B) { return batch_fast() && tcb_enabled() && B > 32; }
// Default (two-term) precision: from kSbMinStreams streams on every linear of the step runs on the tcgen05 pipeline
// (rwkvq_gemm_sb.cu), fed with fp16 pairs and block sums by the LayerNorm kernels and, for the output projection and the
// ffn value, by a pass over the fp32 rows.  Below, the mma.sync form: few tokens give its 3 MMAs per step little to do.  The
// line is that kernel's second tile of 8 tokens (ms, mma.sync / pipeline: 1.5B sb6 at 8 1.67 / 1.71, at 10 1.88 / 1.73, sym 1.71 / 1.66
// and 1.90 / 1.67, 2.9B sb6 2.77 / 2.88 and 3.35 / 2.90), which also costs it the accumulator of its own that its main sum has
// up to 8 (error of the logits against 64 bits, sym: 3.2e-6 at 8, 5.2e-6 from 9 on, pipeline 4.1e-6).
// RWKVQ_TCB_EXACT in the environment (read once) overrides: 0 never, 1 at every batch.
constexpr int kSbMinStreams = 9;
int g_tcb_exact = -2;          // -2 environment not read yet, -1 by stream count, 0 never, 1 always
bool sb_wanted(int B) {
    if (g_tcb_exact == -2) {
        const char* e = getenv("RWKVQ_TCB_EXACT");
        g_tcb_exact = (e == nullptr || (e[0] != '0' && e[0] != '1')) ? -1 : e[0] - '0';
    }
    if (batch_fast() || !tcb_enabled() || B <= 2 || B > kBatchMax || g_tcb_exact == 0) return false;
    return g_tcb_exact == 1 || B >= kSbMinStreams;
}
bool sb_model_ok(const rwkvq_model& m) {
    const int D = m.n_embd, F = m.ffn_dim;
    auto ok = [](const rwkvq_qtensor& t, int rows, int cols) { return gemm_sb_ok(t) && t.rows == rows && t.cols == cols; };
    if (!seq_prep_in_place_ok(D) || !ok(m.head, m.vocab_size, D)) return false;
    for (int l = 0; l < m.n_layer; ++l) {
        const rwkvq_layer& L = m.layers[l];
        for (const rwkvq_qtensor* t : {&L.Wr, &L.Wk, &L.Wv, &L.Wo})
            if (!ok(*t, D, D)) return false;
        if (!ok(L.Wfk, F, D) || !ok(L.Wfv, D, F)) return false;
        for (const rwkvq_qtensor* t : {&L.Wk, &L.Wv})
            if (t->kind != L.Wr.kind || t->bits != L.Wr.bits) return false;
    }
    return true;
}

// The pipeline's row preparation reads and writes float4 (the LayerNorm kernels of the other forms take any row)
bool sb_rows_ok(const rwkvq_model& m, float* const* tshift, float* const* cshift) {
    bool ok = aligned(m.lnout_w, 16) && aligned(m.lnout_b, 16);
    for (int l = 0; l < m.n_layer && ok; ++l) {
        const rwkvq_layer& L = m.layers[l];
        for (const float* p : {L.ln1_w, L.ln1_b, L.ln2_w, L.ln2_b, L.x_mix, L.ffn_x_k, const_cast<const float*>(tshift[l]), const_cast<const float*>(cshift[l])})
            ok = ok && aligned(p, 16);
    }
    return ok;
}

// linears of a step that go to rwkvq_gemm: more streams than the small-batch kernels take, or a tensor without their layout
bool linear_on_gemm(const rwkvq_qtensor& t, int B) {
    return B > 2 && (t.kind == RWKVQ_KIND_SB6 || t.kind == RWKVQ_KIND_SYM) && !(batch_path(B) && mma_layout_of(t) >= 0);
}

struct Workspace {
    float *x, *xs, *rkv, *part, *yl, *og, *xk, *hffn, *xo, *v_first, *logits, *argv, *gemm_ws;
    int* status;             // first word of the workspace: RWKVQ_E_TIMEOUT if a bounded device-side wait of a step ran out
    float* amax;             // [10][B] per-row scale inverses / maxima for the small-batch linears: 6 mix rows, og, xk, hffn, xo
    __half *xs16, *xk16, *xo16;     // fp16 forms of the mix rows, the channel-mix row and the final row
    SbRows rkv_pair[3], d_pair, f_pair;     // operand rows of the tcgen05 pipeline: r / k / v; og, xk or xo; hffn
    int n_chunks;
    size_t part_floats;
    size_t bytes;
};

Workspace carve(const rwkvq_model& m, int B, void* base) {
    const size_t D = m.n_embd, F = m.ffn_dim, R = m.max_rank, V = m.vocab_size, b = B;
    Workspace w{};
    size_t off = 0;
    auto take = [&](size_t n) {
        float* p = base ? reinterpret_cast<float*>(static_cast<char*>(base) + off) : nullptr;
        off += ((n * sizeof(float) + 255) / 256) * 256;
        return p;
    };
    w.status = reinterpret_cast<int*>(take(64));
    w.x = take(b * D); w.xs = take(6 * b * D); w.rkv = take(3 * b * D);
    w.n_chunks = static_cast<int>((D + kLdRows - 1) / kLdRows);
    w.part_floats = 4 * static_cast<size_t>(w.n_chunks) * ((b + kLmMaxN - 1) / kLmMaxN * kLmMaxN) * R;   // upper bound (rep = 1)
    w.part = take(w.part_floats);
    w.yl = take(4 * b * D); w.og = take(b * D); w.xk = take(b * D); w.hffn = take(b * F);
    w.xo = take(b * D); w.v_first = take(b * D); w.logits = take(b * V);
    w.argv = take(2 * b * kArgSlices);
    w.amax = take(10 * b);
    w.xs16 = reinterpret_cast<__half*>(take(3 * b * D));
    w.xk16 = reinterpret_cast<__half*>(take((b * D + 1) / 2));
    w.xo16 = reinterpret_cast<__half*>(take((b * D + 1) / 2));
    if (D % 256 == 0 && F % 256 == 0) {
        auto pair = [&](size_t cols) {
            float* un = take(b);
            return sb_rows(reinterpret_cast<__half*>(take((sb_halves(B, static_cast<int>(cols)) + 1) / 2)), un, B, static_cast<int>(cols));
        };
        for (int k = 0; k < 3; ++k) w.rkv_pair[k] = pair(D);
        w.d_pair = pair(D);
        w.f_pair = pair(F);
    }
    size_t gemm_bytes = 0;                  // only for the linears that reach rwkvq_gemm
    auto with_gemm = [&](const rwkvq_qtensor& t) {
        if (linear_on_gemm(t, B)) gemm_bytes = std::max(gemm_bytes, gemm_rows_bytes(t, B));
    };
    for (int l = 0; l < m.n_layer && m.layers; ++l)
        for (const rwkvq_qtensor* t : {&m.layers[l].Wr, &m.layers[l].Wk, &m.layers[l].Wv, &m.layers[l].Wo, &m.layers[l].Wfk, &m.layers[l].Wfv}) with_gemm(*t);
    with_gemm(m.head);
    w.gemm_ws = take((gemm_bytes + sizeof(float) - 1) / sizeof(float));
    w.bytes = off;
    return w;
}

// One quantized linear for B right-hand sides; the single-vector tensor-core kernel gets
// the K split, everything else goes through the public entry point.
// x16 / x_scale: the fp16 form of x with its per-row scale inverses (what the LayerNorm kernels write
// in fast mode), or null with x_scale = max|x| per row for fp32 rows; y_amax: optional slots max|y| per row is
// merged into; ahead: one stream only.
int linear(const rwkvq_qtensor* t, const float* x, int B, int in, float* y, int out, int epi, const float* resid,
           void* gemm_ws, void* stream, const __half* x16 = nullptr, const float* x_scale = nullptr,
           float* y_amax = nullptr, int* status = nullptr, const Ahead* ahead = nullptr) {
    const int ml = mma_layout_of(*t);
    if (B == 1 && ml >= 0) {
        int rc = validate_qtensor(t, "rwkvq_decode_step(linear)");
        if (rc) return rc;
        return launch_gemv_mma(ml, t, 1, x, RWKVQ_F32, in, y, out, epi, resid, 0, static_cast<cudaStream_t>(stream),
                               nullptr, true, ahead);
    }
    if (batch_path(B) && ml >= 0 && x_scale) {            // small batch: weights read once, tokens as MMA columns
        int rc = validate_qtensor(t, "rwkvq_decode_step(linear)");
        if (rc) return rc;
        const void* xs[1] = {x16 ? static_cast<const void*>(x16) : static_cast<const void*>(x)};
        const float* sc[1] = {x_scale};
        float* ys[1] = {y};
        const float* rs[1] = {resid};
        float* ao[1] = {y_amax};
        if (tcb_pays(B) && gemm_tcb_ok(*t))
            return launch_gemm_tcb(t, 1, xs, x16 != nullptr, sc, B, in, ys, out, epi, rs, ao, status, static_cast<cudaStream_t>(stream));
        return launch_gemv_batch(t, 1, xs, x16 != nullptr, sc, B, in, ys, out, epi, rs, ao, static_cast<cudaStream_t>(stream));
    }
    if (linear_on_gemm(*t, B)) {                            // tcgen05 path for large batches
        int rc = validate_qtensor(t, "rwkvq_decode_step(linear)");
        if (rc) return rc;
        return launch_gemm_rows(*t, x, B, in, y, out, epi, resid, gemm_ws, status, nullptr, static_cast<cudaStream_t>(stream));
    }
    return rwkvq_gemv(t, x, RWKVQ_F32, B, in, y, out, epi, resid, stream);
}

int launch_tmix_core_up(const TmixCoreArgs& tc, const LoraVecArgs& up, int H, cudaStream_t s) {
    decode_carveout<tmix_core_up_kernel>();
    const size_t smem = lora_vec_smem(up.first[up.n_br]);
    if (smem > 40 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(tmix_core_up_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kLvMaxSmem);
        if (e != cudaSuccess) return fail(RWKVQ_E_LIMIT, "tmix_core: %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
    }
    cudaError_t e = launch_pdl(tmix_core_up_kernel, dim3(H, 1), dim3(256), smem, s, tc, up);
    if (e != cudaSuccess) return fail(RWKVQ_E_LAUNCH, "tmix_core: %s", cudaGetErrorString(e));
    return RWKVQ_OK;
}

int lora_rep(int B) { return B > kLmMaxN ? 8 : 1; }

// y_br = (act_br(x_br @ W1_br)) @ W2_br for up to 4 branches, B right-hand sides
int lora_pair(const rwkvq_qtensor* const* t1, const rwkvq_qtensor* const* t2, const float* const* xs,
              float* const* ys, const int* acts, int n_br, int B, int D, int max_rank, float* part,
              size_t part_floats, int n_chunks, cudaStream_t s) {
    LoraDownArgs d{};
    LoraUpArgs u{};
    int max_cols = 0;
    for (int i = 0; i < n_br; ++i) {
        int rc = validate_qtensor(t1[i], "rwkvq_decode_step(lora down)");
        if (rc) return rc;
        rc = validate_qtensor(t2[i], "rwkvq_decode_step(lora up)");
        if (rc) return rc;
        RWKVQ_REQUIRE(t1[i]->rows == D && t1[i]->cols == t2[i]->rows && t1[i]->cols <= max_rank &&
                          t1[i]->cols <= kLmMaxRank,
                      RWKVQ_E_SHAPE, "rwkvq_decode_step: LoRA branch %d has shapes [%d,%d] x [%d,%d]", i,
                      t1[i]->rows, t1[i]->cols, t2[i]->rows, t2[i]->cols);
        d.t[i] = make_view(*t1[i]);
        u.t[i] = make_view(*t2[i]);
        u.act[i] = acts[i];
        if (t2[i]->cols > max_cols) max_cols = t2[i]->cols;
    }
    if (lora_mma_ok(t1, t2, n_br, D)) {
        // both products on the tensor cores, matrices read once; the kernels below keep the odd shapes
        const int n_stride = ((B + 63) / 64) * 64;
        if (static_cast<size_t>(4) * n_stride * max_rank <= part_floats)
            return launch_lora_pair_mma(t1, t2, xs, ys, acts, n_br, B, D, max_rank, part, n_stride, s);
    }
    // large batches: a CTA accumulates 8 sub-chunks of 64 rows, so that the up projection adds
    // 8x fewer partial sums per right-hand side; the groups of 8 right-hand sides are grid.z
    const int rep = lora_rep(B);
    const int chunks = (n_chunks + rep - 1) / rep, groups = (B + kLmMaxN - 1) / kLmMaxN;
    d.part = part; d.ldx = D; d.n_chunks = chunks; d.max_rank = max_rank; d.rep = rep;
    u.part = part; u.ldy = D; u.n_chunks = chunks; u.max_rank = max_rank;
    d.n_stride = u.n_stride = groups * kLmMaxN;
    d.n_cols = u.n_cols = B;
    for (int i = 0; i < n_br; ++i) { d.x[i] = xs[i]; u.y[i] = ys[i]; }
    if (rep > 1) launch_pdl(lora_down_kernel<true>, dim3(chunks, n_br, groups), dim3(256), 0, s, d);
    else launch_pdl(lora_down_kernel<false>, dim3(chunks, n_br, groups), dim3(256), 0, s, d);
    launch_pdl(lora_up_kernel, dim3((max_cols + kLuCols - 1) / kLuCols, n_br, groups), dim3(256), 0, s, u);
    return RWKVQ_OK;
}

}  // namespace

extern "C" {

void rwkvq_profiling_tcb_exact(int on) { g_tcb_exact = on < 0 ? -2 : (on ? 1 : 0); }      // rwkvq_profiling.h

int rwkvq_seq_embed_ln0(const rwkvq_qtensor* emb, const int64_t* tokens, const float* ln_w, const float* ln_b, float* x,
                        int64_t n_tokens, int D, void* stream) {
    int rc = validate_qtensor(emb, "rwkvq_seq_embed_ln0");
    if (rc) return rc;
    RWKVQ_REQUIRE(tokens && ln_w && ln_b && x, RWKVQ_E_NULL, "rwkvq_seq_embed_ln0: null pointer");
    RWKVQ_REQUIRE(n_tokens >= 1 && emb->cols == D && D <= kRowThreads * kRowPer, RWKVQ_E_SHAPE,
                  "rwkvq_seq_embed_ln0: %lld tokens, table [%d, %d], D %d (at most %d)", (long long)n_tokens, emb->rows, emb->cols, D,
                  kRowThreads * kRowPer);
    launch_pdl(embed_ln0_kernel, dim3(static_cast<unsigned>(n_tokens)), dim3(kRowThreads), 0, static_cast<cudaStream_t>(stream),
               make_view(*emb), reinterpret_cast<const long long*>(tokens), ln_w, ln_b, x, D);
    return check_launch("rwkvq_seq_embed_ln0");
}

int rwkvq_seq_layer_norm(const float* x, const float* ln_w, const float* ln_b, float* out, int64_t n_rows, int D, void* stream) {
    RWKVQ_REQUIRE(x && ln_w && ln_b && out, RWKVQ_E_NULL, "rwkvq_seq_layer_norm: null pointer");
    RWKVQ_REQUIRE(n_rows >= 1 && D >= 1 && D <= kRowThreads * kRowPer, RWKVQ_E_SHAPE, "rwkvq_seq_layer_norm: %lld rows of %d (at most %d)",
                  (long long)n_rows, D, kRowThreads * kRowPer);
    launch_ln_shift_mix<0>(static_cast<int>(n_rows), static_cast<cudaStream_t>(stream), x, ln_w, ln_b, nullptr, nullptr, out, D, nullptr, nullptr,
                           0, nullptr, nullptr);
    return check_launch("rwkvq_seq_layer_norm");
}

size_t rwkvq_decode_workspace_bytes(const rwkvq_model* m, int B) {
    if (!m || B < 1) return 0;
    return carve(*m, B, nullptr).bytes;
}

int rwkvq_decode_step(const rwkvq_model* m, int B, const int64_t* tokens, float* const* wkv,
                      float* const* tshift, float* const* cshift, void* workspace, size_t workspace_bytes,
                      float* logits, int64_t* next_tokens, void* stream) {
    RWKVQ_REQUIRE(m && m->layers && tokens && wkv && tshift && cshift && workspace, RWKVQ_E_NULL,
                  "rwkvq_decode_step: null pointer");
    RWKVQ_REQUIRE(B >= 1, RWKVQ_E_SHAPE, "rwkvq_decode_step: B=%d", B);
    RWKVQ_REQUIRE(m->head_size == 64, RWKVQ_E_SHAPE, "rwkvq_decode_step: head size %d, only 64 is built", m->head_size);
    RWKVQ_REQUIRE(m->n_embd % 64 == 0 && m->n_embd <= kRowThreads * kRowPer, RWKVQ_E_LIMIT,
                  "rwkvq_decode_step: n_embd %d (multiple of 64, at most %d)", m->n_embd, kRowThreads * kRowPer);
    const Workspace w = carve(*m, B, workspace);
    RWKVQ_REQUIRE(workspace_bytes >= w.bytes, RWKVQ_E_LIMIT, "rwkvq_decode_step: workspace %zu < %zu bytes",
                  workspace_bytes, w.bytes);
    RWKVQ_REQUIRE(aligned(workspace, 256), RWKVQ_E_ALIGN, "rwkvq_decode_step: workspace must be 256-byte aligned");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int D = m->n_embd, H = D / 64, F = m->ffn_dim, V = m->vocab_size;
    const size_t BD = static_cast<size_t>(B) * D;
    int rc = validate_qtensor(&m->emb, "rwkvq_decode_step(emb)");
    if (rc) return rc;
    float* lg = logits ? logits : w.logits;
    for (int l = 0; l < m->n_layer; ++l)
        RWKVQ_REQUIRE(aligned(wkv[l], 16), RWKVQ_E_ALIGN, "rwkvq_decode_step: the WKV state of layer %d must be 16-byte aligned", l);
    const bool sb = sb_wanted(B) && sb_model_ok(*m) && sb_rows_ok(*m, tshift, cshift);
    if (sb) {
        for (int l = 0; l < m->n_layer; ++l)
            for (const rwkvq_qtensor* t : {&m->layers[l].Wr, &m->layers[l].Wk, &m->layers[l].Wv, &m->layers[l].Wo, &m->layers[l].Wfk, &m->layers[l].Wfv}) {
                rc = validate_qtensor(t, "rwkvq_decode_step(linear)");
                if (rc) return rc;
            }
    }

    bool ahead_on = m->n_layer > 0 && ahead_layer_ok(m->layers[0], D, F, true);
    launch_pdl(embed_ln0_kernel, dim3(B), dim3(kRowThreads), 0, s, make_view(m->emb),
               reinterpret_cast<const long long*>(tokens), m->ln0_w, m->ln0_b, w.x, D);
    for (int l = 0; l < m->n_layer; ++l) {
        const rwkvq_layer& L = m->layers[l];
        const bool layer0 = l == 0;
        // ---- time mix
        // the row maxima feed the small-batch linears: slots 0-5 the six mix rows, 6 og, 7 xk, 8 hffn, 9 xo
        const bool bp = batch_path(B);
        const bool h16 = bp && batch_fast();          // fp16 rows for the single-term kernels; else fp32 rows and their maxima
        const int ml = mma_layout_of(L.Wr);
        const bool rkv_fused = ml >= 0 && mma_layout_of(L.Wk) == ml && mma_layout_of(L.Wv) == ml && L.Wk.rows == L.Wr.rows &&
                               L.Wv.rows == L.Wr.rows && L.Wk.cols == L.Wr.cols && L.Wv.cols == L.Wr.cols;
        float* am = bp ? w.amax : nullptr;
        float *am_og = bp ? w.amax + 6 * B : nullptr, *am_xk = bp ? w.amax + 7 * B : nullptr;
        float *am_h = bp ? w.amax + 8 * B : nullptr;
        if (sb) {
            // LayerNorm 1 + shift + lerps, a CTA per stream and mix; r / k / v rows as operand pairs, the LoRA rows fp32
            SeqPrepArgs pa{};
            pa.x = w.x; pa.ln_w = L.ln1_w; pa.ln_b = L.ln1_b; pa.shift_in = tshift[l]; pa.shift_out = tshift[l]; pa.mix = L.x_mix;
            pa.T = 1; pa.D = D; pa.n_mix = 6;
            const int lin[3] = {0, 2, 3};
            for (int q = 0; q < 6; ++q) { pa.f32[q] = w.xs + q * BD; pa.mode[q] = kPrepF32; }
            for (int q = 0; q < 3; ++q) { pa.pair[lin[q]] = w.rkv_pair[q]; pa.mode[lin[q]] = kPrepPair; }
            if (!layer0) pa.mode[3] |= kPrepF32;
            rc = launch_seq_prep(pa, B, s);
            if (rc) return rc;
        } else {
            launch_ln_shift_mix<6>(B, s, w.x, L.ln1_w, L.ln1_b, tshift[l], L.x_mix, w.xs, D, h16 ? w.xs16 : static_cast<__half*>(nullptr), am, 0b001101, am_og,
                       am_h);      // scales of the r, k, v rows
        }
        float *xr = w.xs, *xw = w.xs + BD, *xk = w.xs + 2 * BD, *xv = w.xs + 3 * BD, *xa = w.xs + 4 * BD,
              *xg = w.xs + 5 * BD;
        float *r = w.rkv, *k = w.rkv + BD, *v = w.rkv + 2 * BD;
        const rwkvq_qtensor* t1[4] = {&L.w1, &L.a1, &L.g1, &L.v1};
        const rwkvq_qtensor* t2[4] = {&L.w2, &L.a2, &L.g2, &L.v2};
        const float* x1[4] = {xw, xa, xg, xv};
        const int act[4] = {1, 0, 2, 0};           // tanh (decay), none, sigmoid (gate), none
        const int n_br = layer0 ? 3 : 4;
        const bool ahead_behind = l + 1 < m->n_layer && ahead_layer_ok((&L)[1], D, F, false);
        const LayerAhead ahead = ahead_on ? LayerAhead(L, ahead_behind ? &L + 1 : nullptr, layer0, wkv[l], BD * 64 * sizeof(float)) : LayerAhead();
        ahead_on = ahead_behind;
        float *yw = w.yl, *ya = w.yl + BD, *yv = w.yl + 2 * BD, *yg = w.yl + 3 * BD;
        TmixCoreArgs tc{r, k, v, yw, ya, layer0 ? nullptr : yv, yg, L.w0, L.a0, L.v0, L.k_k, L.k_a, L.r_k,
                        L.lnx_w, L.lnx_b, w.v_first, wkv[l], w.og, D, H, layer0 ? 1 : 0, sb ? nullptr : am_og};
        // One stream: r / k / v and the LoRA down projections in one launch, the up projections inside the time-mix core
        const bool one = B == 1 && ml >= 0 && rkv_fused && L.Wr.rows == D && L.Wr.cols == D && lora_vec_ok(t1, t2, n_br, D);
        if (one) {
            LoraVecArgs down{}, up{};
            for (const rwkvq_qtensor* t : {&L.Wr, &L.Wk, &L.Wv}) {
                rc = validate_qtensor(t, "rwkvq_decode_step(r/k/v)");
                if (rc) return rc;
            }
            for (int i = 0; i < n_br; ++i) {
                rc = validate_qtensor(t1[i], "rwkvq_decode_step(lora down)");
                if (rc) return rc;
                rc = validate_qtensor(t2[i], "rwkvq_decode_step(lora up)");
                if (rc) return rc;
                down.t[i] = make_view(*t1[i]); up.t[i] = make_view(*t2[i]);
                down.x[i] = x1[i]; down.act[i] = act[i];
                down.first[i + 1] = up.first[i + 1] = down.first[i] + t1[i]->cols;
            }
            down.h = up.h = w.part;
            down.n_br = up.n_br = n_br; down.D = up.D = D;
            const rwkvq_qtensor three[3] = {L.Wr, L.Wk, L.Wv};
            const void* x_each[3] = {xr, xk, xv};
            rc = launch_gemv_mma_lora(ml, three, 3, x_each, r, D, down, ahead.rkv, s);
            if (rc) return rc;
            rc = launch_tmix_core_up(tc, up, H, s);
            if (rc) return rc;
        } else {
            SideLane* lane = side_lane(s);
            Fork fork{lane, s};
            cudaStream_t s_lora = s;
            if (lane) {                                  // fork: the LoRA branches leave the chain here
                rc = fork.start();
                if (rc) return rc;
                s_lora = lane->stream;
            }
            // Up to 16 streams the LoRA pair (two dependent launches) is the longer of the two branches: it then
            // stays on the caller's stream, where its first kernel starts programmatically behind the LayerNorm
            // and stages its weights while that still runs, and r / k / v take the side stream.  So it does beside the tcgen05
            // pipeline at any stream count: that leaves some 50 SMs for the second LoRA launch, but none of its CTAs
            // shares an SM with the first (64 streams: 17 + 11 + 6 us in the other order, 13 + 16 in this).
            cudaStream_t s_rkv = s;
            if (lane && (B <= 16 || sb)) { s_rkv = lane->stream; s_lora = s; }
            auto lora = [&]() {
                float* y2[4] = {yw, ya, yg, yv};
                return lora_pair(t1, t2, x1, y2, act, n_br, B, D, m->max_rank, w.part, w.part_floats, w.n_chunks, s_lora);
            };
            if (sb) {                                  // first in the graph too: 64 streams 2.88 -> 2.81 ms (13 on mma.sync lose 1%)
                rc = lora();
                if (rc) return rc;
            }
            if (B == 1 && ml >= 0 && mma_layout_of(L.Wk) == ml && mma_layout_of(L.Wv) == ml && L.Wk.rows == D &&
                L.Wv.rows == D && L.Wr.rows == D && L.Wk.cols == D && L.Wv.cols == D && L.Wr.cols == D) {
                // r, k, v in one launch: three matrices, three inputs (rows 0, 2, 3 of xs)
                for (const rwkvq_qtensor* t : {&L.Wr, &L.Wk, &L.Wv}) {
                    rc = validate_qtensor(t, "rwkvq_decode_step(r/k/v)");
                    if (rc) return rc;
                }
                const rwkvq_qtensor three[3] = {L.Wr, L.Wk, L.Wv};
                const void* x_each[3] = {xr, xk, xv};
                rc = launch_gemv_mma(ml, three, 3, xr, RWKVQ_F32, D, r, D, RWKVQ_EPI_NONE, nullptr, 1, s_rkv, x_each, true, &ahead.rkv);
                if (rc) return rc;
            } else if (sb) {
                const rwkvq_qtensor three[3] = {L.Wr, L.Wk, L.Wv};
                float* y3[3] = {r, k, v};
                rc = launch_gemm_sb(three, 3, w.rkv_pair, B, y3, D, RWKVQ_EPI_NONE, nullptr, nullptr, w.status, 0, s_rkv, &ahead.rkv);
                if (rc) return rc;
            } else if (bp && rkv_fused) {
                for (const rwkvq_qtensor* t : {&L.Wr, &L.Wk, &L.Wv}) {
                    rc = validate_qtensor(t, "rwkvq_decode_step(r/k/v)");
                    if (rc) return rc;
                }
                const rwkvq_qtensor three[3] = {L.Wr, L.Wk, L.Wv};
                const void* x3[3] = {w.xs16, w.xs16 + 2 * BD, w.xs16 + 3 * BD};
                if (!h16) { x3[0] = xr; x3[1] = xk; x3[2] = xv; }
                const float* a3[3] = {am, am + 2 * B, am + 3 * B};
                float* y3[3] = {r, k, v};
                if (tcb_pays(B) && gemm_tcb_ok(L.Wr))
                    rc = launch_gemm_tcb(three, 3, x3, h16, a3, B, D, y3, D, RWKVQ_EPI_NONE, nullptr, nullptr, w.status, s_rkv);
                else
                    rc = launch_gemv_batch(three, 3, x3, h16, a3, B, D, y3, D, RWKVQ_EPI_NONE, nullptr, nullptr, s_rkv);
                if (rc) return rc;
            } else {
                rc = linear(&L.Wr, xr, B, D, r, D, RWKVQ_EPI_NONE, nullptr, w.gemm_ws, s_rkv, h16 ? w.xs16 : nullptr, am, nullptr, w.status);
                if (rc) return rc;
                rc = linear(&L.Wk, xk, B, D, k, D, RWKVQ_EPI_NONE, nullptr, w.gemm_ws, s_rkv,
                            h16 ? w.xs16 + 2 * BD : nullptr, bp ? am + 2 * B : nullptr, nullptr, w.status);
                if (rc) return rc;
                rc = linear(&L.Wv, xv, B, D, v, D, RWKVQ_EPI_NONE, nullptr, w.gemm_ws, s_rkv,
                            h16 ? w.xs16 + 3 * BD : nullptr, bp ? am + 3 * B : nullptr, nullptr, w.status);
                if (rc) return rc;
            }
            if (!sb) {
                rc = lora();
                if (rc) return rc;
            }
            rc = fork.join();                            // before the time-mix core
            if (rc) return rc;
            launch_pdl(tmix_core_kernel, dim3(H, B), dim3(64), 0, s, tc);
        }
        if (sb) {
            const float* res[1] = {w.x};
            float *yx[1] = {w.x}, *yh[1] = {w.hffn};
            rc = launch_split_rows(w.og, D, D, B, w.d_pair, nullptr, s);
            if (rc) return rc;
            rc = launch_gemm_sb(&L.Wo, 1, &w.d_pair, B, yx, D, RWKVQ_EPI_ADD, res, nullptr, w.status, 0, s);
            if (rc) return rc;
            SeqPrepArgs pc{};
            pc.x = w.x; pc.ln_w = L.ln2_w; pc.ln_b = L.ln2_b; pc.shift_in = cshift[l]; pc.shift_out = cshift[l]; pc.mix = L.ffn_x_k;
            pc.T = 1; pc.D = D; pc.n_mix = 1; pc.mode[0] = kPrepPair; pc.pair[0] = w.d_pair;
            rc = launch_seq_prep(pc, B, s);
            if (rc) return rc;
            rc = launch_gemm_sb(&L.Wfk, 1, &w.d_pair, B, yh, F, RWKVQ_EPI_RELU2, nullptr, nullptr, w.status, 0, s, &ahead.key);
            if (rc) return rc;
            rc = launch_split_rows(w.hffn, F, F, B, w.f_pair, nullptr, s);
            if (rc) return rc;
            rc = launch_gemm_sb(&L.Wfv, 1, &w.f_pair, B, yx, D, RWKVQ_EPI_ADD, res, nullptr, w.status, 0, s);
            if (rc) return rc;
            continue;
        }
        rc = linear(&L.Wo, w.og, B, D, w.x, D, RWKVQ_EPI_ADD, w.x, w.gemm_ws, stream, nullptr, am_og, nullptr, w.status);
        if (rc) return rc;
        // ---- channel mix
        launch_ln_shift_mix<1>(B, s, w.x, L.ln2_w, L.ln2_b, cshift[l], L.ffn_x_k, w.xk, D, h16 ? w.xk16 : static_cast<__half*>(nullptr), am_xk, 1, static_cast<float*>(nullptr),
                   static_cast<float*>(nullptr));
        rc = linear(&L.Wfk, w.xk, B, D, w.hffn, F, RWKVQ_EPI_RELU2, nullptr, w.gemm_ws, stream, h16 ? w.xk16 : nullptr, am_xk, am_h,
                    w.status, &ahead.key);
        if (rc) return rc;
        rc = linear(&L.Wfv, w.hffn, B, F, w.x, D, RWKVQ_EPI_ADD, w.x, w.gemm_ws, stream, nullptr, am_h, nullptr, w.status);
        if (rc) return rc;
    }
    if (sb) {
        SeqPrepArgs po{};
        po.x = w.x; po.ln_w = m->lnout_w; po.ln_b = m->lnout_b; po.T = 1; po.D = D; po.n_mix = 1; po.mode[0] = kPrepPair; po.pair[0] = w.d_pair;
        rc = launch_seq_prep(po, B, s);
        if (rc) return rc;
        rc = launch_gemm_sb(&m->head, 1, &w.d_pair, B, &lg, V, RWKVQ_EPI_NONE, nullptr, nullptr, w.status, 0, s);
        if (rc) return rc;
    } else {
        float* am_xo = batch_path(B) ? w.amax + 9 * B : nullptr;
        const bool xo_h16 = am_xo && batch_fast();
        launch_ln_shift_mix<0>(B, s, w.x, m->lnout_w, m->lnout_b, nullptr, nullptr, w.xo, D, xo_h16 ? w.xo16 : static_cast<__half*>(nullptr),
                   am_xo, 1, static_cast<float*>(nullptr), static_cast<float*>(nullptr));
        rc = linear(&m->head, w.xo, B, D, lg, V, RWKVQ_EPI_NONE, nullptr, w.gemm_ws, stream, xo_h16 ? w.xo16 : nullptr, am_xo, nullptr,
                    w.status);
        if (rc) return rc;
    }
    if (next_tokens) {
        float* pv = w.argv;
        int* pi = reinterpret_cast<int*>(w.argv + static_cast<size_t>(B) * kArgSlices);
        launch_pdl(argmax_partial_kernel, dim3(kArgSlices, B), dim3(256), 0, s, static_cast<const float*>(lg), pv, pi, V);
        launch_pdl(argmax_final_kernel, dim3(B), dim3(kArgSlices), 0, s, static_cast<const float*>(pv), static_cast<const int*>(pi), reinterpret_cast<long long*>(next_tokens), V);
    }
    return check_launch("rwkvq_decode_step");
}

}  // extern "C"
