// Block quantizers for the sb6 and sym layouts on the device.  sb6: the search the reference runs in torch on the
// host (rwkv_quant/calibration/groupwise.py:207-300, `_gw_one` with 8 blocks of 32 per super-block).
//
// One THREAD owns one block (32 weights, 16 in the sym layout): its weights stay in registers, so the sums,
// extremes and errors of the search are plain register arithmetic (a warp per super-block with shuffle
// trees took 1263 us for [10240, 2560] at 4 bits, five shuffles for every sum of 32); 8 (16) adjacent lanes hold a
// super-block.  Sums add in the order of a butterfly over the block (i with i + 16, then + 8, ..).
// A code rint(u / s) is found by one saturating multiply-add and the addition and subtraction of 1.5 * 2^23; only where
// that comes within its error of a half does the block repeat the step with the rounded division, so every
// code is the division's.  Two neighbouring weights share a packed instruction everywhere else.  The packed entry points write
// the file buffers from the same registers.
// Bound: instruction issue (some 230 scalar operations a weight in the 8-factor search) and, at 160 registers, three CTAs an SM;
// [10240, 2560] at 4 bits 268 -> 192 us against scalar code with the clamp as two operations (235 registers).
//   per block      s0 = max((max - min) / qmax, 1e-8); with search, for each factor f of
//                  {0.7 .. 1.05}: q = clamp(rint((w - min) / (f s0))), the closed-form least-squares
//                  (s, m) for those codes (weights E[x^2] of the input channel when given), the codes
//                  again with (s, m), their squared error; the (s, m) with the smallest error wins,
//                  the first factor on ties
//   per super-block  d = fp16(max s / 63), qs = clamp(rint(s / d), 1, 63), dm = fp16(max|m| / 31),
//                  qm = clamp(rint(m / dm), -31, 31); s' = max(fp16(qs d), 1e-8), m' = fp16(qm dm)
//   per weight     q = clamp(rint((w - m') / s'), 0, qmax)
// All in fp32 with IEEE division and round-half-to-even, like the torch code.  The sums run in the
// order above, torch's in its own: (s, m) agree to their last bits, so a code can differ
// where a quotient sits within an ulp of a rounding boundary or two factors tie (measured: 3 codes
// per million against tensors packed by the reference).
#include <cuda_fp16.h>

#include "rwkvq_common.cuh"

namespace rwkvq {

namespace {

__device__ __forceinline__ float hrt(float x) { return __half2float(__float2half_rn(x)); }
__device__ __forceinline__ float clampf(float v, float lo, float hi) { return fminf(fmaxf(v, lo), hi); }

// A block's values as pairs of neighbours, so that one packed instruction serves two weights: the search is bound by
// instruction issue.  Every packed operation rounds each half as its scalar form does.
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
// A packed product is a multiply-add onto nz = -0, which the launch passes in: the compiler draws a packed product (stated
// rounding or not) into a packed sum behind it, and of two errors near a tie the other one is then the smaller.
__device__ __forceinline__ uint64_t bits2(float2 v) { return (static_cast<uint64_t>(__float_as_uint(v.y)) << 32) | __float_as_uint(v.x); }
__device__ __forceinline__ float2 of_bits(uint64_t v) { return make_float2(__uint_as_float(static_cast<uint32_t>(v)), __uint_as_float(static_cast<uint32_t>(v >> 32))); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(bits2(a)), "l"(bits2(b)));
    return of_bits(r);
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(bits2(a)), "l"(bits2(b)), "l"(bits2(c)));
    return of_bits(r);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b, float nz) { return fma2(a, b, both(nz)); }
// sum of 2 N values in butterfly order (value i with i + N, then + N / 2, ..)
template <int N>
__device__ __forceinline__ float tree(float2 (&v)[N]) {
#pragma unroll
    for (int h = N / 2; h > 0; h >>= 1)
#pragma unroll
        for (int i = 0; i < N / 2; ++i)
            if (i < h) v[i] = add2(v[i], v[i + h]);
    return __fadd_rn(v[0].x, v[0].y);
}
// maximum over the G adjacent lanes of a super-block
template <int G>
__device__ __forceinline__ float gmax(float v) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
    return v;
}

// q[i] = clamp(rint((x[i] - m) / s), lo, hi) for a block (lo, hi integers), as the rounded subtraction and division give it.
template <int N>
__device__ __forceinline__ void codes_exact(const float2 (&x)[N], float m, float s, float lo, float hi, float2 (&q)[N]) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
        q[i].x = clampf(rintf(__fdiv_rn(__fsub_rn(x[i].x, m), s)), lo, hi);
        q[i].y = clampf(rintf(__fdiv_rn(__fsub_rn(x[i].y, m), s)), lo, hi);
    }
}
// The quotient's place in [lo, hi] as v = saturate((x - m) / (R s) - lo / R), R = hi - lo: the clamp is part of the
// multiply-add (a NaN gives 0 there, code lo; the division with the clamp behind it gives lo too), rint(R v) comes from
// adding and subtracting 1.5 * 2^23.  Distance of R v from the rounded quotient plus -lo, for quotients Q the clamp does
// not decide (|Q| <= H = max(-lo, hi) + 1), in units of 2^-24: 3 each from 1 / s, 1 / R and their product on |x / s| <=
// |m / s| + H, 4 on |m / s|, 1 on -lo / R, 1 on v (R <= 2 H), 2 in the rounded subtraction and division.  Together below
// 5e-7 (H + |m / s|); a block with a product that near to a half takes the division instead.
template <int N>
__device__ __forceinline__ void codes_of(const float2 (&x)[N], float m, float s, float lo, float hi, float2 (&q)[N]) {
    const float inv = __fdiv_rn(1.0f, s), R = hi - lo, r1 = __fmul_rn(inv, __fdiv_rn(1.0f, R)), c = __fmaf_rn(-m, r1, -__fdiv_rn(lo, R));
    float dev = 0.f;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const float2 v = make_float2(__saturatef(__fmaf_rn(x[i].x, r1, c)), __saturatef(__fmaf_rn(x[i].y, r1, c)));
        const float2 r = add2(fma2(v, both(R), both(12582912.f)), both(-12582912.f));
        const float2 d = fma2(v, both(-R), r);
        dev = fmaxf(dev, fmaxf(fabsf(d.x), fabsf(d.y)));
        q[i] = lo == 0.f ? r : add2(r, both(lo));
    }
    if (dev > 0.5f - 5e-7f * (fmaxf(-lo, hi) + 1.0f + fabsf(m) * inv)) codes_exact(x, m, s, lo, hi, q);
}

struct QuantOut {                    // unpacked parts, or file buffers (those that are null are not written)
    uint8_t* q;                      // [rows, cols] codes (sym: int8)
    uint8_t* qs;                     // [rows, blocks]
    int8_t* qm;                      // [rows, blocks] (sb6)
    __half *d, *dm;
    uint8_t *packed, *qh, *qh2, *qsqm;
};

template <int N>
__device__ __forceinline__ void load_pairs(const float* w, float2 (&x)[N]) {
    if ((reinterpret_cast<uintptr_t>(w) & 15) == 0) {
#pragma unroll
        for (int i = 0; i < N / 2; ++i) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(w) + i);
            x[2 * i] = make_float2(v.x, v.y);
            x[2 * i + 1] = make_float2(v.z, v.w);
        }
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) x[i] = make_float2(__ldg(w + 2 * i), __ldg(w + 2 * i + 1));
    }
}

template <bool AW>
__global__ void __launch_bounds__(128) quant_sb6_kernel(const float* __restrict__ w, long long ldw, int rows, int nsb, int bits, int search,
                                                        const float* __restrict__ ex2, const QuantOut o, float nz) {
    const long long blk = static_cast<long long>(blockIdx.x) * 128 + threadIdx.x, n_blocks = static_cast<long long>(rows) * nsb * 8;
    const bool live = blk < n_blocks;                     // whole super-blocks (8 adjacent lanes) together
    const long long bb = live ? blk : n_blocks - 1;
    const int nb = nsb * 8, row = static_cast<int>(bb / nb), bi = static_cast<int>(bb % nb);
    const float* wp = w + static_cast<size_t>(row) * ldw + bi * 32;
    const float qmax = static_cast<float>((1 << bits) - 1);
    float2 x[16], e[AW ? 16 : 1];
    load_pairs(wp, x);
    if (AW) {
#pragma unroll
        for (int i = 0; i < 16; ++i)
            e[AW ? i : 0] = make_float2(fmaxf(__ldg(ex2 + bi * 32 + 2 * i), 1e-12f), fmaxf(__ldg(ex2 + bi * 32 + 2 * i + 1), 1e-12f));
    }
    float mn = x[0].x, mx = x[0].x;
#pragma unroll
    for (int i = 0; i < 16; ++i) { mn = fminf(mn, fminf(x[i].x, x[i].y)); mx = fmaxf(mx, fmaxf(x[i].x, x[i].y)); }
    float scale = fmaxf(__fdiv_rn(__fsub_rn(mx, mn), qmax), 1e-8f);
    if (search) {
        float2 t[16];
        float es = 32.f;
        if (AW) {
#pragma unroll
            for (int i = 0; i < 16; ++i) t[i] = e[AW ? i : 0];
            es = tree(t);
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) t[i] = AW ? mul2(e[AW ? i : 0], x[i], nz) : x[i];
        const float wm = __fdiv_rn(tree(t), es);
        float best_s = 0.f, best_m = 0.f, best_e = 0.f;
        const float factors[8] = {0.7f, 0.75f, 0.8f, 0.85f, 0.9f, 0.95f, 1.0f, 1.05f};
#pragma unroll 1
        for (int fi = 0; fi < 8; ++fi) {
            const float sc = __fmul_rn(scale, factors[fi]);
            float2 q[16];
            codes_of<16>(x, mn, sc, 0.f, qmax, q);
#pragma unroll
            for (int i = 0; i < 16; ++i) t[i] = AW ? mul2(e[AW ? i : 0], q[i], nz) : q[i];
            const float qmean = __fdiv_rn(tree(t), es);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                q[i] = add2(q[i], both(-qmean));
                const float2 dx = add2(x[i], both(-wm));
                t[i] = AW ? mul2(mul2(e[AW ? i : 0], q[i], nz), dx, nz) : mul2(q[i], dx, nz);
            }
            const float cov = tree(t);
#pragma unroll
            for (int i = 0; i < 16; ++i) t[i] = AW ? mul2(mul2(e[AW ? i : 0], q[i], nz), q[i], nz) : mul2(q[i], q[i], nz);
            const float var = fmaxf(tree(t), 1e-12f);
            float s_ls = __fdiv_rn(cov, var);
            const float m_ls = __fsub_rn(wm, __fmul_rn(s_ls, qmean));       // separate multiply and subtract, as in torch
            s_ls = s_ls > 1e-8f ? s_ls : sc;
            codes_of<16>(x, m_ls, s_ls, 0.f, qmax, q);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                // w - (q * s + m), no contraction; its square is that of the reference's difference
                const float2 r = add2(add2(mul2(q[i], both(-s_ls), nz), both(-m_ls)), x[i]);
                t[i] = AW ? mul2(e[AW ? i : 0], mul2(r, r, nz), nz) : mul2(r, r, nz);
            }
            const float err = tree(t);
            if (fi == 0 || err < best_e) { best_s = s_ls; best_m = m_ls; best_e = err; }
        }
        scale = fmaxf(best_s, 1e-8f);
        mn = best_m;
    }
    // super-block: 8 adjacent lanes
    const float d = hrt(fmaxf(__fdiv_rn(fmaxf(gmax<8>(scale), 0.f), 63.f), 1e-12f));
    const float dm = hrt(fmaxf(__fdiv_rn(gmax<8>(fabsf(mn)), 31.f), 1e-12f));
    const float qsv = clampf(rintf(__fdiv_rn(scale, d)), 1.f, 63.f);
    // an all-zero super-block has dm = fp16(1e-12) = 0: min code 0 (the reference's 0 / 0 leaves NaN there)
    const float qmv = (dm > 0.f || mn != 0.f) ? clampf(rintf(__fdiv_rn(mn, dm)), -31.f, 31.f) : 0.f;
    const float s2 = fmaxf(hrt(__fmul_rn(qsv, d)), 1e-8f);
    const float m2 = hrt(__fmul_rn(qmv, dm));
    float2 q[16];
    codes_of<16>(x, m2, s2, 0.f, qmax, q);
    // the super-block's 8 scale and 8 min codes as two 48-bit streams, for the lane that stores them
    uint64_t ss = 0, ms = 0;
    const uint32_t mine = static_cast<uint32_t>(qsv) | (static_cast<uint32_t>(static_cast<int>(qmv) + 31) << 8);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t v = __shfl_sync(0xFFFFFFFFu, mine, i, 8);
        ss |= static_cast<uint64_t>(v & 63u) << (6 * i);
        ms |= static_cast<uint64_t>((v >> 8) & 63u) << (6 * i);
    }
    if (!live) return;
    const size_t B = static_cast<size_t>(blk);
    uint32_t c[32];
#pragma unroll
    for (int i = 0; i < 16; ++i) { c[2 * i] = static_cast<uint32_t>(q[i].x); c[2 * i + 1] = static_cast<uint32_t>(q[i].y); }
    if ((bi & 7) == 0) {
        o.d[B >> 3] = __float2half_rn(d);
        o.dm[B >> 3] = __float2half_rn(dm);
        if (o.qsqm) {
            uint32_t* p = reinterpret_cast<uint32_t*>(o.qsqm + (B >> 3) * 12);
            p[0] = static_cast<uint32_t>(ss);
            p[1] = static_cast<uint32_t>(ss >> 32) | (static_cast<uint32_t>(ms) << 16);
            p[2] = static_cast<uint32_t>(ms >> 16);
        }
    }
    if (o.q) {
        uint32_t b[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) b[i] = c[4 * i] | (c[4 * i + 1] << 8) | (c[4 * i + 2] << 16) | (c[4 * i + 3] << 24);
        uint4* p = reinterpret_cast<uint4*>(o.q + B * 32);
        p[0] = make_uint4(b[0], b[1], b[2], b[3]);
        p[1] = make_uint4(b[4], b[5], b[6], b[7]);
        o.qs[B] = static_cast<uint8_t>(qsv);
        o.qm[B] = static_cast<int8_t>(qmv);
    }
    if (o.packed) {                   // byte j of a block: column j (low nibble), column j + 16 (high nibble)
        uint32_t b[4] = {0, 0, 0, 0}, h = 0, h2 = 0;
#pragma unroll
        for (int i = 0; i < 16; ++i) b[i >> 2] |= ((c[i] & 15u) | ((c[i + 16] & 15u) << 4)) << (8 * (i & 3));
#pragma unroll
        for (int i = 0; i < 32; ++i) { h |= ((c[i] >> 4) & 1u) << i; h2 |= ((c[i] >> 5) & 1u) << i; }
        reinterpret_cast<uint4*>(o.packed)[B] = make_uint4(b[0], b[1], b[2], b[3]);
        if (o.qh) reinterpret_cast<uint32_t*>(o.qh)[B] = h;
        if (o.qh2) reinterpret_cast<uint32_t*>(o.qh2)[B] = h2;
    }
}

// The symmetric layout (blocks of 16, int8 block-scale codes against one fp16 per 256 weights;
// calibration/groupwise.py:358-473 `_sym_one`): 16 adjacent lanes hold a super-block.  Per block
// s0 = max(max|w|, 1e-12) / qmax and, over the caller's factors (the
// reference's 19 float32 nodes of linspace(0.7, 1.15), or 1.0 alone), the s = f s0 with the
// smallest (weighted) squared error of w - clamp(rint(w / s)) s, the first on ties; then
// d = fp16(max s / 127), qs = clamp(rint(s / d), -128, 127), s' = fp16(qs d) and
// q = clamp(rint(w / s')) (0 where s' is 0).
template <bool AW>
__global__ void __launch_bounds__(128) quant_sym_kernel(const float* __restrict__ w, long long ldw, int rows, int nsb, int bits,
                                                        const float* __restrict__ factors, int n_factors, const float* __restrict__ ex2,
                                                        const QuantOut o, float nz) {
    const long long blk = static_cast<long long>(blockIdx.x) * 128 + threadIdx.x, n_blocks = static_cast<long long>(rows) * nsb * 16;
    const bool live = blk < n_blocks;
    const long long bb = live ? blk : n_blocks - 1;
    const int nb = nsb * 16, row = static_cast<int>(bb / nb), bi = static_cast<int>(bb % nb);
    const float* wp = w + static_cast<size_t>(row) * ldw + bi * 16;
    const float qmax = static_cast<float>((1 << (bits - 1)) - 1), qmin = -qmax - 1.f;
    float2 x[8], e[AW ? 8 : 1];
    load_pairs(wp, x);
    float mx = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (AW) e[AW ? i : 0] = make_float2(fmaxf(__ldg(ex2 + bi * 16 + 2 * i), 1e-12f), fmaxf(__ldg(ex2 + bi * 16 + 2 * i + 1), 1e-12f));
        mx = fmaxf(mx, fmaxf(fabsf(x[i].x), fabsf(x[i].y)));
    }
    const float base = __fdiv_rn(fmaxf(mx, 1e-12f), qmax);
    float best_s = base, best_e = 0.f;
    float2 q[8], t[8];
#pragma unroll 1
    for (int fi = 0; fi < n_factors; ++fi) {
        const float s = __fmul_rn(base, __ldg(factors + fi));
        codes_of<8>(x, 0.f, s, qmin, qmax, q);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float2 dlt = add2(x[i], mul2(q[i], both(-s), nz));
            t[i] = AW ? mul2(e[AW ? i : 0], mul2(dlt, dlt, nz), nz) : mul2(dlt, dlt, nz);
        }
        const float err = tree(t);
        if (fi == 0 || err < best_e) { best_s = s; best_e = err; }
    }
    const float d = hrt(fmaxf(__fdiv_rn(fmaxf(gmax<16>(best_s), 0.f), 127.f), 1e-12f));
    float qsv = clampf(rintf(__fdiv_rn(best_s, d)), -128.f, 127.f);
    if (!(qsv == qsv)) qsv = 0.f;           // 0 / 0: code 0, as the reference writes
    const float s2 = hrt(__fmul_rn(qsv, d));
    if (fabsf(s2) > 0.f) {
        codes_of<8>(x, 0.f, s2, qmin, qmax, q);
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) q[i] = both(0.f);
    }
    if (!live) return;
    int v[16];
#pragma unroll
    for (int i = 0; i < 8; ++i) { v[2 * i] = static_cast<int>(q[i].x); v[2 * i + 1] = static_cast<int>(q[i].y); }
    const size_t B = static_cast<size_t>(blk);
    o.qs[B] = static_cast<uint8_t>(static_cast<int8_t>(qsv));
    if ((bi & 15) == 0) o.d[B >> 4] = __float2half_rn(d);
    if (o.q) {
        uint32_t b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            b[i] = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) b[i] |= (static_cast<uint32_t>(v[4 * i + k]) & 0xFFu) << (8 * k);
        }
        reinterpret_cast<uint4*>(o.q)[B] = make_uint4(b[0], b[1], b[2], b[3]);
    }
    if (o.packed) {                   // stored code = value + 32; byte j of a block: column j (low nibble), column j + 8 (high nibble)
        uint32_t c[16], b[2] = {0, 0}, h = 0, h2 = 0;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            c[i] = static_cast<uint32_t>(v[i] + 32);
            h |= ((c[i] >> 4) & 1u) << i;
            h2 |= ((c[i] >> 5) & 1u) << i;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) b[i >> 2] |= ((c[i] & 15u) | ((c[i + 8] & 15u) << 4)) << (8 * (i & 3));
        reinterpret_cast<uint2*>(o.packed)[B] = make_uint2(b[0], b[1]);
        reinterpret_cast<unsigned short*>(o.qh)[B] = static_cast<unsigned short>(h);
        reinterpret_cast<unsigned short*>(o.qh2)[B] = static_cast<unsigned short>(h2);
    }
}

int run_sb6(const char* who, const float* w, int64_t ldw, int rows, int cols, int bits, int search, const float* ex2, const QuantOut& o,
            cudaStream_t s) {
    RWKVQ_REQUIRE(rows >= 1 && cols >= 256 && cols % 256 == 0 && ldw >= cols, RWKVQ_E_SHAPE,
                  "%s: [%d, %d] (columns in multiples of 256), ldw %lld", who, rows, cols, (long long)ldw);
    RWKVQ_REQUIRE(bits >= 4 && bits <= 6, RWKVQ_E_DTYPE, "%s: %d bits (4, 5 or 6)", who, bits);
    const int nsb = cols / 256;
    const long long ctas = (static_cast<long long>(rows) * nsb * 8 + 127) / 128;
    RWKVQ_REQUIRE(ctas <= 0x7FFFFFFFLL, RWKVQ_E_LIMIT, "%s: tensor too large for one launch", who);
    if (ex2 && search) quant_sb6_kernel<true><<<static_cast<unsigned>(ctas), 128, 0, s>>>(w, ldw, rows, nsb, bits, search, ex2, o, -0.0f);
    else quant_sb6_kernel<false><<<static_cast<unsigned>(ctas), 128, 0, s>>>(w, ldw, rows, nsb, bits, search, ex2, o, -0.0f);
    return check_launch(who);
}
int run_sym(const char* who, const float* w, int64_t ldw, int rows, int cols, int bits, const float* factors, int n_factors,
            const float* ex2, const QuantOut& o, cudaStream_t s) {
    RWKVQ_REQUIRE(rows >= 1 && cols >= 256 && cols % 256 == 0 && ldw >= cols, RWKVQ_E_SHAPE,
                  "%s: [%d, %d] (columns in multiples of 256), ldw %lld", who, rows, cols, (long long)ldw);
    RWKVQ_REQUIRE(bits == 6 || bits == 8, RWKVQ_E_DTYPE, "%s: %d bits (6 or 8)", who, bits);
    RWKVQ_REQUIRE(n_factors >= 1 && n_factors <= 64, RWKVQ_E_LIMIT, "%s: %d factors", who, n_factors);
    const int nsb = cols / 256;
    const long long ctas = (static_cast<long long>(rows) * nsb * 16 + 127) / 128;
    RWKVQ_REQUIRE(ctas <= 0x7FFFFFFFLL, RWKVQ_E_LIMIT, "%s: tensor too large for one launch", who);
    if (ex2) quant_sym_kernel<true><<<static_cast<unsigned>(ctas), 128, 0, s>>>(w, ldw, rows, nsb, bits, factors, n_factors, ex2, o, -0.0f);
    else quant_sym_kernel<false><<<static_cast<unsigned>(ctas), 128, 0, s>>>(w, ldw, rows, nsb, bits, factors, n_factors, ex2, o, -0.0f);
    return check_launch(who);
}

}  // namespace
}  // namespace rwkvq

using namespace rwkvq;

extern "C" int rwkvq_quantize_sb6(const float* w, int64_t ldw, int rows, int cols, int bits, int search, const float* ex2,
                                  uint8_t* q, uint8_t* qs, int8_t* qm, void* d, void* dm, void* stream) {
    RWKVQ_REQUIRE(w && q && qs && qm && d && dm, RWKVQ_E_NULL, "rwkvq_quantize_sb6: null pointer");
    RWKVQ_REQUIRE(aligned(q, 16), RWKVQ_E_ALIGN, "rwkvq_quantize_sb6: q must be 16-byte aligned");
    QuantOut o{};
    o.q = q; o.qs = qs; o.qm = qm; o.d = static_cast<__half*>(d); o.dm = static_cast<__half*>(dm);
    return run_sb6("rwkvq_quantize_sb6", w, ldw, rows, cols, bits, search, ex2, o, static_cast<cudaStream_t>(stream));
}

extern "C" int rwkvq_quantize_sb6_packed(const float* w, int64_t ldw, int rows, int cols, int bits, int search, const float* ex2,
                                         uint8_t* codes_packed, uint8_t* qh, uint8_t* qh2, uint8_t* qsqm, void* d, void* dm, void* stream) {
    RWKVQ_REQUIRE(w && codes_packed && qsqm && d && dm && (bits < 5 || qh) && (bits < 6 || qh2), RWKVQ_E_NULL,
                  "rwkvq_quantize_sb6_packed: null pointer");
    RWKVQ_REQUIRE(aligned(codes_packed, 16) && aligned(qh, 4) && aligned(qh2, 4) && aligned(qsqm, 4), RWKVQ_E_ALIGN,
                  "rwkvq_quantize_sb6_packed: unaligned buffer");
    QuantOut o{};
    o.packed = codes_packed; o.qh = bits >= 5 ? qh : nullptr; o.qh2 = bits >= 6 ? qh2 : nullptr; o.qsqm = qsqm;
    o.d = static_cast<__half*>(d); o.dm = static_cast<__half*>(dm);
    return run_sb6("rwkvq_quantize_sb6_packed", w, ldw, rows, cols, bits, search, ex2, o, static_cast<cudaStream_t>(stream));
}

extern "C" int rwkvq_quantize_sym(const float* w, int64_t ldw, int rows, int cols, int bits, const float* factors, int n_factors,
                                  const float* ex2, int8_t* q, int8_t* qs, void* d, void* stream) {
    RWKVQ_REQUIRE(w && q && qs && d && factors, RWKVQ_E_NULL, "rwkvq_quantize_sym: null pointer");
    RWKVQ_REQUIRE(aligned(q, 16), RWKVQ_E_ALIGN, "rwkvq_quantize_sym: q must be 16-byte aligned");
    QuantOut o{};
    o.q = reinterpret_cast<uint8_t*>(q); o.qs = reinterpret_cast<uint8_t*>(qs); o.d = static_cast<__half*>(d);
    return run_sym("rwkvq_quantize_sym", w, ldw, rows, cols, bits, factors, n_factors, ex2, o, static_cast<cudaStream_t>(stream));
}

extern "C" int rwkvq_quantize_sym6_packed(const float* w, int64_t ldw, int rows, int cols, const float* factors, int n_factors,
                                          const float* ex2, uint8_t* codes_packed, uint8_t* qh, uint8_t* qh2, int8_t* qs, void* d, void* stream) {
    RWKVQ_REQUIRE(w && codes_packed && qh && qh2 && qs && d && factors, RWKVQ_E_NULL, "rwkvq_quantize_sym6_packed: null pointer");
    RWKVQ_REQUIRE(aligned(codes_packed, 8) && aligned(qh, 2) && aligned(qh2, 2), RWKVQ_E_ALIGN, "rwkvq_quantize_sym6_packed: unaligned buffer");
    QuantOut o{};
    o.packed = codes_packed; o.qh = qh; o.qh2 = qh2; o.qs = reinterpret_cast<uint8_t*>(qs); o.d = static_cast<__half*>(d);
    return run_sym("rwkvq_quantize_sym6_packed", w, ldw, rows, cols, 6, factors, n_factors, ex2, o, static_cast<cudaStream_t>(stream));
}
