// Time-mix core of long sequences: decay / gates / key normalisation, the WKV-7 recurrence and the
// group-norm tail in two kernels, the recurrence in chunks of kC = 8 steps (chunked form of the delta rule).
//
// With P_t the product of the decays of steps 1 .. t of a chunk, S_0 the state before it and, per key column,
//     a~_t = P_{t-1} a_t,  r~_t = P_t r_t,  b~_t = b_t / P_t,  k~_t = k_t / P_t
// a state row's recurrence (backends/metal/quant_model.py:118-125, math models/rwkv7_ref.py:244-254) unrolls to
//     u_t = S_0 a~_t + sum_{j<t}  u_j L_tj + v_j K_tj         L_tj = b~_j a~_t,  K_tj = k~_j a~_t
//     y_t = S_0 r~_t + sum_{j<=t} u_j E_tj + v_j F_tj         E_tj = b~_j r~_t,  F_tj = k~_j r~_t
//     S   = (S_0 + sum_j u_j b~_j^T + v_j k~_j^T) diag(P_8)
// and with M = (I - L)^-1 (unit lower triangular, by substitution)
//     u_t = S_0 a^_t + sum_j N_tj v_j      a^ = M a~,        N = M K
//     y_t = S_0 r^_t + sum_j G_tj v_j      r^ = r~ + E M a~, G = F + E N
// Nothing in that depends on the state but the products with S_0, which are independent of one another: the
// first kernel makes the operands of every chunk of every head in parallel, and the second, the only serial one,
// is left with dense products.  Step by step, every step waited for a reduction over the key columns.
// All fp32; the model's decays are above exp(-0.6066) = 0.54, so P_t stays above 0.0077.
//
// Measured per layer, 32 heads, against the step-by-step scan with its separate pre and tail kernels: T = 512 batch 1
// 112 -> 86 us, batch 16 552 -> 505 us (under ncu: operands 203, scan 315).  What bounds the scan: shared-memory reads into
// registers on small grids (128 bytes per clock and SM), issue latency at 7 warps per SM on large ones.
#include "rwkvq_wkv_chunk.cuh"

#include <algorithm>

#include "rwkvq_decode_parts.cuh"
#include "rwkvq_tc.cuh"

namespace rwkvq {

constexpr int kC = 8, kS = 64;
// one chunk of one head, contiguous: a^, r^, b~, k~, v [kC][64], P_8 [64], N [t][j], G [t][j]
constexpr int kOffA = 0, kOffR = kC * kS, kOffB = 2 * kC * kS, kOffK = 3 * kC * kS, kOffV = 4 * kC * kS, kOffP = 5 * kC * kS,
              kOffN = kOffP + kS, kOffG = kOffN + kC * kC, kChunkFloats = kOffG + kC * kC;
static_assert(kChunkFloats * 4 % 16 == 0, "bulk copies");

size_t wkv_chunk_floats(int B, int T, int H) { return static_cast<size_t>(B) * ((T + kC - 1) / kC) * H * kChunkFloats; }

// ------------------------------------------------------------------ operands
// 64 threads (one per channel) per (chunk, head), four heads side by side in a CTA.  Bound: HBM (seven rows
// read, five written per token).
constexpr int kPreUnits = 4, kPrePitch = kS + 4;
constexpr size_t kPreStage = sizeof(float) * 7 * kC * kPreUnits * kS;      // 8 rows hit 8 different 16-byte bank groups
struct PreSmem {
    float a[kC][kPrePitch], r[kC][kPrePitch], b[kC][kPrePitch], k[kC][kPrePitch];
    float L[kC][kC], K[kC][kC], E[kC][kC], F[kC][kC], M[kC][kC], A[kC][kC];     // A = E M
    float red[2][2 * kC];
};

__device__ __forceinline__ float gate_sigmoid(float x) { return __frcp_rn(1.0f + expf(-x)); }      // a NaN stays one, +-inf give 1 and 0

__global__ void __launch_bounds__(64 * kPreUnits, 3) wkv_operands_kernel(const WkvChunkArgs p, int n_chunks) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int unit = threadIdx.x >> 6, d = threadIdx.x & 63, wp = d >> 5, lane = d & 31;
    PreSmem& s = reinterpret_cast<PreSmem*>(smem_raw)[unit];
    const int groups = (p.H + kPreUnits - 1) / kPreUnits;
    const int hg = blockIdx.x % groups, bc = blockIdx.x / groups, hd = hg * kPreUnits + unit;
    const int b = bc / n_chunks, ch = bc % n_chunks;
    auto sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(1 + unit) : "memory"); };
    const bool live = hd < p.H;
    const int c = (live ? hd : 0) * kS + d, D = p.H * kS;
    const float w0 = __ldg(p.w0 + c), a0 = __ldg(p.a0 + c), kkw = __ldg(p.k_k + c), kaw = __ldg(p.k_a + c), rkw = __ldg(p.r_k + c);
    const float v0 = p.yv ? __ldg(p.v0 + c) : 0.f;
    const int t0 = ch * kC, n = min(kC, p.T - t0);
    // all rows of the four heads' chunk as bulk copies of 1 KB into shared memory (56 loads a thread would not all
    // stay in flight in registers); the room is used again for the operands once the rows are in registers
    __shared__ uint64_t full;
    if (threadIdx.x == 0) {
        mbar_init(&full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_launch_dependents();
    pdl_wait();
    float* stage = reinterpret_cast<float*>(smem_raw);             // [7][kC][kPreUnits * 64]
    const int arrays = p.yv ? 7 : 5, heads = min(kPreUnits, p.H - hg * kPreUnits);
    if (threadIdx.x == 0) mbar_expect_tx(&full, static_cast<uint32_t>(arrays * n * heads * kS * 4));
    __syncthreads();
    if (static_cast<int>(threadIdx.x) < arrays * n) {
        const int ar = threadIdx.x / n, t = threadIdx.x % n;
        const float* base = ar == 0 ? p.r : ar == 1 ? p.k : ar == 2 ? p.v : ar == 3 ? p.yw : ar == 4 ? p.ya : ar == 5 ? p.yv : p.v_first;
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         smem_addr(stage + (ar * kC + t) * (kPreUnits * kS))),
                     "l"(base + (static_cast<size_t>(b) * p.T + t0 + t) * D + hg * kPreUnits * kS), "r"(heads * kS * 4), "r"(smem_addr(&full))
                     : "memory");
    }
    if (!mbar_wait_bounded(&full, 0) && threadIdx.x == 0) atomicCAS(p.status, 0, RWKVQ_E_TIMEOUT);
    // steps beyond T are neutral: decay 1, everything else 0
    float r[kC], k[kC], v[kC], yw[kC], ya[kC], yv[kC], vf[kC];
#pragma unroll
    for (int t = 0; t < kC; ++t) {
        const bool in = live && t < n;
        const float* q = stage + t * (kPreUnits * kS) + threadIdx.x;
        constexpr int AS = kC * kPreUnits * kS;
        r[t] = in ? q[0] : 0.f;
        k[t] = in ? q[AS] : 0.f;
        v[t] = in ? q[2 * AS] : 0.f;
        yw[t] = in ? q[3 * AS] : 0.f;
        ya[t] = in ? q[4 * AS] : 0.f;
        yv[t] = (in && p.yv) ? q[5 * AS] : 0.f;
        vf[t] = (in && p.yv) ? q[6 * AS] : 0.f;
    }
    __syncthreads();
    if (!live) return;
    float q[2 * kC];                                   // sums over the head: |k k_k|^2 and r k' r_k of every step
#pragma unroll
    for (int t = 0; t < kC; ++t) {
        yw[t] = t < n ? expf(-0.606531f * gate_sigmoid(yw[t] + w0)) : 1.f;        // the decay
        ya[t] = gate_sigmoid(ya[t] + a0);                                        // the gate
        if (p.yv) v[t] = t < n ? v[t] + (vf[t] - v[t]) * gate_sigmoid(yv[t] + v0) : 0.f;
        vf[t] = k[t] * kkw;                                                    // un-normalised removal key
        k[t] = k[t] * (1.0f + (ya[t] - 1.0f) * kaw);
        q[t] = vf[t] * vf[t];
        q[kC + t] = r[t] * k[t] * rkw;
    }
    // 16 sums over the 32 lanes, halving the live values at each of the first four stages; lane bits 0..3 select
#pragma unroll
    for (int m = 1, live_n = 2 * kC; m < 32; m <<= 1) {
        if (live_n > 1) {
            const int half = live_n >> 1;
            const bool up = (lane & m) != 0;
#pragma unroll
            for (int i = 0; i < kC; ++i) {
                if (i < half) {
                    const float send = up ? q[i] : q[i + half], keep = up ? q[i + half] : q[i];
                    q[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, m);
                }
            }
            live_n = half;
        } else {
            q[0] += __shfl_xor_sync(0xFFFFFFFFu, q[0], m);
        }
    }
    if (lane < 16) s.red[wp][(lane & 1) * 8 + (lane & 2) * 2 + ((lane & 4) >> 1) + ((lane & 8) >> 3)] = q[0];
    sync();
    float P = 1.f, at_[kC];
    // 1 / |k k_k| of the 8 steps, a step per lane: the rounded root is some 15 instructions
    const float inv_mine = __frsqrt_rn(s.red[0][lane & (kC - 1)] + s.red[1][lane & (kC - 1)] + 1e-12f);
#pragma unroll
    for (int t = 0; t < kC; ++t) {
        const float inv = __shfl_sync(0xFFFFFFFFu, inv_mine, t);
        const float kk = vf[t] * inv, a = -kk, bb = kk * ya[t];
        at_[t] = P * a;                                                        // P_{t-1} a_t
        P *= yw[t];
        const float ip = __frcp_rn(P);
        s.a[t][d] = at_[t];
        r[t] *= P;
        s.r[t][d] = r[t];
        yw[t] = ip * bb;
        k[t] *= ip;
        s.b[t][d] = yw[t];
        s.k[t][d] = k[t];
    }
    if (d < kC && d < n) p.dp[(static_cast<size_t>(b) * p.T + t0 + d) * p.H + hd] = s.red[0][kC + d] + s.red[1][kC + d];
    sync();
    {
        const int j = d >> 3, t = d & 7;
        float2 l = make_float2(0.f, 0.f), kx = l, e = l, f = l;
#pragma unroll 4
        for (int i = 0; i < kS; i += 4) {
            const float4 x = *reinterpret_cast<const float4*>(&s.a[t][i]), y = *reinterpret_cast<const float4*>(&s.r[t][i]);
            const float4 u = *reinterpret_cast<const float4*>(&s.b[j][i]), g = *reinterpret_cast<const float4*>(&s.k[j][i]);
            const float2 x0 = make_float2(x.x, x.y), x1 = make_float2(x.z, x.w), y0 = make_float2(y.x, y.y), y1 = make_float2(y.z, y.w);
            const float2 u0 = make_float2(u.x, u.y), u1 = make_float2(u.z, u.w), g0 = make_float2(g.x, g.y), g1 = make_float2(g.z, g.w);
            l = __ffma2_rn(x0, u0, l); l = __ffma2_rn(x1, u1, l);
            kx = __ffma2_rn(x0, g0, kx); kx = __ffma2_rn(x1, g1, kx);
            e = __ffma2_rn(y0, u0, e); e = __ffma2_rn(y1, u1, e);
            f = __ffma2_rn(y0, g0, f); f = __ffma2_rn(y1, g1, f);
        }
        s.L[t][j] = j < t ? l.x + l.y : 0.f;
        s.K[t][j] = j < t ? kx.x + kx.y : 0.f;
        s.E[t][j] = j <= t ? e.x + e.y : 0.f;
        s.F[t][j] = j <= t ? f.x + f.y : 0.f;
    }
    sync();
    float* blk = p.ops + ((static_cast<size_t>(b) * p.H + hd) * n_chunks + ch) * kChunkFloats;
    if (d < 2 * kC) {                                  // columns of M (d < 8) and N: substitution with I and K on the right
        const int col = d & 7;
        const bool is_n = d >= kC;
        float X[kC];
#pragma unroll
        for (int t = 0; t < kC; ++t) {
            float x = is_n ? s.K[t][col] : (t == col ? 1.f : 0.f);
#pragma unroll
            for (int i = 0; i < t; ++i) x = fmaf(s.L[t][i], X[i], x);
            X[t] = x;
        }
#pragma unroll
        for (int t = 0; t < kC; ++t) {
            float y = is_n ? s.F[t][col] : 0.f;
#pragma unroll
            for (int i = 0; i <= t; ++i) y = fmaf(s.E[t][i], X[i], y);
            if (is_n) {
                blk[kOffN + t * kC + col] = X[t];
                blk[kOffG + t * kC + col] = y;
            } else {
                s.M[t][col] = X[t];
                s.A[t][col] = y;
            }
        }
    }
    sync();
#pragma unroll
    for (int t = 0; t < kC; ++t) {
        const float4 m0 = *reinterpret_cast<const float4*>(&s.M[t][0]), m1 = *reinterpret_cast<const float4*>(&s.M[t][4]);
        const float4 e0 = *reinterpret_cast<const float4*>(&s.A[t][0]), e1 = *reinterpret_cast<const float4*>(&s.A[t][4]);
        const float m[kC] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w}, e[kC] = {e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, e1.w};
        float x = 0.f, y = r[t];
#pragma unroll
        for (int j = 0; j <= t; ++j) { x = fmaf(m[j], at_[j], x); y = fmaf(e[j], at_[j], y); }
        blk[kOffA + t * kS + d] = x;
        blk[kOffR + t * kS + d] = y;
        blk[kOffB + t * kS + d] = yw[t];
        blk[kOffK + t * kS + d] = k[t];
        blk[kOffV + t * kS + d] = v[t];
    }
    blk[kOffP + d] = P;
}

// ------------------------------------------------------------------ scan
// A thread owns R state rows x 8 columns (columns 4c .. 4c + 3 and 32 + 4c ..: conflict-free 16-byte reads), 8 lanes
// span a row; SPLIT CTAs share a head (the rows are independent).  Operand blocks arrive as single bulk copies
// of 11 KB in a ring.  The partial products of the 8 steps are summed over the 8 lanes of a row by halving the
// live values at each shuffle stage, so that lane c ends with step step_of(c) of all its R rows.
template <int R, int SPLIT>
struct ScanGeo {
    static constexpr int THREADS = 512 / R / SPLIT;
    static constexpr int SLOTS = 4;
    static constexpr int UP = kS + 4;                               // pitch of the u / y exchange: 8 steps in 8 bank groups
    static constexpr size_t SMEM = sizeof(float) * (SLOTS * kChunkFloats + 2 * kC * UP) + 64;
};

__device__ __forceinline__ void chunk_cols(const float* row, int c, float2 (&d)[4]) {
    const float4 lo = *reinterpret_cast<const float4*>(row + 4 * c), hi = *reinterpret_cast<const float4*>(row + 32 + 4 * c);
    d[0] = make_float2(lo.x, lo.y); d[1] = make_float2(lo.z, lo.w);
    d[2] = make_float2(hi.x, hi.y); d[3] = make_float2(hi.z, hi.w);
}
// the same as loads that keep their place in the program: the small tiles' scan is a chain of shared-memory
// latencies unless the loads of a phase all go out before its arithmetic
__device__ __forceinline__ void chunk_cols_now(const float* row, int c, float2 (&d)[4]) {
    const uint32_t a = smem_addr(row + 4 * c);
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(d[0].x), "=f"(d[0].y), "=f"(d[1].x), "=f"(d[1].y) : "r"(a));
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(d[2].x), "=f"(d[2].y), "=f"(d[3].x), "=f"(d[3].y) : "r"(a + 128));
}
__device__ __forceinline__ float chunk_dot(const float2 (&h)[4], const float2 (&x)[4]) {
    float2 p = __fmul2_rn(h[0], x[0]);
    p = __ffma2_rn(h[1], x[1], p);
    p = __ffma2_rn(h[2], x[2], p);
    p = __ffma2_rn(h[3], x[3], p);
    return p.x + p.y;
}
// The partial sums of 8 steps over the 8 lanes of a row.  Lane c takes the steps in the order e ^ my_t, so that at
// every stage it keeps its lower half and sends the upper one, whose steps the partner keeps: no selection.
template <int R>
__device__ __forceinline__ void step_products(const float2 (&h)[R][4], const float* blk, int c, int t, float (&o)[2 * R]) {
    float2 x[4], y[4];
    chunk_cols(blk + kOffA + t * kS, c, x);
    chunk_cols(blk + kOffR + t * kS, c, y);
#pragma unroll
    for (int j = 0; j < R; ++j) {
        o[2 * j] = chunk_dot(h[j], x);
        o[2 * j + 1] = chunk_dot(h[j], y);
    }
}
template <int N>
__device__ __forceinline__ void take_half(float (&keep)[N], const float (&send)[N], int m) {
#pragma unroll
    for (int i = 0; i < N; ++i) keep[i] += __shfl_xor_sync(0xFFFFFFFFu, send[i], m);
}
template <int R>
__device__ __forceinline__ void step_quad(const float2 (&h)[R][4], const float* blk, int c, int my_t, int e, float (&o)[2 * R]) {
    float p[2 * R], q[2 * R];
    step_products<R>(h, blk, c, my_t ^ e, o);
    step_products<R>(h, blk, c, my_t ^ (e + 4), p);
    take_half<2 * R>(o, p, 1);
    step_products<R>(h, blk, c, my_t ^ (e + 2), q);
    step_products<R>(h, blk, c, my_t ^ (e + 6), p);
    take_half<2 * R>(q, p, 1);
    take_half<2 * R>(o, q, 2);
}

template <int R, int SPLIT>
__global__ void __launch_bounds__(ScanGeo<R, SPLIT>::THREADS) wkv_scan_kernel(const WkvChunkArgs p, int n_chunks) {
    using G = ScanGeo<R, SPLIT>;
    constexpr bool TAIL = SPLIT == 1;                               // the CTA sees whole heads: group norm, bonus and gate here
    constexpr int TL = G::THREADS / kC, TR = kS / TL;               // tail: lanes per step, rows per lane
    extern __shared__ __align__(16) float smem[];
    float* su = smem + G::SLOTS * kChunkFloats;                     // [kC][kS]: u_t of the rows
    float* sy = su + kC * G::UP;                                      // [kC][kS]: y_t
    __shared__ uint64_t full[G::SLOTS];
    const int bh = blockIdx.x / SPLIT, b = bh / p.H, hd = bh % p.H;
    const int tid = threadIdx.x, c = tid & 7, dv0 = (blockIdx.x % SPLIT) * (kS / SPLIT) + (tid >> 3) * R;
    const int my_t = (c & 1) * 4 + (c & 2) + ((c & 4) >> 2);        // the step this lane ends up with
    const size_t D = static_cast<size_t>(p.H) * kS, row0 = static_cast<size_t>(b) * p.T * D + hd * kS;
    const float* src = p.ops + static_cast<size_t>(bh) * n_chunks * kChunkFloats;
    auto issue = [&](int ch) {
        const int s = ch % G::SLOTS;
        mbar_expect_tx(&full[s], kChunkFloats * 4);
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         smem_addr(smem + s * kChunkFloats)),
                     "l"(src + static_cast<size_t>(ch) * kChunkFloats), "r"(kChunkFloats * 4), "r"(smem_addr(&full[s]))
                     : "memory");
    };
    if (tid == 0) {
        for (int s = 0; s < G::SLOTS; ++s) mbar_init(&full[s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int ch = 0; ch < G::SLOTS - 1 && ch < n_chunks; ++ch) issue(ch);
    }
    float2 h[R][4];
    const size_t hbase = (static_cast<size_t>(bh) * kS + dv0) * kS;
#pragma unroll
    for (int j = 0; j < R; ++j) {
        if (p.h_in) chunk_cols(p.h_in + hbase + j * kS, c, h[j]);
        else {
#pragma unroll
            for (int q = 0; q < 4; ++q) h[j][q] = make_float2(0.f, 0.f);
        }
    }
    const int tt = tid / TL, tr = (tid % TL) * TR;                  // tail: this thread's step and first row
    float lnw[TAIL ? TR : 1], lnb[TAIL ? TR : 1];
    if constexpr (TAIL) {
#pragma unroll
        for (int i = 0; i < TR; ++i) { lnw[i] = __ldg(p.ln_w + hd * kS + tr + i); lnb[i] = __ldg(p.ln_b + hd * kS + tr + i); }
    }
    bool ok = true;
    for (int ch = 0; ch < n_chunks; ++ch) {
        __syncthreads();                                            // chunk ch - 1 is consumed
        if (tid == 0 && ch + G::SLOTS - 1 < n_chunks) issue(ch + G::SLOTS - 1);
        const int t0 = ch * kC, n = min(kC, p.T - t0);
        float gg[TAIL ? TR : 1], dp = 0.f;
        if constexpr (TAIL) {
            if (tt < n) {
                const float* gp = p.g + row0 + (t0 + tt) * D + tr;
#pragma unroll
                for (int i = 0; i < TR; i += 4) {
                    const float4 v4 = __ldcs(reinterpret_cast<const float4*>(gp + i));
                    gg[i] = v4.x; gg[i + 1] = v4.y; gg[i + 2] = v4.z; gg[i + 3] = v4.w;
                }
                dp = __ldg(p.dp + (static_cast<size_t>(b) * p.T + t0 + tt) * p.H + hd);
            }
        }
        if (ok) ok = mbar_wait_bounded(&full[ch % G::SLOTS], (ch / G::SLOTS) & 1);
        const float* blk = smem + (ch % G::SLOTS) * kChunkFloats;
        float uy[2 * R];                                            // u and y of step my_t for the R rows
        if constexpr (R <= 2) {
            float2 xa[kC][4], xr[kC][4];
#pragma unroll
            for (int e = 0; e < kC; ++e) chunk_cols_now(blk + kOffA + (my_t ^ e) * kS, c, xa[e]);
#pragma unroll
            for (int e = 0; e < kC; ++e) chunk_cols_now(blk + kOffR + (my_t ^ e) * kS, c, xr[e]);
            float u[R][kC], y[R][kC];
#pragma unroll
            for (int j = 0; j < R; ++j)
#pragma unroll
                for (int e = 0; e < kC; ++e) { u[j][e] = chunk_dot(h[j], xa[e]); y[j][e] = chunk_dot(h[j], xr[e]); }
#pragma unroll
            for (int m = 1, half = 4; half > 0; m <<= 1, half >>= 1)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (e < half) {
#pragma unroll
                        for (int j = 0; j < R; ++j) {
                            u[j][e] += __shfl_xor_sync(0xFFFFFFFFu, u[j][e + half], m);
                            y[j][e] += __shfl_xor_sync(0xFFFFFFFFu, y[j][e + half], m);
                        }
                    }
#pragma unroll
            for (int j = 0; j < R; ++j) { uy[2 * j] = u[j][0]; uy[2 * j + 1] = y[j][0]; }
        } else {
            float q[2 * R];
            step_quad<R>(h, blk, c, my_t, 0, uy);
            step_quad<R>(h, blk, c, my_t, 1, q);
            take_half<2 * R>(uy, q, 4);
        }
        float nv[kC], gv[kC];
        {
            const float4* np = reinterpret_cast<const float4*>(blk + kOffN + my_t * kC);
            const float4* gp = reinterpret_cast<const float4*>(blk + kOffG + my_t * kC);
            const float4 n0 = np[0], n1 = np[1], e0 = gp[0], e1 = gp[1];
            nv[0] = n0.x; nv[1] = n0.y; nv[2] = n0.z; nv[3] = n0.w; nv[4] = n1.x; nv[5] = n1.y; nv[6] = n1.z; nv[7] = n1.w;
            gv[0] = e0.x; gv[1] = e0.y; gv[2] = e0.z; gv[3] = e0.w; gv[4] = e1.x; gv[5] = e1.y; gv[6] = e1.z; gv[7] = e1.w;
        }
        auto rows_of = [&](const float* q, float (&o)[R]) {         // R consecutive values
            if constexpr (R >= 4) {
#pragma unroll
                for (int i = 0; i < R; i += 4) {
                    const float4 v4 = *reinterpret_cast<const float4*>(q + i);
                    o[i] = v4.x; o[i + 1] = v4.y; o[i + 2] = v4.z; o[i + 3] = v4.w;
                }
            } else {
#pragma unroll
                for (int i = 0; i < R; ++i) o[i] = q[i];
            }
        };
#pragma unroll
        for (int j = 0; j < kC; ++j) {
            float v[R];
            rows_of(blk + kOffV + j * kS + dv0, v);
            if (j <= my_t) {                                        // not only zero factors: a NaN of a later step stays there
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    uy[2 * i] = fmaf(nv[j], v[i], uy[2 * i]);
                    uy[2 * i + 1] = fmaf(gv[j], v[i], uy[2 * i + 1]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < R; ++i) su[my_t * G::UP + dv0 + i] = uy[2 * i];
        if (TAIL) {
#pragma unroll
            for (int i = 0; i < R; ++i) sy[my_t * G::UP + dv0 + i] = uy[2 * i + 1];
        } else if (my_t < n) {
            float* y = p.y + row0 + (t0 + my_t) * D + dv0;
#pragma unroll
            for (int i = 0; i < R; ++i) y[i] = uy[2 * i + 1];
        }
        if constexpr (R <= 2) {
            float2 xb[kC][4], xk[kC][4];
#pragma unroll
            for (int t = 0; t < kC; ++t) { chunk_cols_now(blk + kOffB + t * kS, c, xb[t]); chunk_cols_now(blk + kOffK + t * kS, c, xk[t]); }
#pragma unroll
            for (int t = 0; t < kC; ++t)
#pragma unroll
                for (int j = 0; j < R; ++j) {
                    const float v = blk[kOffV + t * kS + dv0 + j];
                    const float2 v2 = make_float2(v, v);
#pragma unroll
                    for (int q = 0; q < 4; ++q) h[j][q] = __ffma2_rn(v2, xk[t][q], h[j][q]);
                }
            __syncwarp();
#pragma unroll
            for (int t = 0; t < kC; ++t)
#pragma unroll
                for (int j = 0; j < R; ++j) {
                    const float u = su[t * G::UP + dv0 + j];
                    const float2 u2 = make_float2(u, u);
#pragma unroll
                    for (int q = 0; q < 4; ++q) h[j][q] = __ffma2_rn(u2, xb[t][q], h[j][q]);
                }
        } else {
            __syncwarp();                                               // u of a row group comes from its own 8 lanes
#pragma unroll
            for (int t = 0; t < kC; ++t) {
                float2 x[4], y[4];
                float u[R], v[R];
                chunk_cols(blk + kOffB + t * kS, c, x);
                chunk_cols(blk + kOffK + t * kS, c, y);
                rows_of(su + t * G::UP + dv0, u);
                rows_of(blk + kOffV + t * kS + dv0, v);
#pragma unroll
                for (int j = 0; j < R; ++j) {
                    const float2 u2 = make_float2(u[j], u[j]), v2 = make_float2(v[j], v[j]);
#pragma unroll
                    for (int q = 0; q < 4; ++q) h[j][q] = __ffma2_rn(u2, x[q], __ffma2_rn(v2, y[q], h[j][q]));
                }
            }
        }
        {
            float2 x[4];
            chunk_cols(blk + kOffP, c, x);
#pragma unroll
            for (int j = 0; j < R; ++j)
#pragma unroll
                for (int q = 0; q < 4; ++q) h[j][q] = __fmul2_rn(h[j][q], x[q]);
        }
        if constexpr (TAIL) {
            __syncthreads();
            float y[TR], m = 0.f, var = 0.f;
#pragma unroll
            for (int i = 0; i < TR; i += 4) {
                const float4 v4 = *reinterpret_cast<const float4*>(sy + tt * G::UP + tr + i);
                y[i] = v4.x; y[i + 1] = v4.y; y[i + 2] = v4.z; y[i + 3] = v4.w;
                m += (v4.x + v4.y) + (v4.z + v4.w);
            }
#pragma unroll
            for (int o = 1; o < TL; o <<= 1) m += __shfl_xor_sync(0xFFFFFFFFu, m, o);
            m /= kS;
#pragma unroll
            for (int i = 0; i < TR; ++i) { y[i] -= m; var = fmaf(y[i], y[i], var); }
#pragma unroll
            for (int o = 1; o < TL; o <<= 1) var += __shfl_xor_sync(0xFFFFFFFFu, var, o);
            const float inv = 1.0f / sqrtf(var / kS + 64e-5f);
            if (tt < n) {
                float* o = p.og + row0 + (t0 + tt) * D + tr;
#pragma unroll
                for (int i = 0; i < TR; i += 4) {
                    const float4 v4 = *reinterpret_cast<const float4*>(blk + kOffV + tt * kS + tr + i);
                    *reinterpret_cast<float4*>(o + i) = make_float4((y[i] * inv * lnw[i] + lnb[i] + dp * v4.x) * gg[i],
                                                                    (y[i + 1] * inv * lnw[i + 1] + lnb[i + 1] + dp * v4.y) * gg[i + 1],
                                                                    (y[i + 2] * inv * lnw[i + 2] + lnb[i + 2] + dp * v4.z) * gg[i + 2],
                                                                    (y[i + 3] * inv * lnw[i + 3] + lnb[i + 3] + dp * v4.w) * gg[i + 3]);
                }
            }
        }
    }
    if (!ok) atomicCAS(p.status, 0, RWKVQ_E_TIMEOUT);
#pragma unroll
    for (int j = 0; j < R; ++j) {
        float* o = p.h_out + hbase + j * kS;
        *reinterpret_cast<float4*>(o + 4 * c) = make_float4(h[j][0].x, h[j][0].y, h[j][1].x, h[j][1].y);
        *reinterpret_cast<float4*>(o + 32 + 4 * c) = make_float4(h[j][2].x, h[j][2].y, h[j][3].x, h[j][3].y);
    }
}

// The tail where a scan CTA does not see whole heads: a CTA per token, a thread per 8 channels (v' from the operand blocks),
// whose rows leave as the output projection reads them: fp16 under a power of two per token.  Bound: latency, then L2 (four
// arrays read, one of halves written; as a pass of its own behind an fp32 tail the scaling cost a launch and 8 bytes a value).
__global__ void __launch_bounds__(512) wkv_chunk_tail_kernel(const WkvChunkArgs p, int n_chunks) {
    __shared__ float red[16];
    const bool live = static_cast<int>(threadIdx.x) * 8 < p.H * kS;     // whole warps: H need not be a multiple of 4
    const int c = live ? threadIdx.x * 8 : 0, hd = c / kS, ci = c % kS, b = blockIdx.x / p.T, t = blockIdx.x % p.T;
    const size_t at = static_cast<size_t>(blockIdx.x) * p.H * kS + c;
    pdl_launch_dependents();
    auto load8 = [](const float* q, float (&o)[8]) {
        const float4 lo = __ldcg(reinterpret_cast<const float4*>(q)), hi = __ldcg(reinterpret_cast<const float4*>(q) + 1);
        o[0] = lo.x; o[1] = lo.y; o[2] = lo.z; o[3] = lo.w; o[4] = hi.x; o[5] = hi.y; o[6] = hi.z; o[7] = hi.w;
    };
    float lw[8], lb[8], y[8], g[8], v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) { lw[i] = __ldg(p.ln_w + c + i); lb[i] = __ldg(p.ln_b + c + i); }
    pdl_wait();
    load8(p.y + at, y);
    load8(p.g + at, g);
    load8(p.ops + ((static_cast<size_t>(b) * p.H + hd) * n_chunks + t / kC) * kChunkFloats + kOffV + (t % kC) * kS + ci, v);
    const float dp = __ldcg(p.dp + static_cast<size_t>(blockIdx.x) * p.H + hd);
    // A head's sum over its 8 lanes, from sums of neighbours, in the order of a butterfly over 32 lanes of two channels each: the fp16
    // rounding behind it carries another order's 1e-7 into 2^-11 of a value, 7e-4 of the logits 24 layers on.
    auto head_sum = [](float (&x)[4]) {
#pragma unroll
        for (int o = 4; o > 0; o >>= 1)
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] += __shfl_xor_sync(0xFFFFFFFFu, x[i], o);
        return (x[0] + x[2]) + (x[1] + x[3]);
    };
    float two[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) two[i] = y[2 * i] + y[2 * i + 1];
    const float m = head_sum(two) / kS;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float d0 = y[2 * i] - m, d1 = y[2 * i + 1] - m;
        two[i] = d0 * d0 + d1 * d1;
        y[2 * i] = d0; y[2 * i + 1] = d1;
    }
    const float inv = 1.0f / sqrtf(head_sum(two) / kS + 64e-5f);
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        y[i] = (y[i] * inv * lw[i] + lb[i] + dp * v[i]) * g[i];
        if (live) amax = fmaxf(amax, fabsf(y[i]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
    __syncthreads();
    amax = red[0];
    for (int w = 1; w < static_cast<int>(blockDim.x >> 5); ++w) amax = fmaxf(amax, red[w]);
    int e = 0;                                                      // |x 2^(14 - e)| <= 2^14, as row_scale_kernel
    if (amax > 0.f && amax < INFINITY) frexpf(amax, &e);
    const float sc = ldexpf(1.f, 14 - e);
    if (threadIdx.x == 0) p.og_scale[blockIdx.x] = sc;
    uint32_t h[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __half2 x = __floats2half2_rn(y[2 * i] * sc, y[2 * i + 1] * sc);
        h[i] = *reinterpret_cast<const uint32_t*>(&x);
    }
    if (live) *reinterpret_cast<uint4*>(p.og16 + static_cast<size_t>(blockIdx.x) * p.og_pitch + c) = make_uint4(h[0], h[1], h[2], h[3]);
}

template <int R, int SPLIT>
static int launch_scan(const WkvChunkArgs& p, int n_chunks, cudaStream_t s) {
    using G = ScanGeo<R, SPLIT>;
    // A scan is as slow as its fullest SM: beside the conversions of the side lane CTAs would pile up where those leave room first
    // (1 x 512 tokens 56 -> 95 us), so a grid of up to one or two CTAs per SM asks for as much shared memory as keeps it to that.
    const int ctas = p.B * p.H * SPLIT;
    constexpr size_t kOne = 116 * 1024, kTwo = 78 * 1024;
    static_assert(G::SMEM <= kOne, "the largest a launch may ask for");
    const size_t smem = std::max(G::SMEM, !p.spread ? 0 : ctas <= 148 ? kOne : ctas <= 296 ? kTwo : 0);
    cudaError_t e = cudaFuncSetAttribute(wkv_scan_kernel<R, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kOne));
    if (e != cudaSuccess) return fail(RWKVQ_E_LIMIT, "wkv_scan: %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
    // a plain launch: CTAs that start while the kernel before still fills the chip pile up on the SMs it leaves
    // first, and the scan of one batch element takes three times as long
    wkv_scan_kernel<R, SPLIT><<<ctas, G::THREADS, smem, s>>>(p, n_chunks);
    if (SPLIT == 1) return RWKVQ_OK;
    e = launch_pdl(wkv_chunk_tail_kernel, dim3(static_cast<unsigned>(p.B * p.T)), dim3((p.H * kS / 8 + 31) / 32 * 32), 0, s, p, n_chunks);
    if (e != cudaSuccess) return fail(RWKVQ_E_LAUNCH, "wkv_chunk_tail: %s", cudaGetErrorString(e));
    return RWKVQ_OK;
}

int launch_wkv_chunked(const WkvChunkArgs& p, cudaStream_t s) {
    const int n_chunks = (p.T + kC - 1) / kC, groups = (p.H + kPreUnits - 1) / kPreUnits;
    static_assert(sizeof(PreSmem) * kPreUnits <= kPreStage, "operands over the staged rows");
    const long long blocks = static_cast<long long>(p.B) * n_chunks * groups;
    RWKVQ_REQUIRE(blocks < (1ll << 31), RWKVQ_E_LIMIT, "wkv_chunked: too many tokens");
    RWKVQ_REQUIRE(aligned(p.h_in, 16) && aligned(p.h_out, 16) && p.H <= 64, RWKVQ_E_ALIGN,
                  "wkv_chunked: states on 16-byte boundaries, at most 64 heads");
    cudaError_t e = cudaFuncSetAttribute(wkv_operands_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kPreStage));
    if (e != cudaSuccess) return fail(RWKVQ_E_LIMIT, "wkv_operands: shared memory: %s", cudaGetErrorString(e));
    e = launch_pdl(wkv_operands_kernel, dim3(static_cast<unsigned>(blocks)), dim3(64 * kPreUnits), kPreStage, s, p, n_chunks);
    if (e != cudaSuccess) return fail(RWKVQ_E_LAUNCH, "wkv_operands: %s", cudaGetErrorString(e));
    // Few heads: several CTAs per head, so that a chunk is short, with two rows per thread (one: twice the
    // shared-memory reads, 64 against 56 us at 32 heads; four: one warp per CTA); full grids: the largest tile with
    // the tail inside (4 rows per thread, twice the warps: 302 against 296 us)
    const int pairs = p.B * p.H;
    static_assert(kChunkSplitPairs == 148, "the lines below");
    if (pairs <= 74) return launch_scan<2, 4>(p, n_chunks, s);
    if (pairs <= 148) return launch_scan<2, 2>(p, n_chunks, s);
    return launch_scan<8, 1>(p, n_chunks, s);
}

}  // namespace rwkvq
