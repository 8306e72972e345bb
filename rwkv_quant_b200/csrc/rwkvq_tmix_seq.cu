// Time-mix core of short sequences (speculative-verify runs, prompts of a few tokens): decay / gates / key normalisation,
// the WKV-7 recurrence and the group-norm tail of every token of a (sequence, head) in one CTA, the counterpart of
// tmix_core_kernel (one token) for several.  Reference math: backends/metal/quant_model.py:638-728, fused_tail.py:43-76.
//
// Bound: latency.  As three launches (operands, scan, tail) with five intermediate arrays the links cost more than the
// steps.  Four warps do the steps: rows of the state are independent, so between steps there is no barrier, only the sums
// over a row's eight lanes; a thread's tile of 4 rows x 8 columns takes 11 shared-memory reads a step (a quarter row each for
// 256 threads took 21 and 0.5 us a step).  Four more turn rows into operands a chunk ahead and finish the chunk behind.
// 1.5B, one sequence, whole calls against the three launches: 5 tokens 1.98 -> 1.91 ms, 40 2.74 -> 2.66, 64 2.97 -> 2.95.
#include "rwkvq_tmix_seq.cuh"

#include "rwkvq_decode_parts.cuh"

namespace rwkvq {

constexpr int kTsChunk = 16;                 // tokens whose operands are in shared memory together
constexpr int kTsThreads = 256, kTsSteppers = 128;

struct TsOps { float r[kTsChunk][64], w[kTsChunk][64], k[kTsChunk][64], v[kTsChunk][64], a[kTsChunk][64], b[kTsChunk][64], g[kTsChunk][64]; };
struct TsSmem {
    TsOps op[2];
    float y[2][kTsChunk][64];
    float red[2][2][kTsChunk / 2];
};

// all warps of both roles
__device__ __forceinline__ void ts_sync() { asm volatile("bar.sync 4, %0;" ::"n"(kTsThreads) : "memory"); }

__global__ void __launch_bounds__(kTsThreads, 2) tmix_seq_kernel(const TmixSeqArgs p) {
    extern __shared__ __align__(16) unsigned char ts_smem[];
    TsSmem& s = *reinterpret_cast<TsSmem*>(ts_smem);
    const int hd = blockIdx.x % p.H, b = blockIdx.x / p.H, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const size_t D = static_cast<size_t>(p.H) * 64, row0 = static_cast<size_t>(b) * p.T * D + hd * 64;
    const int n_chunks = (p.T + kTsChunk - 1) / kTsChunk;
    pdl_launch_dependents();
    // tail: a warp per token, channels lane and lane + 32
    const int t0c = hd * 64 + lane;
    const float rk0 = __ldg(p.r_k + t0c), rk1 = __ldg(p.r_k + t0c + 32), lw0 = __ldg(p.ln_w + t0c), lw1 = __ldg(p.ln_w + t0c + 32),
                lb0 = __ldg(p.ln_b + t0c), lb1 = __ldg(p.ln_b + t0c + 32);
    auto finish = [&](int ch, int first, int step) {                    // group norm over the head (two-pass), bonus, gate
        const TsOps& o = s.op[ch & 1];
        const int n = min(kTsChunk, p.T - ch * kTsChunk);
        for (int t = first; t < n; t += step) {
            const float x0 = s.y[ch & 1][t][lane], x1 = s.y[ch & 1][t][lane + 32];
            float sum = x0 + x1, dp = o.r[t][lane] * o.k[t][lane] * rk0 + o.r[t][lane + 32] * o.k[t][lane + 32] * rk1;
#pragma unroll
            for (int i = 16; i > 0; i >>= 1) {
                sum += __shfl_xor_sync(0xFFFFFFFFu, sum, i);
                dp += __shfl_xor_sync(0xFFFFFFFFu, dp, i);
            }
            const float mean = sum / 64.f, d0 = x0 - mean, d1 = x1 - mean;
            float var = d0 * d0 + d1 * d1;
#pragma unroll
            for (int i = 16; i > 0; i >>= 1) var += __shfl_xor_sync(0xFFFFFFFFu, var, i);
            const float inv = 1.0f / sqrtf(var / 64.f + 64e-5f);
            const float o0 = (d0 * inv * lw0 + lb0 + dp * o.v[t][lane]) * o.g[t][lane];
            const float o1 = (d1 * inv * lw1 + lb1 + dp * o.v[t][lane + 32]) * o.g[t][lane + 32];
            float* out = p.og + row0 + static_cast<size_t>(ch * kTsChunk + t) * D + lane;
            out[0] = o0;
            out[32] = o1;
            if (p.og_amax != nullptr) {              // |o| as int bits orders like the float, a NaN above every number
                const int m = __reduce_max_sync(0xFFFFFFFFu, max(__float_as_int(fabsf(o0)), __float_as_int(fabsf(o1))));
                if (lane == 0) atomicMax(reinterpret_cast<int*>(p.og_amax) + static_cast<size_t>(b) * p.T + ch * kTsChunk + t, m);
            }
        }
    };
    if (tid < kTsSteppers) {
        // ------------------------------------------------------------------ steps: 4 state rows x 8 columns a thread
        const int c = tid & 7, dv0 = (tid >> 3) * 4;
        const size_t hbase = (static_cast<size_t>(blockIdx.x) * 64 + dv0) * 64;
        float2 h[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {                // written before the first kernel of this pass started
            if (p.h_in) cols8(p.h_in + hbase + j * 64, c, h[j]);
            else h[j][0] = h[j][1] = h[j][2] = h[j][3] = make_float2(0.f, 0.f);
        }
        pdl_wait();                                  // what this kernel stores may be read by the kernels before it
        ts_sync();
        for (int ch = 0; ch < n_chunks; ++ch) {
            const TsOps& o = s.op[ch & 1];
            const int n = min(kTsChunk, p.T - ch * kTsChunk);
#pragma unroll 2
            for (int t = 0; t < n; ++t) {
                float2 x[4];
                float sa[4], y[4];
                cols8(o.a[t], c, x);
#pragma unroll
                for (int j = 0; j < 4; ++j) sa[j] = dot8(h[j], x);
                const float4 v4 = *reinterpret_cast<const float4*>(&o.v[t][dv0]);
                const float v[4] = {v4.x, v4.y, v4.z, v4.w};
                {
                    float2 w[4], k[4];               // decay and v k^T while the sums cross the lanes
                    cols8(o.w[t], c, w);
                    cols8(o.k[t], c, k);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float2 vj = make_float2(v[j], v[j]);
#pragma unroll
                        for (int q = 0; q < 4; ++q) h[j][q] = __ffma2_rn(w[q], h[j][q], __fmul2_rn(vj, k[q]));
                    }
                }
#pragma unroll
                for (int m = 1; m < 8; m <<= 1)
#pragma unroll
                    for (int j = 0; j < 4; ++j) sa[j] += __shfl_xor_sync(0xFFFFFFFFu, sa[j], m);
                cols8(o.b[t], c, x);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 s2 = make_float2(sa[j], sa[j]);
#pragma unroll
                    for (int q = 0; q < 4; ++q) h[j][q] = __ffma2_rn(s2, x[q], h[j][q]);
                }
                cols8(o.r[t], c, x);
#pragma unroll
                for (int j = 0; j < 4; ++j) y[j] = dot8(h[j], x);
                // four sums over eight lanes, halving the values: lane bits 0 and 1 pick the row
                const float k0 = (c & 1) ? y[2] : y[0], k1 = (c & 1) ? y[3] : y[1], g0 = (c & 1) ? y[0] : y[2], g1 = (c & 1) ? y[1] : y[3];
                const float u0 = k0 + __shfl_xor_sync(0xFFFFFFFFu, g0, 1), u1 = k1 + __shfl_xor_sync(0xFFFFFFFFu, g1, 1);
                float z = ((c & 2) ? u1 : u0) + __shfl_xor_sync(0xFFFFFFFFu, (c & 2) ? u0 : u1, 2);
                z += __shfl_xor_sync(0xFFFFFFFFu, z, 4);
                if (c < 4) s.y[ch & 1][t][dv0 + (c & 1) * 2 + (c >> 1)] = z;
            }
            ts_sync();
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float* o = p.h_out + hbase + j * 64;
            *reinterpret_cast<float4*>(o + 4 * c) = make_float4(h[j][0].x, h[j][0].y, h[j][1].x, h[j][1].y);
            *reinterpret_cast<float4*>(o + 32 + 4 * c) = make_float4(h[j][2].x, h[j][2].y, h[j][3].x, h[j][3].y);
        }
    } else {
        // ------------------------------------------------------------------ rows: 64 threads a token, a channel each
        const int grp = (tid - kTsSteppers) >> 6, c = tid & 63, cc = hd * 64 + c;
        const float w0 = __ldg(p.w0 + cc), a0 = __ldg(p.a0 + cc), kkw = __ldg(p.k_k + cc), kaw = __ldg(p.k_a + cc);
        const float v0 = p.yv ? __ldg(p.v0 + cc) : 0.f;
        constexpr int U = kTsChunk / 2;
        float r[U], k[U], v[U], yw[U], ya[U], yv[U], vf[U], g[U];
        auto load = [&](int ch) {
            const int n = min(kTsChunk, p.T - ch * kTsChunk);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const bool in = grp + 2 * u < n;
                const size_t at = row0 + static_cast<size_t>(ch * kTsChunk + (in ? grp + 2 * u : 0)) * D + c;
                r[u] = in ? __ldcg(p.r + at) : 0.f;
                k[u] = in ? __ldcg(p.k + at) : 0.f;
                v[u] = in ? __ldcg(p.v + at) : 0.f;
                yw[u] = in ? __ldcg(p.yw + at) : 0.f;
                ya[u] = in ? __ldcg(p.ya + at) : 0.f;
                g[u] = in ? __ldcg(p.g + at) : 0.f;
                yv[u] = in && p.yv ? __ldcg(p.yv + at) : 0.f;
                vf[u] = in && p.yv ? __ldcg(p.v_first + at) : 0.f;
            }
        };
        auto operands = [&](int ch) {
            TsOps& o = s.op[ch & 1];
            const int n = min(kTsChunk, p.T - ch * kTsChunk);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int t = grp + 2 * u;
                if (t >= n) break;                                       // the 64 threads of a group together
                float q = k[u] * kkw;
                q *= q;
#pragma unroll
                for (int i = 16; i > 0; i >>= 1) q += __shfl_xor_sync(0xFFFFFFFFu, q, i);
                if (lane == 0) s.red[grp][warp & 1][u] = q;
                ya[u] = sigmoidf_(ya[u] + a0);
                o.w[t][c] = expf(-0.606531f * sigmoidf_(yw[u] + w0));
                o.k[t][c] = k[u] * (1.0f + (ya[u] - 1.0f) * kaw);
                o.r[t][c] = r[u];
                o.v[t][c] = p.yv ? v[u] + (vf[u] - v[u]) * sigmoidf_(yv[u] + v0) : v[u];
                o.g[t][c] = g[u];
            }
            asm volatile("bar.sync %0, 64;" ::"r"(1 + grp) : "memory");
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int t = grp + 2 * u;
                if (t >= n) break;
                const float kn = k[u] * kkw * (1.0f / sqrtf(s.red[grp][0][u] + s.red[grp][1][u] + 1e-12f));
                o.a[t][c] = -kn;
                o.b[t][c] = kn * ya[u];
            }
        };
        pdl_wait();
        load(0);
        operands(0);
        ts_sync();
        for (int ch = 0; ch < n_chunks; ++ch) {
            if (ch + 1 < n_chunks) load(ch + 1);
            if (ch > 0) finish(ch - 1, warp - 4, 4);
            asm volatile("bar.sync 3, %0;" ::"n"(kTsThreads - kTsSteppers) : "memory");      // chunk ch - 1 has been finished: its buffer is free
            if (ch + 1 < n_chunks) operands(ch + 1);
            ts_sync();
        }
    }
    finish(n_chunks - 1, warp, kTsThreads / 32);
}

int launch_tmix_seq(const TmixSeqArgs& p, cudaStream_t s) {
    const long long pairs = static_cast<long long>(p.B) * p.H;
    RWKVQ_REQUIRE(pairs < (1ll << 31) && p.T >= 1, RWKVQ_E_LIMIT, "tmix_seq: %lld heads, %d tokens", pairs, p.T);
    RWKVQ_REQUIRE(aligned(p.h_in, 16) && aligned(p.h_out, 16), RWKVQ_E_ALIGN, "tmix_seq: states on 16-byte boundaries");
    cudaError_t e = cudaFuncSetAttribute(tmix_seq_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sizeof(TsSmem)));
    if (e != cudaSuccess) return fail(RWKVQ_E_LIMIT, "tmix_seq: %zu bytes of shared memory: %s", sizeof(TsSmem), cudaGetErrorString(e));
    e = launch_pdl(tmix_seq_kernel, dim3(static_cast<unsigned>(pairs)), dim3(kTsThreads), sizeof(TsSmem), s, p);
    if (e != cudaSuccess) return fail(RWKVQ_E_LAUNCH, "tmix_seq: %s", cudaGetErrorString(e));
    return RWKVQ_OK;
}

}  // namespace rwkvq
