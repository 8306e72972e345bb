// Tensor-core GEMM of the many-row linears (prefill, long verify runs, LoRA branches of long calls):
//
//     y[tok, row] = sum_k W[row, k] x[tok, k]
//
// with both operands as fp16 matrices in L2 / HBM.  Packed weights become such a matrix in a pass of
// their own (dequant_f16_kernel, into caller scratch small enough to stay in L2): converting inside the
// GEMM costs 512 threads per SM about 4 us per 128 columns, several times the tensor time, and every
// token tile converts again, while the separate pass runs at memory speed (16.8 M weights: 10 us) and
// leaves a GEMM that only TMA and tcgen05 touch.
//
// Two kernels share the layout (K-major tiles of 64 fp16 columns, 128-byte swizzle, weights as the UMMA M):
//   gemm_pair_kernel  a pair of CTAs (cta_group::2) per 256 x 256 tile, persistent, accumulators
//                     double-buffered in tensor memory so that the epilogue of one tile runs beside the
//                     MMAs of the next.  Each CTA stages half of the rows and half of the tokens, i.e. 64 B
//                     of shared-memory reads per MMA cycle instead of 96: for problems that fill the chip.
//   gemm_one_kernel   one CTA per 128 x {64, 128} tile, K split over a cluster of 1 / 2 / 4 / 8 CTAs and reduced in
//                     distributed shared memory in rank order: for problems with few tiles, where the time
//                     is the length of one CTA's K loop.
// Every mbarrier wait is bounded; on expiry the status word is set, all roles run to the common end, and
// tensor memory is freed.
#include "rwkvq_gemm_f16.cuh"
#include "rwkvq_gemm_sb.cuh"

#include <cooperative_groups.h>

#include <algorithm>

#include "rwkvq_decode_parts.cuh"
#include "rwkvq_tc.cuh"

namespace cg = cooperative_groups;

namespace rwkvq {

// ------------------------------------------------------------------ packed weights -> fp16
// A warp converts 32 consecutive items of 32 weights: coalesced 16-byte reads of the codes, and the 2 KB
// of results turned in shared memory so that every store instruction covers 512 contiguous bytes.
// Bound: L2 / HBM writes.
__global__ void __launch_bounds__(256) dequant_f16_kernel(const QView t, int row0, long long n_items, __half* __restrict__ out,
                                                          float* __restrict__ n2) {
    __shared__ __align__(16) uint4 turn[8][128];
    __shared__ int s_n2[128];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ipr = t.cols >> 5, nsb = t.cols >> 8;
    pdl_launch_dependents();
    if (n2 != nullptr) {
        for (int i = threadIdx.x; i < nsb; i += 256) s_n2[i] = 0;
        __syncthreads();
    }
    bool waited = false;
    for (long long base = (static_cast<long long>(blockIdx.x) * 8 + warp) * 32; base < n_items; base += static_cast<long long>(gridDim.x) * 256) {
        const long long item = base + lane < n_items ? base + lane : n_items - 1;
        const int row = static_cast<int>(item / ipr), it = static_cast<int>(item - static_cast<long long>(row) * ipr);
        Packed p;
        load_packed(p, t, row0 + row, it >> 3, it & 7);
        ItemCodes c;
        decode_item(p, t, it & 7, it & 1, c);
        float ss = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint2 a = bytes_to_half4(c.bytes[2 * j], c.bias, c.s2[j >> 1], c.m2[j >> 1]);
            const uint2 b = bytes_to_half4(c.bytes[2 * j + 1], c.bias, c.s2[j >> 1], c.m2[j >> 1]);
            turn[warp][(4 * lane + j) ^ ((lane >> 1) & 7)] = make_uint4(a.x, a.y, b.x, b.y);
            if (n2 != nullptr) {
                const uint32_t w[4] = {a.x, a.y, b.x, b.y};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[e]));
                    ss = fmaf(f.x, f.x, fmaf(f.y, f.y, ss));
                }
            }
        }
        if (n2 != nullptr) {                 // 8 lanes hold one row's 256 columns (items per row are a multiple of 8)
            ss += __shfl_xor_sync(0xFFFFFFFFu, ss, 1);
            ss += __shfl_xor_sync(0xFFFFFFFFu, ss, 2);
            ss += __shfl_xor_sync(0xFFFFFFFFu, ss, 4);
            if ((lane & 7) == 0) atomicMax(&s_n2[it >> 3], __float_as_int(ss));
        }
        __syncwarp();
        if (!waited) { pdl_wait(); waited = true; }      // the scratch may still be read by the kernel before this one
        uint4* o = reinterpret_cast<uint4*>(out) + base * 4;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int ch = 32 * j + lane;
            if (base + (ch >> 2) < n_items) o[ch] = turn[warp][ch ^ ((ch >> 3) & 7)];
        }
        __syncwarp();
    }
    if (n2 != nullptr) {
        __syncthreads();
        pdl_wait();
        for (int i = threadIdx.x; i < nsb; i += 256) atomicMax(reinterpret_cast<int*>(n2) + i, s_n2[i]);
    }
}

int launch_dequant_f16(const rwkvq_qtensor& t, int row0, int rows, __half* out, float* n2, cudaStream_t s, int per_sm) {
    RWKVQ_REQUIRE((t.kind == RWKVQ_KIND_SB6 || t.kind == RWKVQ_KIND_SYM) && t.cols % 256 == 0 && (n2 == nullptr || t.cols <= 32768), RWKVQ_E_DTYPE,
                  "dequant_f16: sb6 / sym tensors (with norms of at most 32768 columns)");
    const long long items = static_cast<long long>(rows) * (t.cols >> 5);
    const long long want = (items + 255) / 256;
    // beside another kernel: room for its CTAs on every SM, and no launch before the one in front has ended (four conversions
    // at once held the threads of every SM, and the scan's operands waited 30 us for them)
    const int most = 148 * (per_sm > 0 ? per_sm : 6);
    const dim3 grid(static_cast<unsigned>(want < most ? want : most));
    if (per_sm > 0) {
        dequant_f16_kernel<<<grid, 256, 0, s>>>(make_view(t), row0, items, out, n2);
        return check_launch("dequant_f16");
    }
    cudaError_t e = launch_pdl(dequant_f16_kernel, grid, dim3(256), 0, s, make_view(t), row0, items, out, n2);
    if (e != cudaSuccess) return fail(RWKVQ_E_LAUNCH, "dequant_f16: %s", cudaGetErrorString(e));
    return RWKVQ_OK;
}

// ---- LoRA matrices, stored [in, out]: tiles of 64 x 64, turned in shared memory
struct TransposeArgs {
    QView t[8];
    __half* out[8];
};
template <int MODE>
__device__ __forceinline__ void transpose_tile(const QView& t, int i0, int c0, __half (&tile)[64][72]) {
    const int nb = MODE == 0 ? (t.cols + t.gs - 1) / t.gs : 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int id = threadIdx.x + 256 * u, i = id >> 4, c = (id & 15) * 4;
        float w[4] = {0.f, 0.f, 0.f, 0.f};
        if (i0 + i < t.rows && c0 + c < t.cols) lora_w4<MODE>(t, i0 + i, c0 + c, nb, MODE == 0 ? (c0 + c) / t.gs : 0, w);
#pragma unroll
        for (int k = 0; k < 4; ++k) tile[c + k][i] = __float2half_rn(w[k]);
    }
}
__global__ void __launch_bounds__(256) dequant_f16_t_kernel(const TransposeArgs a) {
    __shared__ __align__(16) __half tile[64][72];
    const QView& t = a.t[blockIdx.y];
    const int in_tiles = (t.rows + 63) >> 6, out_tiles = (t.cols + 63) >> 6;
    pdl_launch_dependents();
    if (static_cast<int>(blockIdx.x) >= in_tiles * out_tiles) return;
    const int i0 = (blockIdx.x % in_tiles) * 64, c0 = (blockIdx.x / in_tiles) * 64;
    switch (lora_mode(t)) {
        case 0: transpose_tile<0>(t, i0, c0, tile); break;
        case 1: transpose_tile<1>(t, i0, c0, tile); break;
        default: transpose_tile<2>(t, i0, c0, tile); break;
    }
    __syncthreads();
    pdl_wait();
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int id = threadIdx.x + 256 * u, c = id >> 3, ch = id & 7;
        if (c0 + c < t.cols)
            *reinterpret_cast<uint4*>(a.out[blockIdx.y] + static_cast<size_t>(c0 + c) * (in_tiles * 64) + i0 + ch * 8) =
                *reinterpret_cast<const uint4*>(&tile[c][ch * 8]);
    }
}
int launch_dequant_f16_t(const TransposeJob* jobs, int n, cudaStream_t s) {
    TransposeArgs a{};
    int most = 0;
    for (int i = 0; i < n; ++i) {
        a.t[i] = make_view(*jobs[i].t);
        a.out[i] = jobs[i].out;
        const int tiles = ((jobs[i].t->rows + 63) / 64) * ((jobs[i].t->cols + 63) / 64);
        most = tiles > most ? tiles : most;
    }
    cudaError_t e = launch_pdl(dequant_f16_t_kernel, dim3(most, n), dim3(256), 0, s, a);
    if (e != cudaSuccess) return fail(RWKVQ_E_LAUNCH, "dequant_f16_t: %s", cudaGetErrorString(e));
    return RWKVQ_OK;
}

// ------------------------------------------------------------------ GEMM
struct HgDev {                     // a problem as the kernels see it
    int rows, k_stages, a_stages;  // stages of 64 columns: of the whole sum, and after which W's column wraps (two terms)
    int row_tiles, first_tile;
    int out, epilogue, act, lo_off, n_w_n2;
    const float *row_scale, *resid, *w_n2, *x_n2;
    float *y32, *out_scale;
    __half* y16;
    long long ldy;
};
struct HgArgs {
    HgDev p[kHgMaxProbs];
    int n_probs, n_tiles, tok_tiles, M;
    int* status;
};
struct HgMaps { CUtensorMap w[kHgMaxProbs], x[kHgMaxProbs]; };

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
          "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// bound of the squared norm of any row of W (fp16 hidden rows only)
__device__ __forceinline__ float warp_w_n2(const HgDev& p, int lane) {
    float w2 = 0.f;
    if (p.out == HG_RELU2_F16) {
        for (int i = lane; i < p.n_w_n2; i += 32) w2 += __ldcg(p.w_n2 + i);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) w2 += __shfl_xor_sync(0xFFFFFFFFu, w2, o);
    }
    return w2;
}
// Power of two that brings relu(y)^2 of a token below 2^14 whatever row of W meets it (Cauchy-Schwarz);
// rows without a finite bound keep 1 and propagate.
__device__ __forceinline__ float relu2_scale(float w2, float x_n2) {
    const float b2 = w2 * x_n2;                          // bound of y^2
    int e = 0;
    if (!(b2 > 0.f && b2 < INFINITY)) return 1.f;
    frexpf(b2, &e);                                      // b2 < 2^e; rounding of the sums stays within the headroom to 65504
    return ldexpf(1.f, max(-100, min(100, 14 - e)));
}

// Per-token factors of N blocks of 32 tokens `step` apart, one token per lane and block: what the accumulator is multiplied
// with, and (fp16 output) the scale of the stored value.
template <int N>
__device__ __forceinline__ void token_factors(const HgDev& p, int tok, int step, int M, int lane, float (&un)[N], float (&so)[N]) {
    float rs[N], n2[N];
    const float w2 = warp_w_n2(p, lane);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const int t = tok + i * step;
        rs[i] = t < M && p.row_scale != nullptr ? __ldcg(p.row_scale + t) : 1.f;
        n2[i] = t < M && p.out == HG_RELU2_F16 ? __ldcg(p.x_n2 + t) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        un[i] = 1.0f / rs[i];                            // exact: powers of two
        so[i] = relu2_scale(w2, n2[i]);
    }
}

__device__ __forceinline__ float lora_act(float v, int act) {
    if (act == 1) return tanhf(v);
    if (act == 2) return sigmoidf_(v);
    return v;
}

// NB tokens of one output row held by this lane (the 32 lanes hold 32 consecutive rows, so every store
// of a token covers one 128-byte line); lane j of un / so carries token j's factors.  The problem is held
// by value and each output form has its own loop over a moving pointer: with the descriptor read through
// a reference every store forced a reload of it, and a block of 32 took 4 us instead of 0.4.
template <int NB>
__device__ __forceinline__ void finish_block(const HgDev& p, float (&v)[NB], float un, float so, int tok0, int row, int M) {
    const int n = row < p.rows ? min(NB, M - tok0) : 0;
#pragma unroll
    for (int j = 0; j < NB; ++j) v[j] *= __shfl_sync(0xFFFFFFFFu, un, j);
    const long long at = static_cast<long long>(tok0) * p.ldy + row, step = p.ldy;
    if (p.out == HG_F32) {
        float* y = p.y32 + at;
        if (p.epilogue == RWKVQ_EPI_ADD) {
            const float* rs = p.resid + at;
            float r[NB];
#pragma unroll
            for (int j = 0; j < NB; ++j) {
                r[j] = j < n ? __ldcg(rs) : 0.f;
                rs += step;
            }
#pragma unroll
            for (int j = 0; j < NB; ++j) v[j] = __fadd_rn(v[j], r[j]);
        } else if (p.epilogue == RWKVQ_EPI_RELU2) {
#pragma unroll
            for (int j = 0; j < NB; ++j) { v[j] = fmaxf(v[j], 0.f); v[j] *= v[j]; }
        }
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            if (j < n) *y = v[j];
            y += step;
        }
    } else if (p.out == HG_RELU2_F16) {
        __half* y = p.y16 + at;
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            const float x = fmaxf(v[j], 0.f), sj = __shfl_sync(0xFFFFFFFFu, so, j);
            if (j < n) *y = __float2half_rn(x * x * sj);
            y += step;
        }
    } else {
        __half* y = p.y16 + at;
        const int lo = p.lo_off;
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            const float x = lora_act(v[j], p.act);
            const __half hi = __float2half_rn(x);
            if (j < n) { y[0] = hi; y[lo] = __float2half_rn(x - __half2float(hi)); }
            y += step;
        }
    }
}

// by value: see finish_block
__device__ __forceinline__ HgDev problem_of(const HgArgs& a, int tile, int& pi) {
    pi = 0;
    while (pi + 1 < a.n_probs && tile >= a.p[pi + 1].first_tile) ++pi;
    return a.p[pi];
}

// ---- cluster / cta_group::2 wrappers
__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_alloc2(uint32_t* dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(dst_smem)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc2(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrives on the barrier at this offset in both CTAs of the pair once all MMAs issued so far have completed
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_addr(bar)),
        "h"(static_cast<uint16_t>(3))
        : "memory");
}
// 2-D tile into this CTA's shared memory; its bytes count on `bar`, a shared::cluster address (the pair's first CTA)
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_addr(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}

constexpr int kHgABytes = kGmRows * 128;                 // one CTA's weight tile of a stage: 128 rows x 64 columns
constexpr int kHgThreads = 256;
constexpr int kPairStages = 6, kPairTok = 256, kPairEpiWarps = 8, kPairThreads = 128 + 32 * kPairEpiWarps;
constexpr int kPairBBytes = (kPairTok / 2) * 128;
constexpr size_t kPairSmem = static_cast<size_t>(kPairStages) * (kHgABytes + kPairBBytes) + 1024;

// Warp 0: TMA (both CTAs, own halves).  Warp 1 of the first CTA: MMAs for the pair.  Warps 4-11: epilogue
// of the CTA's 128 rows, two warps a quadrant of them with half the tokens each.  Four warps that fetched the factors of
// each block of tokens behind its accumulators (up to four L2 round trips in a row) took longer for a tile than its products:
// 4 x 1024 tokens 23.1 -> 22.5 ms (1.5B) and 48.7 -> 47.0 (2.9B).  (The single-CTA tiles, several to an SM's turn, lose 1 to 2 %
// with their factors fetched ahead.)  A block's code, 32 tokens of three epilogues, stands once: four copies of it are fetched by
// every launch, which costs a launch of one tile a CTA 3 to 7 us (2.9B 4 x 33 tokens 7.20 -> 6.96 ms, 3 x 77 7.63 -> 7.13, 1.5B
// 1 x 512 6.37 -> 6.12, 4 x 1024 22.5 -> 21.9).  192 KB of operands in flight per SM cover the L2 latency; the 256-token tile makes a
// stage 512 tensor cycles.
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
    gemm_pair_kernel(const __grid_constant__ HgArgs a, const __grid_constant__ HgMaps maps) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ uint64_t bar_full[kPairStages], bar_empty[kPairStages], bar_tfull[2], bar_tempty[2];
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_fail;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_rank();
    const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    constexpr int STAGE = kHgABytes + kPairBBytes;

    if (tid == 0) {
        for (int s = 0; s < kPairStages; ++s) { mbar_init(&bar_full[s], 1); mbar_init(&bar_empty[s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&bar_tfull[s], 1); mbar_init(&bar_tempty[s], 2 * kPairEpiWarps); }
        s_fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) tmem_alloc2(&s_tmem, 512);
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                                  // the peer's barriers exist before anything signals them
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    pdl_wait();

    if (warp == 0) {
        if (lane == 0) {
            int st = 0, ph = 0;
            bool ok = true;
            for (int tile = pair; tile < a.n_tiles && ok; tile += n_pairs) {
                int pi;
                const HgDev p = problem_of(a, tile, pi);
                const int lt = tile - p.first_tile, rt = lt % p.row_tiles, tt = lt / p.row_tiles;
                const int row0 = rt * 256 + rank * 128, tok0 = tt * kPairTok + rank * (kPairTok / 2);
                int ka = 0;
                for (int k = 0; k < p.k_stages; ++k) {
                    if (!mbar_wait_bounded(&bar_empty[st], ph ^ 1)) { ok = false; break; }
                    unsigned char* sa = smem + st * STAGE;
                    const uint32_t full = mapa(smem_addr(&bar_full[st]), 0);
                    if (rank == 0) mbar_expect_tx(&bar_full[st], 2 * STAGE);
                    tma_load_2d_pair(sa, &maps.w[pi], ka * kGmK, row0, full);
                    tma_load_2d_pair(sa + kHgABytes, &maps.x[pi], k * kGmK, tok0, full);
                    if (++ka == p.a_stages) ka = 0;
                    if (++st == kPairStages) { st = 0; ph ^= 1; }
                }
            }
            pdl_launch_dependents();                     // all loads are on their way
            // the last stages' releases have to land before this CTA may go
            for (int i = 0; i < kPairStages && ok; ++i) {
                ok = mbar_wait_bounded(&bar_empty[st], ph ^ 1);
                if (++st == kPairStages) { st = 0; ph ^= 1; }
            }
            if (!ok) s_fail = 1;
        }
    } else if (warp == 1) {
        if (rank == 0 && lane == 0) {
            const uint32_t idesc = (1u << 4) | (static_cast<uint32_t>(kPairTok >> 3) << 17) | (static_cast<uint32_t>(256 >> 4) << 24);
            const uint64_t desc0 = umma_desc(smem_addr(smem));
            int st = 0, ph = 0, acc = 0, aph = 0;
            bool ok = true;
            for (int tile = pair; tile < a.n_tiles && ok; tile += n_pairs) {
                int pi;
                const HgDev p = problem_of(a, tile, pi);
                if (!mbar_wait_bounded(&bar_tempty[acc], aph ^ 1)) { ok = false; break; }
                tc_fence_after();
                for (int k = 0; k < p.k_stages; ++k) {
                    if (!mbar_wait_bounded(&bar_full[st], ph)) { ok = false; break; }
                    tc_fence_after();
                    const uint64_t ad = desc0 + (static_cast<uint64_t>(st * STAGE) >> 4), bd = ad + (kHgABytes >> 4);
#pragma unroll
                    for (int kk = 0; kk < kGmK / 16; ++kk) umma_f16_pair(tmem + acc * kPairTok, ad + 2 * kk, bd + 2 * kk, idesc, (k | kk) ? 1u : 0u);
                    umma_commit_pair(&bar_empty[st]);
                    if (++st == kPairStages) { st = 0; ph ^= 1; }
                }
                if (ok) umma_commit_pair(&bar_tfull[acc]);
                if (++acc == 2) { acc = 0; aph ^= 1; }
            }
            if (!ok) s_fail = 1;
        }
    } else if (warp >= 4) {
        int acc = 0, aph = 0;
        constexpr int TOKS = kPairTok / (kPairEpiWarps / 4), BLOCKS = TOKS / 32;
        const int q = warp & 3, share = ((warp - 4) >> 2) * TOKS;
        for (int tile = pair; tile < a.n_tiles; tile += n_pairs) {
            int pi;
            const HgDev p = problem_of(a, tile, pi);
            const int lt = tile - p.first_tile, rt = lt % p.row_tiles, tt = lt / p.row_tiles;
            const int row = rt * 256 + rank * 128 + q * 32 + lane, tok0 = tt * kPairTok + share;
            float un[BLOCKS], so[BLOCKS];
            token_factors<BLOCKS>(p, tok0 + lane, 32, a.M, lane, un, so);
            if (p.out == HG_RELU2_F16 && rt == 0 && rank == 0 && q == 0) {
#pragma unroll
                for (int i = 0; i < BLOCKS; ++i)
                    if (tok0 + 32 * i + lane < a.M) p.out_scale[tok0 + 32 * i + lane] = so[i];
            }
            int got = 1;
            if (lane == 0) got = mbar_wait_bounded(&bar_tfull[acc], aph) ? 1 : 0;
            got = __shfl_sync(0xFFFFFFFFu, got, 0);
            if (!got) { s_fail = 1; break; }
            tc_fence_after();
            const uint32_t base = tmem + acc * kPairTok + share + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll 1
            for (int i = 0; i < BLOCKS; ++i) {
                float v[32], u = un[0], s = so[0];       // a select each: one copy of the block's code
#pragma unroll
                for (int k = 1; k < BLOCKS; ++k) { u = i == k ? un[k] : u; s = i == k ? so[k] : s; }
                tmem_ld32(base + 32 * i, v);
                if (i == BLOCKS - 1) {                   // the accumulator is in registers: the MMA warp may overwrite it
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(mapa(smem_addr(&bar_tempty[acc]), 0));
                }
                if (tok0 + 32 * i < a.M) finish_block<32>(p, v, u, s, tok0 + 32 * i, row, a.M);
            }
            if (++acc == 2) { acc = 0; aph ^= 1; }
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (tid == 0 && s_fail) atomicCAS(a.status, 0, RWKVQ_E_TIMEOUT);
    cluster_sync_all();                                  // neither CTA leaves while the other still signals or multiplies
    tc_fence_after();
    if (warp == 2) tmem_dealloc2(tmem, 512);
}

// One tile of 128 rows x NT tokens per cluster; the CTA of rank z sums stages [z K / ks, (z + 1) K / ks).
template <int NT>
struct OneGeo {
    static constexpr int BBYTES = NT * 128, STAGE = kHgABytes + BBYTES, STAGES = NT >= 128 ? 6 : 8;
    static constexpr int PITCH = kGmRows + 4;            // partial tile in shared memory: [NT][PITCH] floats over the dead stages
    static constexpr size_t SMEM = static_cast<size_t>(STAGES) * STAGE + 1024;
    static_assert(static_cast<size_t>(NT) * PITCH * 4 <= static_cast<size_t>(STAGES) * STAGE, "partial tile");
};

// The CTA of cluster rank z finishes tokens [z, z + 1) NT / ks of the tile, each half of the block NB of them:
// adds the ranks' partial sums in rank order, all remote loads of a rank in flight together.
template <int NB>
__device__ __forceinline__ void reduce_share(const HgDev& p, cg::cluster_group& cluster, float* part, int pitch, int ks, int z, int half,
                                             int rl, int row0, int tok0, int rt, int M, bool good) {
    const int tl = (2 * z + half) * NB, tok = tok0 + tl, lane = threadIdx.x & 31;
    float v[NB];
#pragma unroll
    for (int j = 0; j < NB; ++j) v[j] = 0.f;
    for (int u = 0; u < ks; ++u) {
        const float* src = cluster.map_shared_rank(part, u) + tl * pitch + rl;
#pragma unroll
        for (int j = 0; j < NB; ++j) v[j] += src[j * pitch];
    }
    float un[1], so[1];
    token_factors<1>(p, tok + lane, 0, lane < NB ? M : 0, lane, un, so);
    if (p.out == HG_RELU2_F16 && rt == 0 && rl < 32 && lane < NB && tok + lane < M) p.out_scale[tok + lane] = so[0];
    if (good) finish_block<NB>(p, v, un[0], so[0], tok, row0 + rl, M);
}

template <int NT>
__global__ void __launch_bounds__(kHgThreads, 1) gemm_one_kernel(const __grid_constant__ HgArgs a, const __grid_constant__ HgMaps maps) {
    using G = OneGeo<NT>;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ uint64_t bar_full[G::STAGES], bar_empty[G::STAGES], bar_done;
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_fail;
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ks = gridDim.x, z = blockIdx.x, tile = blockIdx.y;     // the cluster spans grid.x
    int pi;
    const HgDev p = problem_of(a, tile, pi);
    const int lt = tile - p.first_tile, rt = lt % p.row_tiles, tt = lt / p.row_tiles;
    const int row0 = rt * kGmRows, tok0 = tt * NT;
    const int k0 = static_cast<int>(static_cast<long long>(p.k_stages) * z / ks);
    const int k1 = static_cast<int>(static_cast<long long>(p.k_stages) * (z + 1) / ks);
    constexpr uint32_t COLS = NT < 32 ? 32 : NT;

    if (tid == 0) {
        for (int s = 0; s < G::STAGES; ++s) { mbar_init(&bar_full[s], 1); mbar_init(&bar_empty[s], 1); }
        mbar_init(&bar_done, 1);
        s_fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) tmem_alloc(&s_tmem, COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    pdl_wait();

    if (warp == 0) {
        if (lane == 0) {
            int st = 0, ph = 0, ka = k0 % p.a_stages;
            bool ok = true;
            for (int k = k0; k < k1; ++k) {
                if (!mbar_wait_bounded(&bar_empty[st], ph ^ 1)) { ok = false; break; }
                unsigned char* sa = smem + st * G::STAGE;
                mbar_expect_tx(&bar_full[st], G::STAGE);
                tma_load_2d(sa, &maps.w[pi], ka * kGmK, row0, &bar_full[st]);
                tma_load_2d(sa + kHgABytes, &maps.x[pi], k * kGmK, tok0, &bar_full[st]);
                if (++ka == p.a_stages) ka = 0;
                if (++st == G::STAGES) { st = 0; ph ^= 1; }
            }
            pdl_launch_dependents();
            for (int i = 0; i < G::STAGES && ok; ++i) {          // the last stages' releases have landed
                ok = mbar_wait_bounded(&bar_empty[st], ph ^ 1);
                if (++st == G::STAGES) { st = 0; ph ^= 1; }
            }
            if (!ok) s_fail = 1;
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = umma_idesc(NT);
            const uint64_t desc0 = umma_desc(smem_addr(smem));
            int st = 0, ph = 0;
            bool ok = true;
            for (int k = k0; k < k1; ++k) {
                if (!mbar_wait_bounded(&bar_full[st], ph)) { ok = false; break; }
                tc_fence_after();
                const uint64_t ad = desc0 + (static_cast<uint64_t>(st * G::STAGE) >> 4), bd = ad + (kHgABytes >> 4);
#pragma unroll
                for (int kk = 0; kk < kGmK / 16; ++kk) umma_f16(tmem, ad + 2 * kk, bd + 2 * kk, idesc, (k > k0 || kk) ? 1u : 0u);
                umma_commit(&bar_empty[st]);
                if (++st == G::STAGES) { st = 0; ph ^= 1; }
            }
            if (ok) umma_commit(&bar_done);
            else s_fail = 1;
        }
    }
    __syncwarp();
    if (lane == 0 && !s_fail && !mbar_wait_bounded(&bar_done, 0)) s_fail = 1;
    __syncwarp();
    tc_fence_after();
    __syncthreads();
    const bool good = !s_fail;
    if (!good && tid == 0) atomicCAS(a.status, 0, RWKVQ_E_TIMEOUT);
    const int q = warp & 3, half = warp >> 2, rl = q * 32 + lane;
    const uint32_t base = tmem + (static_cast<uint32_t>(q * 32) << 16);
    if (ks == 1) {
        if (good) {
            for (int c0 = half * 32; c0 < NT; c0 += 64) {
                if (tok0 + c0 >= a.M) break;
                float v[32], un[1], so[1];
                tmem_ld32(base + c0, v);
                token_factors<1>(p, tok0 + c0 + lane, 0, a.M, lane, un, so);
                if (p.out == HG_RELU2_F16 && rt == 0 && q == 0 && tok0 + c0 + lane < a.M) p.out_scale[tok0 + c0 + lane] = so[0];
                finish_block<32>(p, v, un[0], so[0], tok0 + c0, row0 + rl, a.M);
            }
        }
    } else {
        float* part = reinterpret_cast<float*>(smem);    // every MMA that read the stages has completed
        for (int c0 = half * 32; c0 < NT; c0 += 64) {
            float v[32];
            tmem_ld32(base + c0, v);
#pragma unroll
            for (int j = 0; j < 32; ++j) part[(c0 + j) * G::PITCH + rl] = v[j];
        }
        cluster.sync();
        if (ks == 2) reduce_share<NT / 4>(p, cluster, part, G::PITCH, 2, z, half, rl, row0, tok0, rt, a.M, good);
        else if (ks == 4) reduce_share<NT / 8>(p, cluster, part, G::PITCH, 4, z, half, rl, row0, tok0, rt, a.M, good);
        else reduce_share<NT / 16>(p, cluster, part, G::PITCH, 8, z, half, rl, row0, tok0, rt, a.M, good);
        cluster.sync();                                  // nobody leaves while a peer still reads its partial tile
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 2) tmem_dealloc(tmem, COLS);
}

// Pre-pass for fp32 activations, one CTA per token: power-of-two scale with |x * scale| <= 2^14 and the
// scaled row as fp16 (the tensor the TMA loads read).
__global__ void __launch_bounds__(256) row_scale_kernel(const float* __restrict__ x, long long ldx, int cols, float* __restrict__ scale,
                                                        __half* __restrict__ x16, long long pitch, int* __restrict__ status) {
    __shared__ float red[8];
    constexpr int kKeep = 4;                             // float4 per thread held between the two uses (4096 columns)
    pdl_launch_dependents();
    pdl_wait();
    if (status != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *status = 0;      // of the product that follows
    const float4* row = reinterpret_cast<const float4*>(x + blockIdx.x * ldx);
    const int n4 = cols >> 2;
    float4 keep[kKeep];
    float amax = 0.f;
    auto upd = [&](const float4& v) { amax = fmaxf(amax, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)))); };
#pragma unroll
    for (int k = 0; k < kKeep; ++k) {
        const int i = threadIdx.x + 256 * k;
        keep[k] = i < n4 ? __ldcg(row + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int k = 0; k < kKeep; ++k) upd(keep[k]);
    for (int i = threadIdx.x + 256 * kKeep; i < n4; i += 256) upd(__ldcg(row + i));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
    __syncthreads();
    amax = red[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) amax = fmaxf(amax, red[w]);
    int e = 0;
    if (amax > 0.f && amax < INFINITY) frexpf(amax, &e);
    const float sc = ldexpf(1.f, 14 - e);
    if (threadIdx.x == 0) scale[blockIdx.x] = sc;
    uint2* out = reinterpret_cast<uint2*>(x16 + static_cast<size_t>(blockIdx.x) * pitch);
    auto put = [&](int i, const float4& v) {
        const __half2 a = __floats2half2_rn(v.x * sc, v.y * sc), b = __floats2half2_rn(v.z * sc, v.w * sc);
        out[i] = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
    };
#pragma unroll
    for (int k = 0; k < kKeep; ++k)
        if (threadIdx.x + 256 * k < n4) put(threadIdx.x + 256 * k, keep[k]);
    for (int i = threadIdx.x + 256 * kKeep; i < n4; i += 256) put(i, __ldcg(row + i));
}

int launch_row_scale(const float* x, long long ldx, int cols, int M, float* scale, __half* x16, long long pitch, int* status, cudaStream_t s) {
    cudaError_t e = launch_pdl(row_scale_kernel, dim3(M), dim3(256), 0, s, x, ldx, cols, scale, x16, pitch, status);
    if (e != cudaSuccess) return fail(RWKVQ_E_LAUNCH, "row_scale: %s", cudaGetErrorString(e));
    return RWKVQ_OK;
}

namespace {

constexpr int kSms = 148;
int g_gemm_acc_mode = 0;             // rwkvq_profiling_gemm_acc_mode: 0 launcher's choice, 1 single-CTA tiles, 2 CTA pairs

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

// the attribute belongs to the (function, device) pair: remembered per device of this process
template <typename K>
int smem_attr(K kernel, size_t bytes, bool (&configured)[64]) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) dev = 0;
    if (dev >= 64 || !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
        if (e != cudaSuccess) return fail(RWKVQ_E_LIMIT, "gemm_f16: %zu bytes of shared memory: %s", bytes, cudaGetErrorString(e));
        if (dev < 64) configured[dev] = true;
    }
    return RWKVQ_OK;
}

template <int NT>
int launch_one(const HgArgs& a, const HgMaps& maps, int ks, cudaStream_t s) {
    static bool configured[64] = {};
    int rc = smem_attr(gemm_one_kernel<NT>, OneGeo<NT>::SMEM, configured);
    if (rc) return rc;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ks, a.n_tiles);
    cfg.blockDim = dim3(kHgThreads);
    cfg.dynamicSmemBytes = OneGeo<NT>::SMEM;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ks; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_one_kernel<NT>, a, maps);
    if (e != cudaSuccess) return fail(RWKVQ_E_LAUNCH, "gemm_f16: %s", cudaGetErrorString(e));
    return RWKVQ_OK;
}

}  // namespace

// fp16 [rows, cols] row-major; box = [box_rows, 64 columns], 128-byte swizzle, zero fill beyond the edges
int make_half_map(CUtensorMap* map, const __half* base, long long rows, long long cols, long long pitch, int box_rows) {
    EncodeTiledFn enc = encode_tiled();
    RWKVQ_REQUIRE(enc != nullptr, RWKVQ_E_ARCH, "gemm_f16: cuTensorMapEncodeTiled is not available");
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(pitch) * sizeof(__half)};
    const cuuint32_t box[2] = {kGmK, static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half*>(base), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    RWKVQ_REQUIRE(r == CUDA_SUCCESS, RWKVQ_E_LAUNCH, "gemm_f16: cuTensorMapEncodeTiled failed (%d)", static_cast<int>(r));
    return RWKVQ_OK;
}

int make_byte_map(CUtensorMap* map, const void* base, long long rows, long long row_bytes, int box_bytes, int box_rows) {
    EncodeTiledFn enc = encode_tiled();
    RWKVQ_REQUIRE(enc != nullptr, RWKVQ_E_ARCH, "gemm_f16: cuTensorMapEncodeTiled is not available");
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(row_bytes), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(row_bytes)};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(box_bytes), static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t estr[2] = {1, 1};
    const CUtensorMapSwizzle swizzle = box_bytes == 128  ? CU_TENSOR_MAP_SWIZZLE_128B
                                       : box_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B
                                       : box_bytes == 32 ? CU_TENSOR_MAP_SWIZZLE_32B
                                                         : CU_TENSOR_MAP_SWIZZLE_NONE;
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    RWKVQ_REQUIRE(r == CUDA_SUCCESS, RWKVQ_E_LAUNCH, "gemm_sb: cuTensorMapEncodeTiled failed (%d)", static_cast<int>(r));
    return RWKVQ_OK;
}

// Which kernel and tile: the smallest modelled time of the slowest SM in tensor cycles.  A stage of 64
// columns costs four MMAs: 512 cycles for the pair's 256-token tile, 200 / 300 for one CTA's 64- / 128-token
// tile (bound by its shared-memory reads); a launch adds its ramp and the epilogue, a K split the
// cluster barriers and the remote reads.  The pair kernel needs enough tiles for its 74 pairs and loses
// to the small tiles where one wave of those is shorter than its single long tile.
int launch_gemm_f16(const HgProb* probs, int n_probs, int M, int* status, cudaStream_t s) {
    RWKVQ_REQUIRE(n_probs >= 1 && n_probs <= kHgMaxProbs && M >= 1, RWKVQ_E_SHAPE, "gemm_f16: %d problems, M=%d", n_probs, M);
    int k_most = 0, k_least = 1 << 30;
    for (int i = 0; i < n_probs; ++i) {
        const HgProb& p = probs[i];
        RWKVQ_REQUIRE(p.k % kGmK == 0 && p.k > 0 && p.terms >= 1 && p.terms <= 2 && p.rows >= 1, RWKVQ_E_SHAPE, "gemm_f16: rows %d, k %d", p.rows, p.k);
        RWKVQ_REQUIRE(p.w && p.x && aligned(p.w, 16) && aligned(p.x, 16) && p.w_pitch % 8 == 0 && p.x_pitch % 8 == 0, RWKVQ_E_ALIGN,
                      "gemm_f16: operands must be 16-byte aligned");
        const int st = p.k / kGmK * p.terms;
        k_most = st > k_most ? st : k_most;
        k_least = st < k_least ? st : k_least;
    }
    auto tiles_of = [&](int rows_per, int toks_per) {
        long long n = 0;
        for (int i = 0; i < n_probs; ++i) n += static_cast<long long>((probs[i].rows + rows_per - 1) / rows_per) * ((M + toks_per - 1) / toks_per);
        return n;
    };
    const long long pairs = tiles_of(256, kPairTok);
    double best = static_cast<double>((pairs + kSms / 2 - 1) / (kSms / 2)) * (k_most * 530.0) + 5000.0;
    // a few tiles with a long sum always split K: shorter, and shorter chains of accumulator roundings
    const bool pair_ok = g_gemm_acc_mode != 1 && (pairs >= 16 || k_most <= 4096 / kGmK);
    if (!pair_ok) best = 1e300;
    int nt = 0, ks = 1;
    for (int cand = 64; cand <= 128 && !(g_gemm_acc_mode == 2 && pair_ok); cand *= 2) {
        const long long n = tiles_of(kGmRows, cand);
        for (int z = 1; z <= 8; z *= 2) {
            if (z > k_least || n > 65535) break;       // grid.y
            const double waves = static_cast<double>((n * z + kSms - 1) / kSms);
            const double t = waves * ((k_most + z - 1) / z * (cand == 64 ? 200.0 : 300.0) + 2500.0 + (z > 1 ? 2000.0 + 300.0 * z : 0.0)) + 1500.0;
            if (t < best) { best = t; nt = cand; ks = z; }
        }
    }
    HgArgs a{};
    HgMaps maps;
    a.n_probs = n_probs; a.M = M; a.status = status;
    const int rows_per = nt == 0 ? 256 : kGmRows, toks_per = nt == 0 ? kPairTok : nt;
    a.tok_tiles = (M + toks_per - 1) / toks_per;
    for (int i = 0; i < n_probs; ++i) {
        const HgProb& p = probs[i];
        HgDev& d = a.p[i];
        d.rows = p.rows; d.a_stages = p.k / kGmK; d.k_stages = d.a_stages * p.terms;
        d.row_tiles = (p.rows + rows_per - 1) / rows_per;
        d.first_tile = a.n_tiles;
        a.n_tiles += d.row_tiles * a.tok_tiles;
        d.out = p.out; d.epilogue = p.epilogue; d.act = p.act; d.lo_off = p.lo_off; d.n_w_n2 = p.n_w_n2;
        d.row_scale = p.row_scale; d.resid = p.resid; d.w_n2 = p.w_n2; d.x_n2 = p.x_n2;
        d.y32 = p.y32; d.y16 = p.y16; d.out_scale = p.out_scale; d.ldy = p.ldy;
        int rc = make_half_map(&maps.w[i], p.w, p.w_rows ? p.w_rows : p.rows, p.k, p.w_pitch, kGmRows);
        if (rc) return rc;
        rc = make_half_map(&maps.x[i], p.x, M, static_cast<long long>(p.k) * p.terms, p.x_pitch, nt == 0 ? kPairTok / 2 : nt);
        if (rc) return rc;
    }
    if (nt == 128) return launch_one<128>(a, maps, ks, s);
    if (nt == 64) return launch_one<64>(a, maps, ks, s);
    static bool configured[64] = {};
    int rc = smem_attr(gemm_pair_kernel, kPairSmem, configured);
    if (rc) return rc;
    const int grid_pairs = a.n_tiles < kSms / 2 ? a.n_tiles : kSms / 2;
    cudaError_t e = launch_pdl(gemm_pair_kernel, dim3(2 * grid_pairs), dim3(kPairThreads), kPairSmem, s, a, maps);
    if (e != cudaSuccess) return fail(RWKVQ_E_LAUNCH, "gemm_f16(pair): %s", cudaGetErrorString(e));
    return RWKVQ_OK;
}

}  // namespace rwkvq

using namespace rwkvq;

// ------------------------------------------------------------------ rwkvq_gemm
// workspace: status word (256 bytes) | row scales [M] | fp16 activations [M, IN + 64] | fp16 weights of a row chunk
namespace {
// Row pitch of the fp16 activation copy: 128 bytes more than the row, so that the rows of a TMA box do
// not all map to the same L2 slice (a power-of-two pitch does).
inline size_t x16_pitch(int cols) { return static_cast<size_t>(cols) + 64; }
inline size_t up256(size_t n) { return (n + 255) / 256 * 256; }
// Weights are converted in chunks of rows that fit this scratch, half of L2: it is read back at once.  Whole tiles of
// 256 rows up to 131072 columns, at least one row beyond.
constexpr size_t kGemmScratch = 64u << 20;
inline int gemm_chunk_rows(int cols) {
    const size_t n = kGemmScratch / sizeof(__half) / cols;
    return n >= 256 ? static_cast<int>(n / 256 * 256) : n > 0 ? static_cast<int>(n) : 1;
}
// converted weights of a tensor, a chunk of it where it is larger
inline size_t gemm_scratch(int rows, int cols) {
    return up256(sizeof(__half) * cols * static_cast<size_t>(std::min(rows, gemm_chunk_rows(cols))));
}
inline size_t ws_x16_off(size_t m) { return 256 + up256(sizeof(float) * m); }
inline size_t ws_w_off(size_t m, int x_cols) { return ws_x16_off(m) + (x_cols > 0 ? up256(sizeof(__half) * m * x16_pitch(x_cols)) : 0); }

int gemm_chunks(const rwkvq_qtensor* t, const __half* x16, const float* row_scale, int M, float* y, int64_t ldy, int epilogue,
                const float* resid, __half* scratch, int* status, cudaStream_t s) {
    const int chunk = gemm_chunk_rows(t->cols);
    for (int r0 = 0; r0 < t->rows; r0 += chunk) {
        const int rows = t->rows - r0 < chunk ? t->rows - r0 : chunk;
        int rc = launch_dequant_f16(*t, r0, rows, scratch, nullptr, s);
        if (rc) return rc;
        HgProb p{};
        p.w = scratch; p.w_pitch = t->cols; p.x = x16; p.x_pitch = static_cast<long long>(x16_pitch(t->cols));
        p.rows = rows; p.k = t->cols; p.terms = 1; p.row_scale = row_scale; p.out = HG_F32; p.epilogue = epilogue;
        p.y32 = y + r0; p.resid = resid ? resid + r0 : nullptr; p.ldy = ldy;
        rc = launch_gemm_f16(&p, 1, M, status, s);
        if (rc) return rc;
    }
    return RWKVQ_OK;
}
}  // namespace

size_t rwkvq::gemm_rows_bytes(const rwkvq_qtensor& t, int M) { return ws_w_off(M, t.cols) - 256 + gemm_scratch(t.rows, t.cols); }
int rwkvq::launch_gemm_rows(const rwkvq_qtensor& t, const float* x, int M, long long ldx, float* y, long long ldy, int epilogue,
                            const float* resid, void* scratch, int* status, int* clear, cudaStream_t s) {
    char* ws = static_cast<char*>(scratch) - 256;        // the offsets are those of the workspace, whose head is the status word
    float* scale = reinterpret_cast<float*>(ws + 256);
    __half* x16 = reinterpret_cast<__half*>(ws + ws_x16_off(M));
    int rc = launch_row_scale(x, ldx, t.cols, M, scale, x16, static_cast<long long>(x16_pitch(t.cols)), clear, s);
    if (rc) return rc;
    return gemm_chunks(&t, x16, scale, M, y, ldy, epilogue, resid, reinterpret_cast<__half*>(ws + ws_w_off(M, t.cols)), status, s);
}

extern "C" {

void rwkvq_profiling_gemm_acc_mode(int mode) { g_gemm_acc_mode = mode; }      // rwkvq_profiling.h

size_t rwkvq_gemm_x16_pitch(int cols) { return x16_pitch(cols); }
size_t rwkvq_gemm_workspace_bytes_for(int M, int max_cols) {
    return ws_w_off(static_cast<size_t>(M < 1 ? 1 : M), max_cols) + std::max(kGemmScratch, sizeof(__half) * static_cast<size_t>(max_cols));
}
size_t rwkvq_gemm_workspace_bytes_of(const rwkvq_qtensor* t, int M, int with_rows) {
    if (!t || M < 1 || t->rows < 1 || t->cols < 1) return 0;
    return ws_w_off(M, with_rows ? t->cols : 0) + gemm_scratch(t->rows, t->cols);
}
size_t rwkvq_gemm_workspace_bytes(int M) { return rwkvq_gemm_workspace_bytes_for(M, 16384); }

static int gemm_check(const rwkvq_qtensor* t, const char* who, int M, int64_t ldy, int epilogue, const float* resid) {
    int rc = validate_qtensor(t, who);
    if (rc) return rc;
    RWKVQ_REQUIRE(t->kind == RWKVQ_KIND_SB6 || t->kind == RWKVQ_KIND_SYM, RWKVQ_E_DTYPE,
                  "%s: only sb6 and sym tensors have a tensor-core path (kind %d)", who, t->kind);
    RWKVQ_REQUIRE(M >= 1 && ldy >= t->rows, RWKVQ_E_SHAPE, "%s: M=%d ldy=%lld", who, M, (long long)ldy);
    RWKVQ_REQUIRE(epilogue >= RWKVQ_EPI_NONE && epilogue <= RWKVQ_EPI_ADD, RWKVQ_E_DTYPE, "%s: epilogue %d", who, epilogue);
    RWKVQ_REQUIRE(epilogue != RWKVQ_EPI_ADD || resid, RWKVQ_E_NULL, "%s: resid is null", who);
    return RWKVQ_OK;
}

int rwkvq_gemm(const rwkvq_qtensor* t, const float* x, int M, int64_t ldx, float* y, int64_t ldy, int epilogue,
               const float* resid, void* workspace, size_t workspace_bytes, void* stream) {
    RWKVQ_REQUIRE(x && y && workspace, RWKVQ_E_NULL, "rwkvq_gemm: null pointer");
    int rc = gemm_check(t, "rwkvq_gemm", M, ldy, epilogue, resid);
    if (rc) return rc;
    RWKVQ_REQUIRE(ldx >= t->cols, RWKVQ_E_SHAPE, "rwkvq_gemm: ldx=%lld", (long long)ldx);
    RWKVQ_REQUIRE(aligned(x, 16) && ldx % 4 == 0 && aligned(workspace, 256), RWKVQ_E_ALIGN,
                  "rwkvq_gemm: x and its row stride must be 16-byte aligned, the workspace 256-byte aligned");
    RWKVQ_REQUIRE(workspace_bytes >= rwkvq_gemm_workspace_bytes_of(t, M, 1), RWKVQ_E_LIMIT,
                  "rwkvq_gemm: workspace %zu < %zu bytes", workspace_bytes, rwkvq_gemm_workspace_bytes_of(t, M, 1));
    int* status = static_cast<int*>(workspace);
    rc = launch_gemm_rows(*t, x, M, ldx, y, ldy, epilogue, resid, static_cast<char*>(workspace) + 256, status, status,
                          static_cast<cudaStream_t>(stream));
    return rc ? rc : check_launch("rwkvq_gemm");
}

int rwkvq_gemm_x16(const rwkvq_qtensor* t, const void* x16, const float* row_scale, int M, float* y, int64_t ldy,
                   int epilogue, const float* resid, void* workspace, size_t workspace_bytes, void* stream) {
    RWKVQ_REQUIRE(x16 && row_scale && y && workspace, RWKVQ_E_NULL, "rwkvq_gemm_x16: null pointer");
    int rc = gemm_check(t, "rwkvq_gemm_x16", M, ldy, epilogue, resid);
    if (rc) return rc;
    RWKVQ_REQUIRE(aligned(x16, 16) && aligned(workspace, 256), RWKVQ_E_ALIGN,
                  "rwkvq_gemm_x16: x16 must be 16-byte aligned, the workspace 256-byte aligned");
    RWKVQ_REQUIRE(workspace_bytes >= rwkvq_gemm_workspace_bytes_of(t, M, 0), RWKVQ_E_LIMIT, "rwkvq_gemm_x16: workspace %zu < %zu bytes",
                  workspace_bytes, rwkvq_gemm_workspace_bytes_of(t, M, 0));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    char* ws = static_cast<char*>(workspace);
    int* status = reinterpret_cast<int*>(ws);
    if (cudaMemsetAsync(status, 0, sizeof(int), s) != cudaSuccess) return check_launch("rwkvq_gemm_x16(status)");
    rc = gemm_chunks(t, static_cast<const __half*>(x16), row_scale, M, y, ldy, epilogue, resid,
                     reinterpret_cast<__half*>(ws + ws_w_off(M, 0)), status, s);
    return rc ? rc : check_launch("rwkvq_gemm_x16");
}

}  // extern "C"
