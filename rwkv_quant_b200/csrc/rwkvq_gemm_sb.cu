// Quantized linear for small batches (9 to 256 right-hand sides) on the tcgen05 tensor cores at fp32 grade:
// packed weights converted on the way into the operands, every byte read once per 128 tokens.
//
//     y[n, o] = epi( sum_c W[o, c] x[n, c] )
//
// Both operands are carried as two fp16 terms (weights: p = fp16(q s) and its exact rounding error e;
// activations: hi + lo of x * 2^s, |x * 2^s| <= 2^9); per 16 columns p multiplies [hi | lo] side by side as one MMA of 2 NT
// token columns, so that shared memory delivers a weight once for both terms of x, and e multiplies hi.  p hi has an fp32
// accumulator of its own in tensor memory: an accumulator is truncated at every step, and e hi beside p lo costs p hi none
// (error of the logits against 64 bits at 17 streams 1.09e-5 -> 7.0e-6, at 64 1.10e-5 -> 7.1e-6, no time).  sb6
// block mins (fp16 by definition) times the block sums of x (as a pair too) are one more MMA of 16 columns per super-block.
//
// A CTA owns 128 rows and a K slice (cluster of ks CTAs along K, reduced through distributed shared memory in rank
// order) and is a pipeline over units of 128 columns, two of them in flight:
//   warps 0-15   weights, four groups of 128 threads: group g turns block g (32 columns) of every unit into p and e, a thread
//                its own row, into tensor memory (the A operand of the MMA: lane = row), so that shared memory carries the
//                activations only (with p and e there their stores and the MMAs' reads bound 64 columns at 0.52 us)
//   warp 16      TMA of the activation pairs, which split_rows_kernel or the LayerNorm kernels have made once
//   warp 17      MMAs, the loop run by the whole warp so that descriptors stay in uniform registers
//   warp 18      TMA of the packed weights, super-blocks of 256 columns, two ahead; they do not depend on the producer of x
// Bound: the turn of the MMA warp.  With conversion, stores and MMAs all switched off, a super-block of four units still took 1.6 of its
// 1.7 us: a wait and a commit are some 400 cycles whatever lies between them.  Hence units of 128 columns with one barrier for
// all of their weights and activations, and waits that poll: 1.5B step of 64 streams 2.76 -> 2.60 ms, of 100 4.19 -> 3.59 (128 tokens a tile:
// its MMAs are next, 1.4 us a super-block).  Weights by per-thread cp.async cost the load pipe a line per lane: 2.4 us until
// the first bytes were asked for, 0.5 by TMA.
// The mma.sync form of the same product (rwkvq_gemv_batch.cu) issues 3 MMAs of 16 x 8 x 16 per warp and step and tops out
// at 0.92 G MMA/s per SM.
// Every mbarrier wait is bounded.  A warp whose wait ran out waits and arrives no more (an arrival for a unit that it did not wait for
// would count towards a phase whose copies are still on their way), the status word is set and all roles run to the common end.
// The two warps that issue copies leave their part only when those have landed, or a wait for them has run out too.
#include "rwkvq_gemm_sb.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "rwkvq_ahead.cuh"
#include "rwkvq_tc.cuh"

namespace cg = cooperative_groups;

namespace rwkvq {

constexpr int kSbGroups = 4;                      // = blocks of 32 columns in a unit
constexpr int kSbWeightThreads = kSbGroups * kGmRows, kSbThreads = kSbWeightThreads + 96;
constexpr int kSbTmaWarp = kSbWeightThreads / 32, kSbMmaWarp = kSbTmaWarp + 1, kSbRawWarp = kSbTmaWarp + 2;
constexpr int kSbACols = 128;                     // tensor-memory columns of a unit: p 64, e 64
constexpr uint32_t kSbTmemCols = 512;
constexpr int kSbPitch = kGmRows + 4;             // partial tile [NT][kSbPitch]
constexpr int kSbMaxMats = 4;

struct SbArgs {
    QView t[kSbMaxMats];
    const __half* sums[kSbMaxMats];
    const float* unscale[kSbMaxMats];
    float* y[kSbMaxMats];
    const float* resid[kSbMaxMats];
    float* amax_out[kSbMaxMats];
    long long ldy;
    int n_tokens, epilogue;
    int nt;                                       // tokens of a CTA's tile: 16, 32, 64 or, where NT is 128, any multiple of 16
    int row_tiles;                                // of one matrix
    int n_tiles;                                  // matrices * row_tiles
    int n_sb;                                     // super-blocks of a row
    int ks;
    int* status;
};
struct SbMaps { CUtensorMap hi[kSbMaxMats], lo[kSbMaxMats], codes[kSbMaxMats], rec[kSbMaxMats], planes[kSbMaxMats]; };

// A super-block of 128 packed rows in shared memory, as TMA leaves it: codes in boxes of 128 bytes a row and planes, swizzled by
// the width of their rows so that a thread's 16-byte pieces of its own row meet no bank conflict, and the scale records.
template <int L>
struct SbLayout {
    static constexpr bool SB6 = L <= ML_SB6_6;
    static constexpr int CODE_ROW = L == ML_SYM8 ? 256 : 128, PLANE_ROW = L == ML_SB6_5 ? 32 : (L == ML_SB6_6 || L == ML_SYM6) ? 64 : 0;
    static constexpr int OFF_P = kGmRows * CODE_ROW, OFF_R = OFF_P + kGmRows * PLANE_ROW, RAW = OFF_R + kGmRows * 16;
    static_assert(RAW % 1024 == 0, "swizzle");
};

template <int L, int NT>
struct SbGeo {
    static constexpr int U = 2;                                      // units of operands in flight (three: no gain at 3 to 100 streams)
    static constexpr int AHEAD = 2;                                  // super-blocks of packed weights in flight (three: no gain either)
    static constexpr int BATOM = 2 * NT * 128, BSLAB = 2 * BATOM;     // activation pairs of 64 columns, of a unit
    static constexpr int MA = SbLayout<L>::SB6 ? kGmRows * 32 : 0, MB = SbLayout<L>::SB6 ? 2 * NT * 32 : 0;     // min operands of a super-block
    static constexpr int PART = NT * kSbPitch * 4;                   // partial tile of a K slice, over the operands
    static constexpr int OFF_MA = U * BSLAB, OFF_MB = OFF_MA + 2 * MA, OFF_RAW = OFF_MB + 2 * MB,
                         SMEM = OFF_RAW + AHEAD * SbLayout<L>::RAW;
    // one CTA per SM: two could wait for each other's tensor memory inside a cluster
    static constexpr size_t BYTES = (SMEM > 119 * 1024 ? SMEM : 119 * 1024) + 1024;
    static_assert(PART <= SMEM, "partial tile");
    static_assert(2 * NT + U * kSbACols <= static_cast<int>(kSbTmemCols), "tensor memory");
    static_assert(BYTES <= 226 * 1024, "shared memory");
    static_assert(OFF_RAW % 1024 == 0, "swizzle");
};

__device__ __forceinline__ void sb_tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
                 "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}
// A from tensor memory (lane = row, a 32-bit column = two consecutive k)
__device__ __forceinline__ void umma_f16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
template <int NC>
__device__ __forceinline__ void sb_tmem_ld(uint32_t taddr, float (&v)[NC]) {
    uint32_t r[NC];
    if constexpr (NC == 4) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr));
    } else if constexpr (NC == 8) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "r"(taddr));
    } else {
        static_assert(NC == 16, "columns");
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                       "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                     : "r"(taddr));
    }
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < NC; ++i) v[i] = __uint_as_float(r[i]);
}

// Codes of a block of 32 columns as bytes in column order; its relayouted planes (pl, pl2) give the high bits of four codes with
// one shift and mask.
template <int L>
__device__ __forceinline__ void sb_codes(const uint4& c0, const uint4& c1, uint32_t pl, uint32_t pl2, uint32_t (&bytes)[8]) {
    const uint32_t w[4] = {c0.x, c0.y, c0.z, c0.w};
    if constexpr (SbLayout<L>::SB6) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {              // byte k of the block: column k (low), k + 16 (high)
            bytes[i] = w[i] & 0x0F0F0F0Fu;
            bytes[4 + i] = (w[i] >> 4) & 0x0F0F0F0Fu;
            if (L == ML_SB6_5) {
                bytes[i] |= (pl << (4 - i)) & 0x10101010u;
                bytes[4 + i] |= (pl >> i) & 0x10101010u;
            } else if (L == ML_SB6_6) {
                bytes[i] |= (i < 2 ? (pl << (4 - 2 * i)) : (pl >> (2 * i - 4))) & 0x30303030u;
                bytes[4 + i] |= (i < 2 ? (pl2 << (4 - 2 * i)) : (pl2 >> (2 * i - 4))) & 0x30303030u;
            }
        }
    } else if constexpr (L == ML_SYM8) {
        const uint32_t w8[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) bytes[i] = w8[i] ^ 0x80808080u;          // code + 128
    } else {
#pragma unroll
        for (int h = 0; h < 2; ++h) {              // block h of 16: words 2h, 2h + 1; byte k: column k (low), column k + 8 (high)
            const uint32_t p = h ? pl2 : pl;
            bytes[4 * h] = (w[2 * h] & 0x0F0F0F0Fu) | ((p << 4) & 0x30303030u);
            bytes[4 * h + 1] = (w[2 * h + 1] & 0x0F0F0F0Fu) | ((p << 2) & 0x30303030u);
            bytes[4 * h + 2] = ((w[2 * h] >> 4) & 0x0F0F0F0Fu) | (p & 0x30303030u);
            bytes[4 * h + 3] = ((w[2 * h + 1] >> 4) & 0x0F0F0F0Fu) | ((p >> 2) & 0x30303030u);
        }
    }
}
// Two bytes of `two` (scale codes) times the fp16 in both halves of dd
__device__ __forceinline__ __half2 sb_sym_scales(uint32_t two, uint32_t dd) {
    const uint32_t x = two ^ 0x8080u, u = (x & 0xFFu) | ((x << 8) & 0x00FF0000u) | 0x64006400u;      // 1024 + code + 128
    return __hmul2(__hsub2(*reinterpret_cast<const __half2*>(&u), __float2half2_rn(1152.f)), *reinterpret_cast<const __half2*>(&dd));
}

// a whole warp: one answer, and together again behind it
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity) { return __all_sync(0xFFFFFFFFu, mbar_poll_bounded(bar, parity)); }

template <int L, int NT>
__global__ void __launch_bounds__(kSbThreads, 1) gemm_sb_kernel(const __grid_constant__ SbArgs a, const __grid_constant__ SbMaps maps, const __grid_constant__ Ahead ahead) {
    using G = SbGeo<L, NT>;
    using Y = SbLayout<L>;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    // the operands of a unit are complete (16 weight warps + the TMA bytes) / have been multiplied.  A super-block's min
    // operands are part of its units: mins with the weights of each, block sums with the activations of the first.
    // Two buffers of them need no barrier of their own: the unit that writes buffer s % 2 again has waited for the MMA that
    // read it, or for one behind (unit 2 s + 4 - U, U <= 3).
    __shared__ uint64_t bar_full[G::U], bar_empty[G::U], bar_done;
    __shared__ uint64_t raw_full[G::AHEAD], raw_empty[G::AHEAD];      // packed weights have arrived / are in registers (16 warps)
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_fail;
    __shared__ float s_un[NT];
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ks = a.ks, z = blockIdx.x % ks, first_tile = blockIdx.x / ks, tile_step = gridDim.x / ks;
    const int nt = NT > 64 ? a.nt : NT, n0 = blockIdx.y * nt, nn = min(nt, a.n_tokens - n0);
    const int sb0 = a.n_sb * z / ks, n_super = a.n_sb * (z + 1) / ks - sb0;     // this CTA's K slice
    const int n_my = (a.n_tiles - first_tile + tile_step - 1) / tile_step;

    if (tid == 0) {
        for (int s = 0; s < G::U; ++s) { mbar_init(&bar_full[s], kSbWeightThreads / 32 + 1); mbar_init(&bar_empty[s], 1); }
        for (int s = 0; s < G::AHEAD; ++s) { mbar_init(&raw_full[s], 1); mbar_init(&raw_empty[s], kSbWeightThreads / 32); }
        mbar_init(&bar_done, 1);
        s_fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    pdl_launch_dependents();
    if (warp == kSbMmaWarp) tmem_alloc(&s_tmem, kSbTmemCols);
    if (Y::SB6) {                                                    // K 8-15 of the min operands and the rows beyond nn stay zero
        for (int i = tid; i < 2 * (G::MA + G::MB) / 16; i += kSbThreads) reinterpret_cast<uint4*>(smem + G::OFF_MA)[i] = make_uint4(0, 0, 0, 0);
        fence_async_smem();
    }

    // weight threads: group grp takes block grp of every unit, thread wrow its row
    const int grp = tid / kGmRows, wrow = tid % kGmRows;
    if (warp == kSbTmaWarp) ahead_prefetch(ahead, blockIdx.x + gridDim.x * blockIdx.y, gridDim.x * gridDim.y);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    if (warp == kSbTmaWarp) pdl_wait();                              // the activations; the others wait before they read or store

    int sb_before = 0;                                               // super-blocks of the tiles before
    bool alive = true;                                               // no wait of this warp has run out
    uint32_t done_phase = 0;
    for (int ti = 0; ti < n_my; ++ti) {
        const int tile = first_tile + ti * tile_step, mat = tile / a.row_tiles, row0 = (tile % a.row_tiles) * kGmRows;
        const QView& t = a.t[mat];
        if (warp == kSbMmaWarp) {
            // ------------------------------------------------------------------ MMA issuer (whole warp, one lane elected)
            const uint32_t id2 = umma_idesc(2 * nt), id1 = umma_idesc(nt);
            const uint64_t b0 = umma_desc(smem_addr(smem));
            const uint64_t ma0 = umma_desc_plain(smem_addr(smem + G::OFF_MA), kGmRows * 16, 128);
            const uint64_t mb0 = umma_desc_plain(smem_addr(smem + G::OFF_MB), 2 * nt * 16, 128);
            if (ti == 0) pdl_wait();
            for (int n = lane; n < nt; n += 32) s_un[n] = n < nn ? __ldcg(a.unscale[mat] + n0 + n) : 0.f;   // read behind bar_done
            uint32_t elected;
            asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xFFFFFFFF;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(elected));
            int buf = (2 * sb_before) % G::U, ph = (2 * sb_before / G::U) & 1;
            for (int u = 0; u < 2 * n_super; ++u) {
                alive = alive && warp_wait(&bar_full[buf], ph);
                if (!alive) break;
                tc_fence_after();
                const uint32_t pa = tmem + 2 * NT + buf * kSbACols, ea = pa + kSbACols / 2;
                const uint64_t bd = b0 + (static_cast<uint64_t>(buf * G::BSLAB) >> 4);
                if (elected) {
#pragma unroll
                    for (int k = 0; k < 8; ++k) {                    // e meets the high halves only (e lo is below 2^-22), beside p lo
                        const uint64_t bk = bd + (static_cast<uint64_t>((k >> 2) * G::BATOM) >> 4) + 2 * (k & 3);
                        umma_f16_ta(tmem, pa + 8 * k, bk, id2, (u | k) ? 1u : 0u);
                        umma_f16_ta(tmem + nt, ea + 8 * k, bk, id1, 1u);
                    }
                    if (Y::SB6 && (u & 1)) {                         // the super-block's mins are complete with its second unit
                        const int ms = (sb_before + (u >> 1)) & 1;
                        umma_f16(tmem, ma0 + (static_cast<uint64_t>(ms * G::MA) >> 4), mb0 + (static_cast<uint64_t>(ms * G::MB) >> 4), id2, 1u);
                    }
                    umma_commit(&bar_empty[buf]);
                }
                __syncwarp();
                if (++buf == G::U) { buf = 0; ph ^= 1; }
            }
            if (alive && elected) umma_commit(&bar_done);
        } else if (warp == kSbRawWarp) {
            // ------------------------------------------------------------------ packed weights: do not depend on the producer of x
            if (lane == 0 && alive) {
                int qi = sb_before;
                for (; qi < sb_before + n_super; ++qi) {
                    const int sb = qi - sb_before, slot = qi % G::AHEAD;
                    alive = alive && (qi < G::AHEAD || mbar_poll_bounded(&raw_empty[slot], (qi / G::AHEAD - 1) & 1));
                    if (!alive) break;
                    unsigned char* w = smem + G::OFF_RAW + slot * Y::RAW;
                    mbar_expect_tx(&raw_full[slot], Y::RAW);
#pragma unroll
                    for (int c = 0; c < Y::CODE_ROW / 128; ++c)
                        tma_load_2d(w + c * (kGmRows * 128), &maps.codes[mat], (sb0 + sb) * Y::CODE_ROW + c * 128, row0, &raw_full[slot]);
                    if (Y::PLANE_ROW > 0) tma_load_2d(w + Y::OFF_P, &maps.planes[mat], (sb0 + sb) * Y::PLANE_ROW, row0, &raw_full[slot]);
                    tma_load_2d(w + Y::OFF_R, &maps.rec[mat], (sb0 + sb) * 16, row0, &raw_full[slot]);
                }
                if (!alive || ti == n_my - 1)                        // the last copy of each slot: all others were waited for
                    for (int q = max(0, qi - G::AHEAD); q < qi; ++q) mbar_poll_bounded(&raw_full[q % G::AHEAD], (q / G::AHEAD) & 1);
            }
        } else if (warp == kSbTmaWarp) {
            // ------------------------------------------------------------------ activation pairs
            if (lane == 0 && alive) {
                int g = 2 * sb_before;
                for (; g < 2 * (sb_before + n_super); ++g) {
                    const int u = g - 2 * sb_before, buf = g % G::U;
                    alive = alive && (g < G::U || mbar_poll_bounded(&bar_empty[buf], (g / G::U - 1) & 1));
                    if (!alive) break;
                    unsigned char* b = smem + buf * G::BSLAB;
                    const bool with_sums = Y::SB6 && (u & 1) == 0;
                    mbar_expect_tx(&bar_full[buf], 4 * nt * 128 + (with_sums ? 2 * nn * 16 : 0));
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const int x = sb0 * 256 + u * 128 + c * 64;
                        tma_load_2d(b + c * G::BATOM, &maps.hi[mat], x, n0, &bar_full[buf]);
                        tma_load_2d(b + c * G::BATOM + nt * 128, &maps.lo[mat], x, n0, &bar_full[buf]);
                    }
                    if (with_sums) {
                        unsigned char* m = smem + G::OFF_MB + ((g >> 1) & 1) * G::MB;
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                             smem_addr(m + h * nt * 16)),
                                         "l"(a.sums[mat] + ((static_cast<size_t>(sb0 + (u >> 1)) * 2 + h) * a.n_tokens + n0) * 8), "r"(nn * 16),
                                         "r"(smem_addr(&bar_full[buf]))
                                         : "memory");
                    }
                }
                if (!alive || ti == n_my - 1)                        // the last unit of each buffer has been multiplied
                    for (int d = max(0, g - G::U); d < g; ++d) mbar_poll_bounded(&bar_empty[d % G::U], (d / G::U) & 1);
            }
        } else {
            // ------------------------------------------------------------------ weights
            // sym: the super-scale is not part of the staged record; one super-block ahead
            const __half* dp = Y::SB6 ? nullptr : t.d + static_cast<size_t>(min(row0 + wrow, t.rows - 1)) * (t.cols >> 8) + sb0;
            uint32_t d_next = Y::SB6 ? 0u : __half_as_ushort(__ldg(dp));
            const __half2 bias = __float2half2_rn(L == ML_SYM8 ? 1152.f : L == ML_SYM6 ? 1056.f : 1024.f);
            const uint32_t lane_base = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + 2 * NT;
#pragma unroll 1
            for (int sb = 0; sb < n_super; ++sb) {
                const int qi = sb_before + sb, slot = qi % G::AHEAD;
                alive = alive && warp_wait(&raw_full[slot], (qi / G::AHEAD) & 1);
                const unsigned char* raw = smem + G::OFF_RAW + slot * Y::RAW;
                // blocks grp and 4 + grp of the super-block
                uint4 code[2], code2[2];
                uint32_t pl[2] = {0u, 0u}, pl2[2] = {0u, 0u};
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (Y::CODE_ROW == 128) {
                        code[h] = code2[h] = *reinterpret_cast<const uint4*>(raw + wrow * 128 + (((4 * h + grp) ^ (wrow & 7)) << 4));
                    } else {                                         // 32 bytes a block, four blocks a box
                        const unsigned char* crow = raw + h * (kGmRows * 128) + wrow * 128;
                        code[h] = *reinterpret_cast<const uint4*>(crow + (((2 * grp) ^ (wrow & 7)) << 4));
                        code2[h] = *reinterpret_cast<const uint4*>(crow + (((2 * grp + 1) ^ (wrow & 7)) << 4));
                    }
                    if (Y::PLANE_ROW == 64) {                        // 8 bytes a block
                        const uint4 p4 = *reinterpret_cast<const uint4*>(raw + Y::OFF_P + wrow * 64 + (((2 * h + (grp >> 1)) ^ ((wrow >> 1) & 3)) << 4));
                        pl[h] = grp & 1 ? p4.z : p4.x;
                        pl2[h] = grp & 1 ? p4.w : p4.y;
                    }
                    if (Y::PLANE_ROW == 32) {                        // 4 bytes a block
                        const uint4 p4 = *reinterpret_cast<const uint4*>(raw + Y::OFF_P + wrow * 32 + ((h ^ ((wrow >> 2) & 1)) << 4));
                        pl[h] = word_of(p4, grp);
                    }
                }
                const uint4 rec = *reinterpret_cast<const uint4*>(raw + Y::OFF_R + wrow * 16);
                __syncwarp();
                if (lane == 0 && alive) mbar_arrive(&raw_empty[slot]);        // the super-block is in registers
                const uint32_t dd = d_next * 0x00010001u;
                if (!Y::SB6 && sb + 1 < n_super) d_next = __half_as_ushort(__ldg(dp + sb + 1));
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int g = 2 * qi + h, buf = g % G::U;
                    // scales of the block's halves of 16 columns and its min; fp16 values by the codec's definition: one half-precision
                    // multiply of the exact small integer
                    __half2 s_lo, s_hi, mins = __float2half2_rn(0.f);
                    if (Y::SB6) {
                        __half2 hs;
                        sb6_pair_scales_h2(rec, 2 * h + (grp >> 1), hs, mins);
                        s_lo = s_hi = grp & 1 ? __high2half2(hs) : __low2half2(hs);
                    } else {
                        const uint32_t w = h ? (grp & 2 ? rec.w : rec.z) : (grp & 2 ? rec.y : rec.x);
                        const __half2 s4 = sb_sym_scales(grp & 1 ? w >> 16 : w & 0xFFFFu, dd);
                        s_lo = __low2half2(s4);
                        s_hi = __high2half2(s4);
                    }
                    uint32_t bytes[8], pw[16], ew[16];
                    sb_codes<L>(code[h], code2[h], pl[h], pl2[h], bytes);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        uint2 pa, ea;
                        bytes_to_half4_pair(bytes[j], bias, j < 4 ? s_lo : s_hi, pa, ea);
                        pw[2 * j] = pa.x; pw[2 * j + 1] = pa.y;
                        ew[2 * j] = ea.x; ew[2 * j + 1] = ea.y;
                    }
                    if (g >= G::U) {                                 // the MMAs that read this buffer have completed
                        alive = alive && warp_wait(&bar_empty[buf], (g / G::U - 1) & 1);
                        tc_fence_after();
                    }
                    const uint32_t ta = lane_base + buf * kSbACols + 16 * grp;
                    sb_tmem_st16(ta, pw);
                    sb_tmem_st16(ta + kSbACols / 2, ew);
                    if (Y::SB6) {
                        *reinterpret_cast<__half*>(smem + G::OFF_MA + (qi & 1) * G::MA + wrow * 16 + (4 * h + grp) * 2) =
                            grp & 1 ? __high2half(mins) : __low2half(mins);
                        fence_async_smem();
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0 && alive) mbar_arrive(&bar_full[buf]);
                }
            }
        }
        sb_before += n_super;
        // ---------------------------------------------------------------------- epilogue of the tile
        __syncwarp();
        if (warp != kSbTmaWarp && warp != kSbRawWarp) {
            alive = alive && warp_wait(&bar_done, done_phase);
            done_phase ^= 1;
            tc_fence_after();
            if (ti == 0) pdl_wait();                                 // token scales, residual, output
        }
        constexpr int TC = NT < 64 ? NT / 4 : 16;                    // tokens a warp takes at a time; four warps share a lane quadrant
        const int q = warp & 3, tg = warp >> 2, rl = q * 32 + lane, row = row0 + rl;
        if (!alive) s_fail = 1;
        const bool row_ok = row < t.rows && alive && !s_fail;
        float* y = a.y[mat] + static_cast<size_t>(n0) * a.ldy + row;
        const float* rs = a.resid[mat] ? a.resid[mat] + static_cast<size_t>(n0) * a.ldy + row : nullptr;
        float* am_out = a.amax_out[mat] ? a.amax_out[mat] + n0 : nullptr;
        const bool add = a.epilogue == RWKVQ_EPI_ADD;
        // a lane's U values at tokens first + j * step (whole warps; 32 lanes = 32 consecutive rows).  Loads first: behind
        // a store each would wait for its own L2 round trip (16 of them: 5 us).
        auto load_resid = [&](auto& r, int first, int step, int end) {
#pragma unroll
            for (int j = 0; j < static_cast<int>(sizeof(r) / sizeof(r[0])); ++j) {
                const int n = first + j * step;
                r[j] = add && row_ok && n < end ? __ldcg(rs + static_cast<size_t>(n) * a.ldy) : 0.f;
            }
        };
        auto store = [&](const auto& v, const auto& r, int first, int step, int end) {
#pragma unroll
            for (int j = 0; j < static_cast<int>(sizeof(v) / sizeof(v[0])); ++j) {
                const int n = first + j * step;
                float o = v[j];
                if (a.epilogue == RWKVQ_EPI_RELU2) { o = fmaxf(o, 0.f); o = o * o; }
                else if (add) o = __fadd_rn(o, r[j]);
                if (row_ok && n < end) y[static_cast<size_t>(n) * a.ldy] = o;
                if (am_out != nullptr && n < end) {                  // |o| as bits orders like the float, a NaN above every number
                    const unsigned m = __reduce_max_sync(0xFFFFFFFFu, row_ok ? __float_as_uint(fabsf(o)) : 0u);
                    if (lane == 0 && m != 0u) atomicMax(reinterpret_cast<unsigned*>(am_out) + n, m);
                }
            }
        };
        auto accumulators = [&](float (&v)[TC], int c0) {
            float lo[TC];
            const uint32_t base = tmem + (static_cast<uint32_t>(q * 32) << 16) + c0;
            sb_tmem_ld<TC>(base, v);
            sb_tmem_ld<TC>(base + nt, lo);
#pragma unroll
            for (int j = 0; j < TC; ++j) v[j] = (v[j] + lo[j]) * s_un[c0 + j];
        };
        if (ks == 1) {
            if (warp < kSbTmaWarp) {
#pragma unroll 1
                for (int c = 0; c < NT; c += 4 * TC) {              // one pass up to 64 tokens
                    const int c0 = c + tg * TC;
                    if (c0 >= nt) break;
                    float v[TC], r[TC];
                    load_resid(r, c0, 1, nn);
                    accumulators(v, c0);
                    store(v, r, c0, 1, nn);
                }
                tc_fence_before();
            }
            // the accumulator is free for the next tile
            if (warp != kSbTmaWarp && warp != kSbRawWarp) asm volatile("bar.sync 1, %0;" ::"n"(kSbThreads - 64) : "memory");
            tc_fence_after();
        } else {
            float* part = reinterpret_cast<float*>(smem);            // every MMA that read the operands has completed
            if (warp < kSbTmaWarp) {
#pragma unroll 1
                for (int c = 0; c < NT; c += 4 * TC) {              // one pass up to 64 tokens
                    const int c0 = c + tg * TC;
                    if (c0 >= nt) break;
                    float v[TC];
                    accumulators(v, c0);
#pragma unroll
                    for (int j = 0; j < TC; ++j) part[(c0 + j) * kSbPitch + rl] = v[j];
                }
                tc_fence_before();
            }
            // this CTA's share of the tokens, ranks added in order; U tokens of K ranks in flight per thread
            const int per = (nn + ks - 1) / ks, first = z * per + tg, end = min(nn, (z + 1) * per);
            auto reduce = [&](auto u_tag, auto k_tag) {
                constexpr int U = decltype(u_tag)::value, K = decltype(k_tag)::value;
                float r[U];
                if (warp < kSbTmaWarp) load_resid(r, first, 4, end);
                cluster.sync();
                if (warp < kSbTmaWarp) {
#pragma unroll 1
                    for (int nb = first; nb < end; nb += 4 * U) {
                        float pv[K][U], v[U];
                        if (nb != first) load_resid(r, nb, 4, end);
#pragma unroll
                        for (int u = 0; u < K; ++u) {
                            const float* src = cluster.map_shared_rank(part, u < ks ? u : 0);
#pragma unroll
                            for (int j = 0; j < U; ++j) pv[u][j] = u < ks ? src[min(nb + 4 * j, nt - 1) * kSbPitch + rl] : 0.f;
                        }
#pragma unroll
                        for (int j = 0; j < U; ++j) {
                            v[j] = pv[0][j];
#pragma unroll
                            for (int u = 1; u < K; ++u) v[j] += pv[u][j];
                        }
                        store(v, r, nb, 4, end);
                    }
                }
            };
            if (ks == 2) reduce(std::integral_constant<int, NT >= 64 ? 8 : 4>{}, std::integral_constant<int, 2>{});
            else if (ks <= 4) reduce(std::integral_constant<int, 4>{}, std::integral_constant<int, 4>{});
            else reduce(std::integral_constant<int, 4>{}, std::integral_constant<int, 8>{});
            cluster.sync();                                          // nobody leaves while a peer still reads its partial tile
        }
    }
    __syncthreads();
    if (tid == 0 && s_fail) atomicCAS(a.status, 0, RWKVQ_E_TIMEOUT);
    tc_fence_after();
    if (warp == kSbMmaWarp) tmem_dealloc(tmem, kSbTmemCols);
}

// fp32 rows -> pairs, one CTA per row.  Bound: latency (a load, a block maximum, the stores); rows of up to 8192 columns
// stay in registers between the two uses.
__global__ void __launch_bounds__(512) split_rows_kernel(const float* __restrict__ x, long long ldx, int cols, const SbRows o, int N, int* status) {
    __shared__ float red[16];
    pdl_launch_dependents();
    pdl_wait();
    if (status != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *status = 0;      // of the product that follows
    const int n = blockIdx.x, n8 = cols >> 3;                        // n8 is a multiple of 32: whole warps take a pass together
    const float4* row = reinterpret_cast<const float4*>(x + static_cast<size_t>(n) * ldx);
    constexpr int kKeep = 2;
    float4 f[kKeep][2];
    float m = 0.f;
    auto upd = [&](const float4& v) {
        m = fmaxf(m, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
        if (!(fabsf(v.x) + fabsf(v.y) + fabsf(v.z) + fabsf(v.w) < INFINITY)) m = INFINITY;
    };
#pragma unroll
    for (int k = 0; k < kKeep; ++k) {
        const int i = threadIdx.x + k * 512;
        f[k][0] = i < n8 ? __ldcg(row + 2 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
        f[k][1] = i < n8 ? __ldcg(row + 2 * i + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int k = 0; k < kKeep; ++k) { upd(f[k][0]); upd(f[k][1]); }
    for (int i = threadIdx.x + kKeep * 512; i < n8; i += 512) { upd(__ldcg(row + 2 * i)); upd(__ldcg(row + 2 * i + 1)); }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, s));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    m = red[threadIdx.x & 15];
#pragma unroll
    for (int s = 8; s > 0; s >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, s));
    float s1, u1;
    sb_scale(m, s1, u1);
    if (threadIdx.x == 0) o.unscale[n] = u1;
    auto put = [&](int i, const float4& a, const float4& b) {
        const float v[8] = {a.x * s1, a.y * s1, a.z * s1, a.w * s1, b.x * s1, b.y * s1, b.z * s1, b.w * s1};
        sb_store_pair(o, n, N, i, v);
    };
#pragma unroll
    for (int k = 0; k < kKeep; ++k)
        if (static_cast<int>(threadIdx.x) + k * 512 < n8) put(threadIdx.x + k * 512, f[k][0], f[k][1]);
    for (int i = threadIdx.x + kKeep * 512; i < n8; i += 512) put(i, __ldcg(row + 2 * i), __ldcg(row + 2 * i + 1));
}

int launch_split_rows(const float* x, long long ldx, int cols, int N, const SbRows& o, int* status, cudaStream_t s) {
    cudaError_t e = launch_pdl(split_rows_kernel, dim3(N), dim3(512), 0, s, x, ldx, cols, o, N, status);
    if (e != cudaSuccess) return fail(RWKVQ_E_LAUNCH, "split_rows: %s", cudaGetErrorString(e));
    return RWKVQ_OK;
}

namespace {

int sb_layout_of(const rwkvq_qtensor& t) {
    if (t.kind == RWKVQ_KIND_SB6) return ML_SB6_4 + (t.bits - 4);
    return t.bits == 8 ? ML_SYM8 : ML_SYM6;
}

// Clusters of c CTAs the device holds at once (one CTA per SM): whole clusters of a GPC, e.g. 16 of 6 but not of 7.
template <int L, int NT>
int resident_clusters(int dev, int c) {
    static int known[64][9] = {};
    if (dev < 64 && known[dev][c] > 0) return known[dev][c];
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(c);
    cfg.blockDim = dim3(kSbThreads);
    cfg.dynamicSmemBytes = SbGeo<L, NT>::BYTES;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = c; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_sb_kernel<L, NT>, &cfg) != cudaSuccess || n < 1) {
        cudaGetLastError();
        n = std::max(1, 96 / c);
    }
    if (dev < 64) known[dev][c] = n;
    return n;
}

template <int L, int NT>
int launch_sb(SbArgs& a, const SbMaps& maps, int groups, int force_ks, const Ahead& ahead, cudaStream_t s) {
    static bool configured[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) dev = 0;
    if (dev >= 64 || !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(gemm_sb_kernel<L, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(SbGeo<L, NT>::BYTES));
        if (e != cudaSuccess) return fail(RWKVQ_E_LIMIT, "gemm_sb: %zu bytes of shared memory: %s", SbGeo<L, NT>::BYTES, cudaGetErrorString(e));
        for (int c = 2; c <= 8; ++c) resident_clusters<L, NT>(dev, c);
        if (dev < 64) configured[dev] = true;
    }
    // K split into up to 8 slices of whole super-blocks, by a model of the slowest CTA in microseconds fitted to
    // [2048, 2048] .. [65536, 2048] at 8 to 128 rows: 0.37 to 0.55 per 64 columns by the tile's width, 5 for ramp and store, 3.5 for the
    // cluster reduction; without a split the CTAs are persistent and pay the ramp once.  (Fitted to units of 64 columns; with units of
    // 128, 0.30, 0.33 and 0.41 per 64 at 13, 64 and 100 rows, it still picks the fastest split or one within 2 % of it: 8 shapes
    // [2048, 2048] .. [10240, 2560] and [2560, 10240], sb6 4 bits and sym 8 bits, at those rows, every split from 1 to 8)
    const double stage = std::max(0.37, 0.41 + 0.0022 * (a.nt - 64));
    double best = 1e300;
    a.ks = 1;
    for (int c = 1; c <= 8 && c <= a.n_sb; ++c) {
        const int fit = c == 1 ? 148 : resident_clusters<L, NT>(dev, c);
        const double waves = static_cast<double>((a.n_tiles * groups + fit - 1) / fit), work = ((a.n_sb + c - 1) / c) * 4 * stage;
        const double t = c == 1 ? waves * (work + 1.5) + 4.0 : waves * (work + 5.0) + 3.5;
        if (t < best) { best = t; a.ks = c; }
    }
    if (force_ks > 0 && force_ks <= 8 && force_ks <= a.n_sb) a.ks = force_ks;
    cudaLaunchConfig_t cfg{};
    // one wave of persistent CTAs where K is not split
    cfg.gridDim = dim3(a.ks > 1 ? a.n_tiles * a.ks : std::min(a.n_tiles, std::max(1, 148 / groups)), groups);
    cfg.blockDim = dim3(kSbThreads);
    cfg.dynamicSmemBytes = SbGeo<L, NT>::BYTES;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = a.ks; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_sb_kernel<L, NT>, a, maps, ahead);
    if (e != cudaSuccess) return fail(RWKVQ_E_LAUNCH, "gemm_sb: %s", cudaGetErrorString(e));
    return RWKVQ_OK;
}

template <int L>
int launch_sb_nt(SbArgs& a, const SbMaps& maps, int nt, int groups, int force_ks, const Ahead& ahead, cudaStream_t s) {
    if (nt <= 16) return launch_sb<L, 16>(a, maps, groups, force_ks, ahead, s);
    if (nt <= 32) return launch_sb<L, 32>(a, maps, groups, force_ks, ahead, s);
    if (nt <= 64) return launch_sb<L, 64>(a, maps, groups, force_ks, ahead, s);
    return launch_sb<L, 128>(a, maps, groups, force_ks, ahead, s);
}

}  // namespace

bool gemm_sb_ok(const rwkvq_qtensor& t) {
    // 16-byte copies of codes, records (sym: block scales) and planes; the mma.sync form reads block scales by 8 bytes
    return gemm_tcb_ok(t) && (t.kind == RWKVQ_KIND_SB6 || t.kind == RWKVQ_KIND_SYM) && mma_layout_of(t) >= 0 && aligned(t.codes, 16) &&
           aligned(t.kind == RWKVQ_KIND_SB6 ? static_cast<const void*>(t.dev_meta) : static_cast<const void*>(t.qs), 16) && aligned(t.dev_planes, 16);
}
// Whether this kernel takes a product the mma.sync kernel serves too: from that one's second tile of 8 rows on (us at 9 rows,
// mma.sync / this, sb6 4 bits: [2048, 2048] 10.3 / 8.0, [8192, 2048] 14.3 / 12.0, [2048, 8192] 17.5 / 15.1, [2560, 10240] 29.5 / 17.5; at 8
// mma.sync 8.8, 12.6, 17.1 and 21.7).  Up to 8 rows it keeps its main sum in an accumulator without the low terms
// and is the more precise.
constexpr int kSbLeastRows = 9;
bool gemm_sb_pays(const rwkvq_qtensor& t, int N) {
    return tcb_enabled() && gemm_sb_ok(t) && N >= kSbLeastRows;
}

int launch_gemm_sb(const rwkvq_qtensor* ts, int n_mats, const SbRows* rows, int N, float* const* ys, long long ldy, int epilogue,
                   const float* const* resids, float* const* amax_outs, int* status, int force_ks, cudaStream_t s, const Ahead* ahead_or_null) {
    const Ahead none{}, &ahead = ahead_or_null ? *ahead_or_null : none;
    RWKVQ_REQUIRE(n_mats >= 1 && n_mats <= kSbMaxMats, RWKVQ_E_LIMIT, "gemm_sb: %d matrices", n_mats);
    SbArgs a{};
    SbMaps maps;
    // token groups of at most 128, tiles as wide as they need (the tensor time of a stage goes with the width: 100 rows
    // 4.24 -> 4.18 ms per decode step); up to 64 the width is the template's (known to the epilogue: 2.83 against 2.88 ms)
    const int groups = (N + 127) / 128, per = (N + groups - 1) / groups;
    const int nt = per <= 16 ? 16 : per <= 32 ? 32 : per <= 64 ? 64 : (per + 15) / 16 * 16;
    a.nt = nt;
    for (int k = 0; k < n_mats; ++k) {
        RWKVQ_REQUIRE(gemm_sb_ok(ts[k]) && ts[k].kind == ts[0].kind && ts[k].bits == ts[0].bits && ts[k].rows == ts[0].rows &&
                          ts[k].cols == ts[0].cols, RWKVQ_E_SHAPE, "gemm_sb: fused matrices must share layout and shape");
        RWKVQ_REQUIRE(rows[k].hi && rows[k].lo && rows[k].sums && rows[k].unscale && ys[k], RWKVQ_E_NULL, "gemm_sb: x pairs or y is null");
        a.t[k] = make_view(ts[k]);
        a.sums[k] = rows[k].sums; a.unscale[k] = rows[k].unscale; a.y[k] = ys[k];
        a.resid[k] = resids ? resids[k] : nullptr;
        a.amax_out[k] = amax_outs ? amax_outs[k] : nullptr;
        RWKVQ_REQUIRE(epilogue != RWKVQ_EPI_ADD || a.resid[k], RWKVQ_E_NULL, "gemm_sb: resid is null");
        int rc = make_half_map(&maps.hi[k], rows[k].hi, N, ts[0].cols, rows[k].pitch, nt);
        if (rc) return rc;
        rc = make_half_map(&maps.lo[k], rows[k].lo, N, ts[0].cols, rows[k].pitch, nt);
        if (rc) return rc;
        const rwkvq_qtensor& t = ts[k];
        const long long nsb = t.cols / 256;
        const bool sb6 = t.kind == RWKVQ_KIND_SB6, byte_codes = !sb6 && t.bits == 8;
        const int plane_row = sb6 ? (t.bits == 5 ? 32 : t.bits == 6 ? 64 : 0) : (t.bits == 6 ? 64 : 0);
        rc = make_byte_map(&maps.codes[k], t.codes, t.rows, nsb * (byte_codes ? 256 : 128), 128, kGmRows);
        if (rc) return rc;
        rc = make_byte_map(&maps.rec[k], sb6 ? t.dev_meta : t.qs, t.rows, nsb * 16, 16, kGmRows);
        if (rc) return rc;
        if (plane_row) rc = make_byte_map(&maps.planes[k], t.dev_planes, t.rows, nsb * plane_row, plane_row, kGmRows);
        if (rc) return rc;
    }
    a.ldy = ldy; a.n_tokens = N; a.epilogue = epilogue; a.status = status;
    a.row_tiles = (ts[0].rows + kGmRows - 1) / kGmRows;
    a.n_tiles = a.row_tiles * n_mats;
    a.n_sb = ts[0].cols / 256;
    switch (sb_layout_of(ts[0])) {
        case ML_SB6_4: return launch_sb_nt<ML_SB6_4>(a, maps, nt, groups, force_ks, ahead, s);
        case ML_SB6_5: return launch_sb_nt<ML_SB6_5>(a, maps, nt, groups, force_ks, ahead, s);
        case ML_SB6_6: return launch_sb_nt<ML_SB6_6>(a, maps, nt, groups, force_ks, ahead, s);
        case ML_SYM6: return launch_sb_nt<ML_SYM6>(a, maps, nt, groups, force_ks, ahead, s);
        default: return launch_sb_nt<ML_SYM8>(a, maps, nt, groups, force_ks, ahead, s);
    }
}

}  // namespace rwkvq
