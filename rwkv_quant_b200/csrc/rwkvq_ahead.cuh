// Memory that a launch of the decode chain brings into L2 for the launches behind it.
//
// The chain is a series of short dependent kernels: one stream reads 34 MB of weights a layer in 39 us, a seventh of the HBM
// rate, and each linear still waits for DRAM when it starts, since its CTAs become resident only as those of the
// kernel before leave.  A linear therefore asks L2 (126 MB) for the weights of the linears behind it while it runs its own:
// one cp.async.bulk.prefetch.L2 per region and CTA, whose bytes no SM ever sees.
#pragma once
#include <algorithm>

#include "rwkvq_gemv_mma.cuh"

namespace rwkvq {

constexpr int kAheadRegions = 32;            // a lane each
// Weights and WKV state of a layer, together, up to which they are asked for: somewhat more than half of L2.  What has to stay there
// until it is used is then thrown out by what flows through.  us a step without / with (MiB of a layer with one stream, and more a stream):
//   1.5B compression (31.6, 0.5)  1 stream 908 / 906, 13 1777 / 1727, 32 2000 / 1966, 64 2480 / 2441, 72 2944 / 2946, 80 3021 / 3043, 128 3622 / 3636
//   1.5B reduction   (46.0, 0.5)  1 1074 / 1082, 13 1728 / 1686, 32 1966 / 1964, 48 2336 / 2341, 72 2930 / 2964, 128 3589 / 3655
//   2.9B compression (48.9, 0.6)  1 1658 / 1557, 13 3003 / 2923, 32 3509 / 3451, 40 4054 / 4056, 64 4288 / 4355, 128 6486 / 6577
//   2.9B reduction   (71.4, 0.6)  1 1610 / 1633, 13 2912 / 2937, 32 3398 / 3411, 64 4203 / 4330, 128 6468 / 6652
// Steps of 2 to 8 streams, on the mma.sync kernel beside the LoRA pair, ask for nothing (without / with, 1.5B compression 2 streams 1600 /
// 1617, 4 1623 / 1635, reduction 1632 / 1654, 1662 / 1677, 2.9B 2645 / 2689, 2701 / 2699); its forward calls do (1.5B 5 drafts 1930 / 1908).
constexpr size_t kAheadMost = 70u << 20;

struct Ahead {
    const unsigned char* p[kAheadRegions];
    unsigned n[kAheadRegions];               // bytes, multiples of 16
    int count;
};

__host__ inline void ahead_region(Ahead& a, const void* p, size_t bytes) {
    if (p == nullptr || !aligned(p, 16) || a.count >= kAheadRegions || bytes < 16) return;
    a.p[a.count] = static_cast<const unsigned char*>(p);
    a.n[a.count++] = static_cast<unsigned>(std::min<size_t>(bytes, 1u << 30) & ~size_t(15));
}
// the streams that the kernels of the decode step read of a linear's tensor, or of a LoRA matrix
__host__ inline void ahead_tensor(Ahead& a, const rwkvq_qtensor& t) {
    const size_t n = static_cast<size_t>(t.rows) * t.cols;
    if (t.kind == RWKVQ_KIND_SB6) {
        if (mma_layout_of(t) < 0) return;
        ahead_region(a, t.codes, n / 2);
        ahead_region(a, t.dev_meta, n / 16);
        if (t.bits > 4) ahead_region(a, t.dev_planes, t.bits == 5 ? n / 8 : n / 4);
    } else if (t.kind == RWKVQ_KIND_SYM) {
        if (mma_layout_of(t) < 0) return;
        ahead_region(a, t.codes, t.bits == 8 ? n : n / 2);
        if (t.bits == 6) ahead_region(a, t.dev_planes, n / 4);
        ahead_region(a, t.qs, n / 16);
        ahead_region(a, t.d, n / 256 * sizeof(__half));
    } else if (t.kind == RWKVQ_KIND_ASYM) {
        const size_t blocks = static_cast<size_t>(t.rows) * ((t.cols + t.gs - 1) / t.gs);
        ahead_region(a, t.codes, n);
        ahead_region(a, t.scale, blocks * sizeof(float));
        ahead_region(a, t.mn, blocks * sizeof(float));
    } else if (t.kind == RWKVQ_KIND_RTN && t.bits > 4) {
        ahead_region(a, t.codes, n);
    }
}

// Whether a layer's descriptors describe its tensors: what is refused where its turn comes must not be asked for before.
inline bool ahead_layer_ok(const rwkvq_layer& L, int D, int F, bool layer0) {
    auto ok = [](const rwkvq_qtensor& t, int rows, int cols) { return t.rows == rows && t.cols == cols && validate_qtensor(&t, "ahead") == RWKVQ_OK; };
    auto pair = [&](const rwkvq_qtensor& t1, const rwkvq_qtensor& t2) { return ok(t1, D, t1.cols) && ok(t2, t1.cols, D); };
    return ok(L.Wr, D, D) && ok(L.Wk, D, D) && ok(L.Wv, D, D) && ok(L.Wo, D, D) && ok(L.Wfk, F, D) && ok(L.Wfv, D, F) && pair(L.w1, L.w2) &&
           pair(L.a1, L.a2) && pair(L.g1, L.g2) && (layer0 || pair(L.v1, L.v2));
}

// What a layer's launches ask for: its r / k / v launch the state, the LoRA up matrices, the output projection and the ffn key, its
// ffn key the ffn value and the r / k / v and LoRA down matrices of the layer behind it (null: none).
struct LayerAhead {
    Ahead rkv{}, key{};
    LayerAhead() = default;
    LayerAhead(const rwkvq_layer& L, const rwkvq_layer* behind, bool layer0, const float* state, size_t state_bytes) {
        ahead_region(rkv, state, state_bytes);
        for (const rwkvq_qtensor* t : {&L.w2, &L.a2, &L.g2}) ahead_tensor(rkv, *t);
        if (!layer0) ahead_tensor(rkv, L.v2);
        ahead_tensor(rkv, L.Wo);
        ahead_tensor(rkv, L.Wfk);
        ahead_tensor(key, L.Wfv);
        if (behind)
            for (const rwkvq_qtensor* t : {&behind->Wr, &behind->Wk, &behind->Wv, &behind->w1, &behind->a1, &behind->g1, &behind->v1}) ahead_tensor(key, *t);
        size_t all = 0;
        for (int i = 0; i < rkv.count; ++i) all += rkv.n[i];
        for (int i = 0; i < key.count; ++i) all += key.n[i];
        if (all > kAheadMost) rkv.count = key.count = 0;
    }
};

// Called by one whole warp of every CTA: its share of each region, whole 128-byte lines
__device__ __forceinline__ void ahead_prefetch(const Ahead& a, unsigned cta, unsigned ctas) {
    const int r = threadIdx.x & 31;
    if (r >= a.count) return;
    const unsigned n = a.n[r], share = ((n + ctas - 1) / ctas + 127u) & ~127u;
    const unsigned long long off = static_cast<unsigned long long>(share) * cta;
    if (off >= n) return;
    const unsigned mine = min(share, n - static_cast<unsigned>(off));
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a.p[r] + off), "r"(mine) : "memory");
}

}  // namespace rwkvq
