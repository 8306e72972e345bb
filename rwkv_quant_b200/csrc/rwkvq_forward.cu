// Whole forward pass over B sequences of T tokens in one call (prefill, speculative verify runs): the
// launch sequence of all layers issued from C, every launch programmatic-dependent.  Issued op by op
// from Python a pass costs 5-8 ms of host time whatever its size; from here ~2 us a launch, which the
// device work hides.
//
// Two regimes by the number of rows N = B * T:
//   N <= 64   fp32-grade small-batch linears (weights read once), operand maxima published by the
//             producers of the rows; the LoRA pair kernels
//   N >  64   fp16 operands on the tensor-core GEMM (rwkvq_gemm_f16.cu): rows scaled to fp16 where they are
//             made, weights and LoRA matrices converted into scratch layer by layer
#include <algorithm>

#include "rwkvq_ahead.cuh"
#include "rwkvq_gemm_f16.cuh"
#include "rwkvq_seq.cuh"
#include "rwkvq_tmix_seq.cuh"
#include "rwkvq_wkv_chunk.cuh"

namespace rwkvq {
namespace {

constexpr int kSmallRows = 64;
constexpr int kChunkedT = 16;        // tokens per sequence from which long calls take the chunked scan (two chunks)

bool chunked(size_t rows, int T) { return rows > kSmallRows && T >= kChunkedT; }
// Shorter calls of many sequences: operands, scan and tail as three launches, whose smaller CTAs fill the chip better than the one
// kernel's (ms, three / one: 1.5B, 32 heads, 44 x 2 tokens 3.81 / 3.75, 50 x 3 3.82 / 3.85, 50 x 9 5.48 / 5.45, 70 x 5 4.97 / 5.21,
// 128 x 2 4.42 / 4.70, 128 x 9 9.26 / 9.61; 2.9B, 40 heads, 36 x 5 6.95 / 7.05, 44 x 9 9.85 / 9.85, 64 x 3 7.17 / 7.43).
constexpr int kSeqPairs = 1600;      // heads of all sequences up to which the one kernel serves
bool three_launches(size_t rows, int B, int T, int H) { return rows > kSmallRows && T < kChunkedT && static_cast<long long>(B) * H > kSeqPairs; }
// Long calls turn every weight matrix into fp16 in front of its product.  Where the scan is long and leaves most of the chip idle, the
// conversions run on the side lane under it, r / k / v and the LoRA matrices a layer ahead: 1.5B, 1 x 512 tokens 6.78 -> 6.35 ms,
// 2 x 256 6.30 -> 5.93, 1 x 256 4.52 -> 4.34 (fp16 rows from the tail, some 0.1 ms, included).  Where it is short (3 x 77: 4.26 -> 4.4 ms,
// also with the conversions of the time mix alone) they outlast it and keep the shared memory that the products behind it
// want; where it fills the chip (16 x 512: 40.4 -> 41.3) there is nothing to run under.
constexpr int kBesideT = 256;        // tokens a sequence from which the scan outlasts a layer's conversions
bool convert_beside(int B, int T, int H) { return chunked(static_cast<size_t>(B) * T, T) && T >= kBesideT && wkv_chunked_f16(B, H); }

struct ForwardWs {
    size_t bytes = 0;
    int* status;
    float *x, *xs, *rkv, *yl, *wkv, *out, *og, *v_first, *amax, *tailx, *taily, *n2tok, *wn2, *hffn, *lora_h, *dp;
    float* scale;                      // [4][N] row scales of the r / k / v (or channel-mix) rows and of og
    float* hscale;                     // [N]
    __half *x16, *og16, *h16, *split, *hl;
    // a layer's weights in fp16, LoRA matrices of this layer and the next: apart where they are converted beside the scan, else in
    // one place in turn
    __half *wrkv16, *wo16, *wfk16, *wfv16, *lw16[2];
    SbRows rkv_pair[3], d_pair, f_pair;      // operand rows of the tcgen05 pipeline (9 to 64 rows): r / k / v; og or xk; hffn
    void* head_ws;
    size_t head_ws_bytes;
};

inline int up64(int n) { return (n + 63) / 64 * 64; }
inline size_t pitch16(size_t cols) { return cols + 64; }

size_t lora16_halves(const rwkvq_model& m) { return static_cast<size_t>(8) * up64(m.max_rank) * up64(m.n_embd); }

ForwardWs carve(const rwkvq_model& m, int B, int T, size_t n_tail, void* base) {
    const size_t N = static_cast<size_t>(B) * T, D = m.n_embd, F = m.ffn_dim;
    ForwardWs w{};
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* p = base ? static_cast<char*>(base) + off : nullptr;
        off += (bytes + 255) / 256 * 256;
        return p;
    };
    auto f32 = [&](size_t n) { return reinterpret_cast<float*>(take(n * sizeof(float))); };
    auto f16 = [&](size_t n) { return reinterpret_cast<__half*>(take(n * sizeof(__half))); };
    w.status = reinterpret_cast<int*>(take(256));
    w.wn2 = f32(static_cast<size_t>(m.n_layer) * 128);
    w.x = f32(N * D); w.rkv = f32(3 * N * D); w.yl = f32(4 * N * D);
    if (three_launches(N, B, T, static_cast<int>(D / 64))) { w.wkv = f32(5 * N * D); w.out = f32(N * D); }
    if (chunked(N, T)) { w.wkv = f32(wkv_chunk_floats(B, T, static_cast<int>(D / 64))); w.dp = f32(N * D / 64); w.out = f32(N * D); }
    w.og = f32(N * D); w.v_first = f32(N * D);
    if (N <= kSmallRows) {
        w.xs = f32(6 * N * D); w.hffn = f32(N * F); w.amax = f32(8 * N);
        w.lora_h = f32(4 * static_cast<size_t>(kSmallRows) * m.max_rank);
        if (D % 256 == 0) {
            auto pair = [&](size_t cols) {
                float* un = f32(N);
                return sb_rows(f16(sb_halves(static_cast<int>(N), static_cast<int>(cols))), un, static_cast<int>(N), static_cast<int>(cols));
            };
            for (int k = 0; k < 3; ++k) w.rkv_pair[k] = pair(D);
            w.d_pair = pair(D);
            w.f_pair = pair(F);
        }
    } else {
        w.x16 = f16(3 * N * pitch16(D)); w.og16 = f16(N * pitch16(D)); w.h16 = f16(N * pitch16(F));
        w.split = f16(4 * N * 2 * D); w.hl = f16(4 * N * 2 * up64(m.max_rank));
        w.scale = f32(4 * N); w.hscale = f32(N); w.n2tok = f32(N);
        const bool apart = convert_beside(B, T, static_cast<int>(D / 64));
        w.wrkv16 = f16(apart ? 3 * D * D : std::max(3 * D * D, F * D));
        w.wo16 = apart ? f16(D * D) : w.wrkv16; w.wfk16 = apart ? f16(F * D) : w.wrkv16; w.wfv16 = apart ? f16(F * D) : w.wrkv16;
        w.lw16[0] = f16(lora16_halves(m));
        w.lw16[1] = apart ? f16(lora16_halves(m)) : w.lw16[0];
    }
    if (n_tail > 0) {
        w.tailx = f32(n_tail * D); w.taily = f32(n_tail * D);
        w.head_ws_bytes = n_tail <= 2 ? 0 : n_tail <= kSmallRows ? gemv_batch_rows_bytes(m.head, static_cast<int>(n_tail))
                                                                : gemm_rows_bytes(m.head, static_cast<int>(n_tail));
        w.head_ws = take(w.head_ws_bytes);
    }
    w.bytes = off;
    return w;
}

bool fp16_gemm_ok(const rwkvq_qtensor& t) { return t.kind == RWKVQ_KIND_SB6 || t.kind == RWKVQ_KIND_SYM; }

// One linear of the small regime; scale: max|x| per row (null: measured by a pre-pass into amax_scratch)
int small_linear(const rwkvq_qtensor* const* ts, int n_mats, const float* const* xs, const float* const* amax, int N, int in, float* const* ys,
                 int out, int epi, const float* resid, float* amax_out, cudaStream_t s, const Ahead* ahead = nullptr) {
    if (N <= 2) {
        for (int k = 0; k < n_mats; ++k) {
            int rc = rwkvq_gemv(ts[k], xs[k], RWKVQ_F32, N, in, ys[k], out, epi, resid, s);
            if (rc) return rc;
        }
        return RWKVQ_OK;
    }
    rwkvq_qtensor t[kHgMaxProbs];
    const void* xv[kHgMaxProbs];
    const float* rs[kHgMaxProbs];
    float* ao[kHgMaxProbs];
    for (int k = 0; k < n_mats; ++k) { t[k] = *ts[k]; xv[k] = xs[k]; rs[k] = resid; ao[k] = amax_out; }
    return launch_gemv_batch(t, n_mats, xv, false, amax, N, in, ys, out, epi, rs, ao, s, ahead);
}

bool same_shape(const rwkvq_qtensor& a, const rwkvq_qtensor& b) {
    return a.kind == b.kind && a.bits == b.bits && a.rows == b.rows && a.cols == b.cols && mma_layout_of(a) == mma_layout_of(b);
}

constexpr int kForkRows = 1024;
constexpr int kBesideCtas = 3;       // CTAs an SM of a conversion beside the scan

struct Pass {
    const rwkvq_model& m;
    const ForwardWs& w;
    int B, T, N, D, F, H;
    cudaStream_t s;

    HgProb prob(const __half* w16, int rows, int cols, const __half* x16, const float* row_scale) const {
        HgProb p{};
        p.w = w16; p.w_pitch = cols; p.rows = rows; p.k = cols; p.terms = 1;
        p.x = x16; p.x_pitch = static_cast<long long>(pitch16(cols)); p.row_scale = row_scale;
        return p;
    }

    // matrices of layer l to fp16
    int convert_rkv(int l, cudaStream_t s, int per_sm) const {
        const rwkvq_layer& L = m.layers[l];
        const rwkvq_qtensor* t3[3] = {&L.Wr, &L.Wk, &L.Wv};
        for (int k = 0; k < 3; ++k) {
            int rc = launch_dequant_f16(*t3[k], 0, D, w.wrkv16 + static_cast<size_t>(k) * D * D, nullptr, s, per_sm);
            if (rc) return rc;
        }
        return RWKVQ_OK;
    }
    int convert_lora(int l, cudaStream_t s) const {
        const rwkvq_layer& L = m.layers[l];
        const rwkvq_qtensor* t12[8] = {&L.w1, &L.w2, &L.a1, &L.a2, &L.g1, &L.g2, &L.v1, &L.v2};
        TransposeJob jobs[8];
        const int n = l == 0 ? 6 : 8;
        __half* o = w.lw16[l & 1];
        for (int i = 0; i < n; ++i) {
            jobs[i] = {t12[i], o};
            o += i & 1 ? static_cast<size_t>(D) * up64(t12[i]->rows) : static_cast<size_t>(t12[i]->cols) * up64(D);
        }
        return launch_dequant_f16_t(jobs, n, s);
    }
    int rkv_large(float* const* y3, cudaStream_t s) const {
        const size_t NP = static_cast<size_t>(N) * pitch16(D);
        HgProb p[kHgMaxProbs];
        for (int k = 0; k < 3; ++k) {
            p[k] = prob(w.wrkv16 + static_cast<size_t>(k) * D * D, D, D, w.x16 + k * NP, w.scale + k * N);
            p[k].out = HG_F32; p[k].epilogue = RWKVQ_EPI_NONE; p[k].y32 = y3[k]; p[k].ldy = D;
        }
        return launch_gemm_f16(p, 3, N, w.status, s);
    }
    // LoRA branches: both products with x (then h) as an fp16 pair, the matrices exact in fp16
    int lora_large(int l) const {
        const rwkvq_layer& L = m.layers[l];
        const size_t ND = static_cast<size_t>(N) * D;
        const rwkvq_qtensor* t1[4] = {&L.w1, &L.a1, &L.g1, &L.v1};
        const int act[4] = {1, 0, 2, 0}, n_br = l == 0 ? 3 : 4;
        HgProb dn[kHgMaxProbs], up[kHgMaxProbs];
        __half* o = w.lw16[l & 1];
        const int Rp = up64(m.max_rank);
        for (int i = 0; i < n_br; ++i) {
            const int r = t1[i]->cols, rp = up64(r);
            __half* hl = w.hl + static_cast<size_t>(i) * N * 2 * Rp;
            dn[i] = HgProb{};
            dn[i].w = o; dn[i].w_pitch = up64(D); dn[i].rows = rp; dn[i].w_rows = r; dn[i].k = D; dn[i].terms = 2;
            dn[i].x = w.split + static_cast<size_t>(i) * N * 2 * D; dn[i].x_pitch = 2 * D;
            dn[i].out = HG_SPLIT; dn[i].act = act[i]; dn[i].y16 = hl; dn[i].ldy = 2 * rp; dn[i].lo_off = rp;
            o += static_cast<size_t>(r) * up64(D);
            up[i] = HgProb{};
            up[i].w = o; up[i].w_pitch = rp; up[i].rows = D; up[i].k = rp; up[i].terms = 2;
            up[i].x = hl; up[i].x_pitch = 2 * rp;
            up[i].out = HG_F32; up[i].epilogue = RWKVQ_EPI_NONE; up[i].y32 = w.yl + i * ND; up[i].ldy = D;
            o += static_cast<size_t>(D) * rp;
        }
        int rc = launch_gemm_f16(dn, n_br, N, w.status, s);
        if (rc) return rc;
        return launch_gemm_f16(up, n_br, N, w.status, s);
    }
};

}  // namespace
}  // namespace rwkvq

using namespace rwkvq;

extern "C" {

int rwkvq_forward_seq_ok(const rwkvq_model* m, int64_t n_rows) {
    if (!m || !m->layers || n_rows < 2 || n_rows >= (1ll << 31) / 64) return 0;
    if (m->head_size != 64 || m->n_embd % 128 != 0 || m->n_embd > 4096 || m->ffn_dim % 256 != 0 || m->ffn_dim > 32768) return 0;
    const bool small = n_rows <= kSmallRows;
    const int D = m->n_embd, F = m->ffn_dim;
    // sizes of the scratch and of every launch follow from the model's dimensions: the tensors must have them too
    auto linear_ok = [&](const rwkvq_qtensor& t, int rows, int cols) {
        return t.rows == rows && t.cols == cols && mma_layout_of(t) >= 0 && (small || fp16_gemm_ok(t));
    };
    for (int l = 0; l < m->n_layer; ++l) {
        const rwkvq_layer& L = m->layers[l];
        for (const rwkvq_qtensor* t : {&L.Wr, &L.Wk, &L.Wv, &L.Wo})
            if (!linear_ok(*t, D, D)) return 0;
        if (!linear_ok(L.Wfk, F, D) || !linear_ok(L.Wfv, D, F)) return 0;
        const rwkvq_qtensor* t1[4] = {&L.w1, &L.a1, &L.g1, &L.v1};
        const rwkvq_qtensor* t2[4] = {&L.w2, &L.a2, &L.g2, &L.v2};
        if (!lora_mma_ok(t1, t2, l == 0 ? 3 : 4, D) || t2[0]->cols != D) return 0;
        for (int i = 0; i < (l == 0 ? 3 : 4); ++i)
            if (t1[i]->cols > m->max_rank) return 0;
    }
    return m->emb.cols == D && m->head.rows == m->vocab_size && m->head.cols == D && mma_layout_of(m->head) >= 0 && fp16_gemm_ok(m->head) ? 1 : 0;
}

size_t rwkvq_forward_seq_workspace_bytes(const rwkvq_model* m, int B, int T, int tail) {
    if (!m || B < 1 || T < 1 || tail < 0 || tail > T) return 0;
    return carve(*m, B, T, static_cast<size_t>(B) * tail, nullptr).bytes;
}

int rwkvq_forward_seq(const rwkvq_model* m, int B, int T, const int64_t* tokens, const float* const* wkv_in, const float* const* tshift_in,
                      const float* const* cshift_in, float* const* wkv_out, float* const* tshift_out, float* const* cshift_out, int tail,
                      float* hidden, float* logits, void* workspace, size_t workspace_bytes, void* stream) {
    return rwkvq_forward_seq_status(m, B, T, tokens, wkv_in, tshift_in, cshift_in, wkv_out, tshift_out, cshift_out, tail, hidden, logits, nullptr,
                                    workspace, workspace_bytes, stream);
}

int rwkvq_forward_seq_status(const rwkvq_model* m, int B, int T, const int64_t* tokens, const float* const* wkv_in, const float* const* tshift_in,
                      const float* const* cshift_in, float* const* wkv_out, float* const* tshift_out, float* const* cshift_out, int tail,
                      float* hidden, float* logits, int32_t* status, void* workspace, size_t workspace_bytes, void* stream) {
    RWKVQ_REQUIRE(m && m->layers && tokens && wkv_in && tshift_in && cshift_in && wkv_out && tshift_out && cshift_out && workspace,
                  RWKVQ_E_NULL, "rwkvq_forward_seq: null pointer");
    RWKVQ_REQUIRE(B >= 1 && T >= 1 && tail >= 0 && tail <= T, RWKVQ_E_SHAPE, "rwkvq_forward_seq: B=%d T=%d tail=%d", B, T, tail);
    RWKVQ_REQUIRE(tail == 0 || logits, RWKVQ_E_NULL, "rwkvq_forward_seq: logits is null");
    const int64_t rows64 = static_cast<int64_t>(B) * T;
    RWKVQ_REQUIRE(rwkvq_forward_seq_ok(m, rows64), RWKVQ_E_DTYPE,
                  "rwkvq_forward_seq: a tensor's layout or shape has no one-call path for %lld rows (rwkvq_forward_seq_ok)", (long long)rows64);
    for (int l = 0; l < m->n_layer; ++l) {
        const rwkvq_layer& L = m->layers[l];
        for (const rwkvq_qtensor* t : {&L.Wr, &L.Wk, &L.Wv, &L.Wo, &L.Wfk, &L.Wfv, &L.w1, &L.w2, &L.a1, &L.a2, &L.g1, &L.g2}) {
            int rc = validate_qtensor(t, "rwkvq_forward_seq");
            if (rc) return rc;
        }
        for (const rwkvq_qtensor* t : {&L.v1, &L.v2}) {
            int rc = l == 0 ? RWKVQ_OK : validate_qtensor(t, "rwkvq_forward_seq");
            if (rc) return rc;
        }
    }
    for (int l = 0; l < m->n_layer; ++l)
        RWKVQ_REQUIRE(wkv_out[l] && tshift_out[l] && cshift_out[l], RWKVQ_E_NULL, "rwkvq_forward_seq: a state of layer %d has nowhere to go", l);
    for (int l = 0; l < m->n_layer; ++l)
        for (const float* p : {wkv_in[l], tshift_in[l], cshift_in[l], const_cast<const float*>(wkv_out[l]),
                               const_cast<const float*>(tshift_out[l]), const_cast<const float*>(cshift_out[l])})
            RWKVQ_REQUIRE(aligned(p, 16), RWKVQ_E_ALIGN, "rwkvq_forward_seq: the states of layer %d must be 16-byte aligned", l);
    int head_rc = validate_qtensor(&m->head, "rwkvq_forward_seq");
    if (head_rc) return head_rc;
    ForwardWs w = carve(*m, B, T, static_cast<size_t>(B) * tail, workspace);
    RWKVQ_REQUIRE(workspace_bytes >= w.bytes && aligned(workspace, 256), RWKVQ_E_LIMIT,
                  "rwkvq_forward_seq: workspace %zu of %zu bytes, 256-byte aligned", workspace_bytes, w.bytes);
    const int N = static_cast<int>(rows64), D = m->n_embd, F = m->ffn_dim, H = D / 64;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const size_t ND = static_cast<size_t>(N) * D, NP = static_cast<size_t>(N) * pitch16(D);
    const bool small = N <= kSmallRows;
    Pass ps{*m, w, B, T, N, D, F, H, s};
    // the status word and every layer's norm bounds (merged by atomic max)
    if (cudaMemsetAsync(w.status, 0, 256 + sizeof(float) * 128 * m->n_layer, s) != cudaSuccess) return check_launch("rwkvq_forward_seq(memset)");
    if (status) w.status = status;
    int rc = rwkvq_seq_embed_ln0(&m->emb, tokens, m->ln0_w, m->ln0_b, w.x, N, D, stream);
    if (rc) return rc;
    // r / k / v beside the LoRA branches while neither fills the chip (5 rows 2.07 -> 2.00 ms, 231 rows 4.46 -> 4.30,
    // 512 rows 6.93 -> 6.78, 1024 rows 8.73 -> 8.58)
    SideLane* lane = side_lane(s);
    const cudaStream_t s_side = lane ? lane->stream : s, s_rkv = N <= kForkRows ? s_side : s;
    const bool beside = lane && convert_beside(B, T, H);
    if (beside && ((rc = ps.convert_rkv(0, s, 0)) != 0 || (rc = ps.convert_lora(0, s)) != 0)) return rc;
    Fork fork{lane, s};
    for (int l = 0; l < m->n_layer; ++l) {
        const rwkvq_layer& L = m->layers[l];
        const bool layer0 = l == 0;
        float *am_og = small ? w.amax + 6 * N : nullptr, *am_h = small ? w.amax + 7 * N : nullptr;
        float *r = w.rkv, *k = w.rkv + ND, *v = w.rkv + 2 * ND;
        if (layer0) v = w.v_first;                           // layer 0's values are the residual of all others
        float* y3[3] = {r, k, v};
        float *yw = w.yl, *ya = w.yl + ND, *yg = w.yl + 2 * ND, *yv = w.yl + 3 * ND;
        SeqPrepArgs a{};
        a.x = w.x; a.ln_w = L.ln1_w; a.ln_b = L.ln1_b; a.shift_in = tshift_in[l]; a.mix = L.x_mix; a.shift_out = tshift_out[l];
        a.T = T; a.D = D; a.n_mix = 6;
        // mix rows: r, w, k, v, a, g
        const bool sb = small && D % 256 == 0 && same_shape(L.Wr, L.Wk) && same_shape(L.Wr, L.Wv) && gemm_sb_pays(L.Wr, N) &&
                        gemm_sb_pays(L.Wo, N) && gemm_sb_pays(L.Wfk, N) && gemm_sb_pays(L.Wfv, N);
        const LayerAhead ahead(L, l + 1 < m->n_layer ? &L + 1 : nullptr, layer0, wkv_in[l], static_cast<size_t>(B) * D * 64 * sizeof(float));
        if (small) {
            for (int q = 0; q < 6; ++q) {
                a.f32[q] = w.xs + q * ND; a.scale[q] = w.amax + q * N;
                a.mode[q] = kPrepF32 | ((q == 0 || q == 2 || q == 3) ? kPrepAmax : 0);
            }
            if (sb) {
                const int lin[3] = {0, 2, 3};
                for (int q = 0; q < 3; ++q) { a.pair[lin[q]] = w.rkv_pair[q]; a.mode[lin[q]] = kPrepPair | (q == 2 && !layer0 ? kPrepF32 : 0); }
            } else {
                a.zero_a = am_og;
                a.zero_b = am_h;
            }
            rc = launch_seq_prep(a, N, s);
            if (rc) return rc;
            if ((rc = fork.start()) != 0) return rc;
            const rwkvq_qtensor* t3[3] = {&L.Wr, &L.Wk, &L.Wv};
            const float* x3[3] = {w.xs, w.xs + 2 * ND, w.xs + 3 * ND};
            const float* a3[3] = {w.amax, w.amax + 2 * N, w.amax + 3 * N};
            if (sb) {
                const rwkvq_qtensor three[3] = {L.Wr, L.Wk, L.Wv};
                rc = launch_gemm_sb(three, 3, w.rkv_pair, N, y3, D, RWKVQ_EPI_NONE, nullptr, nullptr, w.status, 0, s_rkv, &ahead.rkv);
            } else if (same_shape(L.Wr, L.Wk) && same_shape(L.Wr, L.Wv)) {
                rc = small_linear(t3, 3, x3, a3, N, D, y3, D, RWKVQ_EPI_NONE, nullptr, nullptr, s_rkv, &ahead.rkv);
            } else {
                for (int q = 0; q < 3 && !rc; ++q) rc = small_linear(t3 + q, 1, x3 + q, a3 + q, N, D, y3 + q, D, RWKVQ_EPI_NONE, nullptr, nullptr, s_rkv);
            }
            if (rc) return rc;
            const rwkvq_qtensor* t1[4] = {&L.w1, &L.a1, &L.g1, &L.v1};
            const rwkvq_qtensor* t2[4] = {&L.w2, &L.a2, &L.g2, &L.v2};
            const float* x4[4] = {w.xs + ND, w.xs + 4 * ND, w.xs + 5 * ND, w.xs + 3 * ND};
            float* y4[4] = {yw, ya, yg, yv};
            const int act[4] = {1, 0, 2, 0};
            rc = launch_lora_pair_mma(t1, t2, x4, y4, act, layer0 ? 3 : 4, N, D, m->max_rank, w.lora_h, kSmallRows, s);
        } else {
            const int lin[3] = {0, 2, 3}, lora[4] = {1, 4, 5, 3};
            for (int q = 0; q < 3; ++q) {
                a.mode[lin[q]] = kPrepScaled;
                a.x16[lin[q]] = w.x16 + q * NP; a.scale[lin[q]] = w.scale + q * N;
            }
            for (int q = 0; q < (layer0 ? 3 : 4); ++q) {
                a.mode[lora[q]] |= kPrepSplit;
                a.split[lora[q]] = w.split + static_cast<size_t>(q) * 2 * ND;
            }
            rc = launch_seq_prep(a, N, s);
            if (rc) return rc;
            if (beside && (rc = fork.wait()) != 0) return rc;
            if (s_rkv != s && (rc = fork.start()) != 0) return rc;
            if (!beside && (rc = ps.convert_rkv(l, s_rkv, 0)) != 0) return rc;
            if ((rc = ps.rkv_large(y3, s_rkv)) != 0) return rc;
            if (s_rkv == s && beside && (rc = fork.start()) != 0) return rc;
            if (!beside && (rc = ps.convert_lora(l, s)) != 0) return rc;
            rc = ps.lora_large(l);
        }
        if (rc) return rc;
        if (!beside) {
            if ((rc = fork.join()) != 0) return rc;
        } else {
            if (s_rkv != s && ((rc = fork.mark()) != 0 || (rc = fork.wait()) != 0)) return rc;
            if ((rc = launch_dequant_f16(L.Wo, 0, D, w.wo16, nullptr, s_side, kBesideCtas)) != 0) return rc;
            if ((rc = fork.mark()) != 0) return rc;
        }
        if (chunked(N, T)) {
            WkvChunkArgs q{};
            q.r = r; q.k = k; q.v = v; q.yw = yw; q.ya = ya; q.yv = layer0 ? nullptr : yv; q.v_first = layer0 ? nullptr : w.v_first; q.g = yg;
            q.w0 = L.w0; q.a0 = L.a0; q.v0 = L.v0; q.k_k = L.k_k; q.k_a = L.k_a; q.r_k = L.r_k; q.ln_w = L.lnx_w; q.ln_b = L.lnx_b;
            q.h_in = wkv_in[l]; q.h_out = wkv_out[l]; q.og = w.og; q.og16 = w.og16; q.og_scale = w.scale + 3 * N;
            q.og_pitch = static_cast<long long>(pitch16(D)); q.ops = w.wkv; q.dp = w.dp; q.spread = beside; q.y = w.out; q.status = w.status;
            q.B = B; q.T = T; q.H = H;
            rc = launch_wkv_chunked(q, s);
            if (rc) return rc;
        } else if (three_launches(N, B, T, H)) {
            float *dw = w.wkv, *k2 = w.wkv + ND, *v2 = w.wkv + 2 * ND, *na = w.wkv + 3 * ND, *nb = w.wkv + 4 * ND;
            rc = rwkvq_seq_tmix_pre(k, v, yw, ya, layer0 ? nullptr : yv, layer0 ? nullptr : w.v_first, L.w0, L.a0, L.v0, L.k_k, L.k_a, dw,
                                    k2, v2, na, nb, N, H, stream);
            if (rc) return rc;
            rc = rwkvq_wkv7(r, dw, k2, v2, na, nb, wkv_in[l], w.out, wkv_out[l], B, T, H, 64, stream);
            if (rc) return rc;
            rc = rwkvq_wkv_tail(w.out, r, k2, v2, L.r_k, L.lnx_w, L.lnx_b, yg, w.og, N, H, 64, 64e-5f, stream);
            if (rc) return rc;
        } else {
            TmixSeqArgs q{};
            q.r = r; q.k = k; q.v = v; q.yw = yw; q.ya = ya; q.yv = layer0 ? nullptr : yv; q.v_first = layer0 ? nullptr : w.v_first; q.g = yg;
            q.w0 = L.w0; q.a0 = L.a0; q.v0 = L.v0; q.k_k = L.k_k; q.k_a = L.k_a; q.r_k = L.r_k; q.ln_w = L.lnx_w; q.ln_b = L.lnx_b;
            q.h_in = wkv_in[l]; q.h_out = wkv_out[l]; q.og = w.og; q.og_amax = sb ? nullptr : am_og;
            q.B = B; q.T = T; q.H = H;
            rc = launch_tmix_seq(q, s);
            if (rc) return rc;
        }
        // ---- output projection, channel mix
        SeqPrepArgs c{};
        c.x = w.x; c.ln_w = L.ln2_w; c.ln_b = L.ln2_b; c.shift_in = cshift_in[l]; c.mix = L.ffn_x_k; c.shift_out = cshift_out[l];
        c.T = T; c.D = D; c.n_mix = 1;
        if (sb) {
            const float* res[1] = {w.x};
            float *yx[1] = {w.x}, *yh[1] = {w.hffn};
            rc = launch_split_rows(w.og, D, D, N, w.d_pair, nullptr, s);
            if (rc) return rc;
            rc = launch_gemm_sb(&L.Wo, 1, &w.d_pair, N, yx, D, RWKVQ_EPI_ADD, res, nullptr, w.status, 0, s);
            if (rc) return rc;
            c.mode[0] = kPrepPair; c.pair[0] = w.d_pair;
            rc = launch_seq_prep(c, N, s);
            if (rc) return rc;
            rc = launch_gemm_sb(&L.Wfk, 1, &w.d_pair, N, yh, F, RWKVQ_EPI_RELU2, nullptr, nullptr, w.status, 0, s, &ahead.key);
            if (rc) return rc;
            rc = launch_split_rows(w.hffn, F, F, N, w.f_pair, nullptr, s);
            if (rc) return rc;
            rc = launch_gemm_sb(&L.Wfv, 1, &w.f_pair, N, yx, D, RWKVQ_EPI_ADD, res, nullptr, w.status, 0, s);
            if (rc) return rc;
            continue;
        }
        if (small) {
            const rwkvq_qtensor *to[1] = {&L.Wo}, *tk[1] = {&L.Wfk}, *tv[1] = {&L.Wfv};
            const float *xo[1] = {w.og}, *ao[1] = {am_og}, *xk[1] = {w.xs}, *ak[1] = {w.amax}, *xv[1] = {w.hffn}, *av[1] = {am_h};
            float *yx[1] = {w.x}, *yh[1] = {w.hffn};
            rc = small_linear(to, 1, xo, ao, N, D, yx, D, RWKVQ_EPI_ADD, w.x, nullptr, s);
            if (rc) return rc;
            c.mode[0] = kPrepF32 | kPrepAmax; c.f32[0] = w.xs; c.scale[0] = w.amax;
            rc = launch_seq_prep(c, N, s);
            if (rc) return rc;
            rc = small_linear(tk, 1, xk, ak, N, D, yh, F, RWKVQ_EPI_RELU2, nullptr, am_h, s, &ahead.key);
            if (rc) return rc;
            rc = small_linear(tv, 1, xv, av, N, F, yx, D, RWKVQ_EPI_ADD, w.x, nullptr, s);
            if (rc) return rc;
            continue;
        }
        if (!beside && (rc = launch_dequant_f16(L.Wo, 0, D, w.wo16, nullptr, s)) != 0) return rc;
        if (!(chunked(N, T) && wkv_chunked_f16(B, H))) {
            rc = launch_row_scale(w.og, D, D, N, w.scale + 3 * N, w.og16, static_cast<long long>(pitch16(D)), nullptr, s);
            if (rc) return rc;
        }
        if (beside && (rc = fork.wait()) != 0) return rc;
        HgProb p = ps.prob(w.wo16, D, D, w.og16, w.scale + 3 * N);
        p.out = HG_F32; p.epilogue = RWKVQ_EPI_ADD; p.y32 = w.x; p.resid = w.x; p.ldy = D;
        rc = launch_gemm_f16(&p, 1, N, w.status, s);
        if (rc) return rc;
        float* wn2 = w.wn2 + static_cast<size_t>(l) * 128;
        if (beside) {
            if ((rc = launch_dequant_f16(L.Wfk, 0, F, w.wfk16, wn2, s_side, kBesideCtas)) != 0) return rc;
            if ((rc = launch_dequant_f16(L.Wfv, 0, D, w.wfv16, nullptr, s_side, kBesideCtas)) != 0) return rc;
        }
        c.mode[0] = kPrepScaled; c.x16[0] = w.x16; c.scale[0] = w.scale; c.n2 = w.n2tok;
        rc = launch_seq_prep(c, N, s);
        if (rc) return rc;
        if (beside) {
            if ((rc = fork.mark()) != 0 || (rc = fork.wait()) != 0) return rc;
            if (l + 1 < m->n_layer && ((rc = ps.convert_rkv(l + 1, s_side, kBesideCtas)) != 0 || (rc = ps.convert_lora(l + 1, s_side)) != 0 ||
                                       (rc = fork.mark()) != 0))
                return rc;                                   // waited for in front of the next layer's products
        } else if ((rc = launch_dequant_f16(L.Wfk, 0, F, w.wfk16, wn2, s)) != 0) {
            return rc;
        }
        p = ps.prob(w.wfk16, F, D, w.x16, w.scale);
        p.out = HG_RELU2_F16; p.y16 = w.h16; p.ldy = static_cast<long long>(pitch16(F)); p.w_n2 = wn2; p.n_w_n2 = D / 256; p.x_n2 = w.n2tok;
        p.out_scale = w.hscale;
        rc = launch_gemm_f16(&p, 1, N, w.status, s);
        if (rc) return rc;
        if (!beside && (rc = launch_dequant_f16(L.Wfv, 0, D, w.wfv16, nullptr, s)) != 0) return rc;
        p = ps.prob(w.wfv16, D, F, w.h16, w.hscale);
        p.out = HG_F32; p.epilogue = RWKVQ_EPI_ADD; p.y32 = w.x; p.resid = w.x; p.ldy = D;
        rc = launch_gemm_f16(&p, 1, N, w.status, s);
        if (rc) return rc;
    }
    if (hidden) {
        rc = rwkvq_seq_layer_norm(w.x, m->lnout_w, m->lnout_b, hidden, N, D, stream);
        if (rc) return rc;
    }
    if (tail > 0) {
        const int n = B * tail, V = m->vocab_size;
        const size_t row = sizeof(float) * D;
        if (cudaMemcpy2DAsync(w.tailx, tail * row, w.x + static_cast<size_t>(T - tail) * D, T * row, tail * row, B, cudaMemcpyDeviceToDevice,
                              s) != cudaSuccess)
            return check_launch("rwkvq_forward_seq(tail)");
        rc = rwkvq_seq_layer_norm(w.tailx, m->lnout_w, m->lnout_b, w.taily, n, D, stream);
        if (rc) return rc;
        if (n <= 2) rc = rwkvq_gemv(&m->head, w.taily, RWKVQ_F32, n, D, logits, V, RWKVQ_EPI_NONE, nullptr, stream);
        else if (n <= kSmallRows) rc = launch_gemv_batch_rows(m->head, w.taily, n, D, logits, V, RWKVQ_EPI_NONE, nullptr, w.head_ws, w.status, nullptr, s);
        else rc = launch_gemm_rows(m->head, w.taily, n, D, logits, V, RWKVQ_EPI_NONE, nullptr, w.head_ws, w.status, nullptr, s);
        if (rc) return rc;
    }
    return check_launch("rwkvq_forward_seq");
}

}  // extern "C"
