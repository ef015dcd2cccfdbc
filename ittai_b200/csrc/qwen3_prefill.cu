// Host side of the Qwen3 prefill: the whole layer stack queued by one call.  A layer is six or seven launches of a few
// microseconds each at short prompts; issued one by one through the binding they cost 15-20 us of host time apiece, which is
// what a short prefill then took, and a CUDA graph instead has to be captured per shape.  Here a launch is its tensor maps
// and a cudaLaunchKernelEx.
#include <cuda_runtime.h>

#include "../../include/ittai_b200.h"
#include "gemm_split.h"
#include "qwen3_short.h"

namespace ittai {

void set_error(const char* fmt, ...);
int embed_rows_launch(const int32_t* ids, const void* table, void* out, int rows, int vocab, float* stats, float* squares, void* stream);   // rowwise.cu

constexpr int D = ITTAI_Q3_D, DQ = ITTAI_Q3_DQ, DQKV = ITTAI_Q3_DQKV, DGU = ITTAI_Q3_DGU, FF = ITTAI_Q3_FF, HD = ITTAI_Q3_HD, NKV = ITTAI_Q3_NKV;
constexpr int NH = DQ / HD;

static const char* at(const void* base, size_t elems) { return reinterpret_cast<const char*>(base) + 2 * elems; }

static int prefill_launch(const IttaiQwen3Prefill* p, void* st) {
    if (!p || p->n_layers < 1 || p->tokens < 1 || p->n_seqs < 1 || p->max_q_len < 1 || p->kv_cap < 1 || p->vocab < 1) { set_error("prefill: bad sizes"); return ITTAI_E_ARG; }
    if (!p->wqkv || !p->wo || !p->wgu || !p->wd || !p->ln1 || !p->ln2 || !p->qn || !p->kn || !p->embed || !p->rope || !p->ids || !p->pos || !p->seq ||
        !p->slot || !p->seqs || !p->kcache || !p->vcache || !p->h || !p->xn || !p->qkv || !p->attn || !p->act || !p->status ||
        !p->wqkv_f != !p->wgu_f || ((p->wqkv_f || p->split_k) && (!p->stats || !p->zeros))) {
        set_error("prefill: null pointer");
        return ITTAI_E_ARG;
    }
    const int T = p->tokens;
    const bool fused = p->fused_rope && (T > 128 || p->split_k);     // at most 128 rows: only the split-K kernel rotates
    const bool fold = p->wqkv_f != nullptr && T > 128;
    int dev = 0, n_sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n_sms, cudaDevAttrMultiProcessorCount, dev);
    // a small forward: both normalised projections run as split-K GEMMs, which normalise their input themselves
    const bool normed = p->split_k && !fold && gemm_split_wins(T, DGU, n_sms) && gemm_split_wins(T, DQKV, n_sms);
    // shorter still: projections of their own (figures in qwen3_short.cu);
    // the row statistics between them lie in xn, which nothing else uses then
    const bool brief = p->split_k && fused && T <= kShortTokens;
    float* squares = brief ? reinterpret_cast<float*>(p->xn) : nullptr;
    ShortMaps maps;
    int rc = brief ? short_maps(&maps, p) : ITTAI_OK;
    if (rc == ITTAI_OK) rc = embed_rows_launch(p->ids, p->embed, p->h, T, p->vocab, normed && !brief ? p->stats : nullptr, squares, st);
    auto gemm = [&](const void* a, const void* w, void* out, int n, int k, int epi, const void* residual, bool norm, bool stats, const IttaiQkRope* rope,
                    const void* gain = nullptr) {
        if (rc != ITTAI_OK) return;
        IttaiGemm g = {};
        g.m = T; g.n = n; g.k = k; g.epi = epi | (p->split_k ? ITTAI_GEMM_STATIC_W : 0);
        g.a = a; g.w = w; g.out = out; g.residual = residual; g.status = p->status; g.qk_rope = rope;
        if (norm) { g.row_stats = p->stats; g.col_sums = p->zeros; g.stats_parts = D / 128; g.stats_eps = p->eps; g.stats_rms = 1; }
        if (stats) g.stats_out = p->stats;
        rc = gain ? gemm_normed_launch(&g, gain, (cudaStream_t)st) : ittai_gemm_bf16_launch(&g, st);
    };
    auto norm = [&](const void* gain) { if (rc == ITTAI_OK) rc = ittai_rmsnorm_rows(p->h, D, gain, p->xn, D, T, p->eps, st); };
    for (int l = 0; l < p->n_layers && rc == ITTAI_OK; ++l) {
        void* kc = const_cast<char*>(at(p->kcache, (size_t)l * p->kv_layer));
        void* vc = const_cast<char*>(at(p->vcache, (size_t)l * p->kv_layer));
        const void *qn = at(p->qn, (size_t)l * HD), *kn = at(p->kn, (size_t)l * HD);
        // layer 0 reads the embedding rows, which no GEMM epilogue produced: its first norm is a pass of its own
        const bool folded = fold && l > 0;
        IttaiQkRope r = {};
        r.qn = qn; r.kn = kn; r.rope = p->rope; r.pos = p->pos; r.seq = p->seq; r.slot = p->slot;
        r.kcache_layer = kc; r.vcache_layer = vc; r.kv_cap = p->kv_cap; r.eps = p->eps;
        const void *g1 = at(p->ln1, (size_t)l * D), *g2 = at(p->ln2, (size_t)l * D);
        if (!folded && !normed && !brief) norm(g1);
        const void* x = folded || normed ? p->h : p->xn;
        const void* wq = at(folded ? p->wqkv_f : p->wqkv, (size_t)l * DQKV * D);
        if (brief) {
            rc = short_qkv(maps, p, l, r, g1, squares, (cudaStream_t)st);
        } else if (fused) {
            gemm(x, wq, p->qkv, DQKV, D, ITTAI_EPI_QKROPE, nullptr, folded || normed, false, &r, normed ? g1 : nullptr);
        } else {
            gemm(x, wq, p->qkv, DQKV, D, ITTAI_EPI_NONE, nullptr, folded || normed, false, nullptr, normed ? g1 : nullptr);
            if (rc == ITTAI_OK) rc = ittai_qwen3_qk_rope_scatter(p->qkv, qn, kn, p->rope, p->pos, p->seq, p->slot, kc, vc, T, p->kv_cap, p->eps, st);
        }
        IttaiAttention a = {};
        a.q = p->qkv; a.k = kc; a.v = vc; a.o = p->attn;
        a.q_row = DQKV; a.q_head = HD; a.o_row = DQ; a.o_head = HD;
        a.k_row = a.v_row = p->k_row; a.k_head = a.v_head = p->k_head; a.k_seq = a.v_seq = p->k_seq;
        a.seqs = p->seqs; a.n_seqs = p->n_seqs; a.n_heads = NH; a.group = NH / NKV; a.head_dim = HD; a.causal = 1; a.max_q_len = p->max_q_len;
        a.q_rows_total = T; a.kv_rows_total = (int32_t)p->kv_rows_total; a.status = p->status; a.seqs_ready = 1;
        if (rc == ITTAI_OK) rc = ittai_attention_packed_launch(&a, st);
        if (brief) {
            if (rc == ITTAI_OK) rc = short_o(maps, p, l, squares, (cudaStream_t)st);
            if (rc == ITTAI_OK) rc = short_gate_up(maps, p, l, g2, squares, (cudaStream_t)st);
            if (rc == ITTAI_OK) rc = short_down(maps, p, l, squares, (cudaStream_t)st);
            continue;
        }
        gemm(p->attn, at(p->wo, (size_t)l * D * DQ), p->h, D, DQ, ITTAI_EPI_NONE, p->h, false, fold || normed, nullptr);
        if (!fold && !normed) norm(g2);
        gemm(fold || normed ? p->h : p->xn, at(fold ? p->wgu_f : p->wgu, (size_t)l * DGU * D), p->act, DGU, D, ITTAI_EPI_SWIGLU, nullptr, fold || normed, false, nullptr, normed ? g2 : nullptr);
        gemm(p->act, at(p->wd, (size_t)l * D * FF), p->h, D, FF, ITTAI_EPI_NONE, p->h, false, (fold || normed) && l + 1 < p->n_layers, nullptr);
    }
    return rc;
}

}  // namespace ittai

extern "C" int ittai_qwen3_prefill_launch(const IttaiQwen3Prefill* p, void* stream) { return ittai::prefill_launch(p, stream); }
