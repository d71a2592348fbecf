// Host side of the batched prompt pass: workspace, TMA tensor maps, and the per-layer
// sequence of tensor-core GEMMs (prefill.cuh).  Restates the naive forward of the reference
// (full_model.rs:336-437 and layer.rs:1287-1431) for the prompt positions only, with the
// residual stream in fp32 and 16-bit GEMM inputs; K and V go straight into the pages the
// decode kernels read.  Used by cd_prefill for bf16 / fp16 models on one GPU; every other
// case keeps feeding the prompt one token at a time.
#include "pf_launch.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "model.h"
#include "sample_attn.cuh"
#include "step.cuh"

namespace cd {
namespace {

struct SampleGraphKey {
    int ns = 0, mode = 0, top_k = 0;
    float t = 0.f, softcap = 0.f;
    int split = 0;
    int len0 = -1;  // the prompt length the graphs were captured for: the number of shared prompt tokens is a launch argument
    bool operator==(const SampleGraphKey& o) const {
        return ns == o.ns && mode == o.mode && top_k == o.top_k && t == o.t && softcap == o.softcap && split == o.split && len0 == o.len0;
    }
};

struct PrefillCtx {
    EncodeTiledFn encode = nullptr;
    SampleGraphKey s_key;
    std::map<int, cudaGraphExec_t> s_graphs;  // captured multi-sample steps by their attention's slices (SaSplit::id)
    uint64_t s_graph_nodes = 0;
    std::vector<CUtensorMap> k_pages, v_pages;  // per layer, built once
    std::vector<CUtensorMap> sk_qkv, sk_o, sk_13, sk_2;  // the same matrices in 128-row boxes (multi-sample decode)
    CUtensorMap sk_head;
    // FP8 linears: one layer's four matrices widened to 16 bits before its GEMMs
    void *f8_qkv = nullptr, *f8_o = nullptr, *f8_13 = nullptr, *f8_2 = nullptr;
    // multi-sample decode workspace (one arena, sized for s_cap samples)
    int s_cap = 0;
    char* s_arena = nullptr;
    float *sx = nullptr, *sq = nullptr, *slogits = nullptr, *spart_acc = nullptr, *spart_ml = nullptr;
    float* sksum = nullptr;  // [8 K slices][16][dim] partial sums of the linears that are cut along K
    float *sblock_vals = nullptr, *stopk_vals = nullptr, *smaxes = nullptr, *ssums = nullptr;
    uint32_t *sblock_idxs = nullptr, *stopk_idxs = nullptr, *sout_token = nullptr, *sring = nullptr;
    unsigned int *scounters = nullptr, *shead_counters = nullptr;
    void *sxn = nullptr, *sgate = nullptr;  // [2][s_cap][...] hi, lo
    DevState* sst = nullptr;
    // workspace (grow-only)
    size_t rows = 0;
    float* x = nullptr;       // [rows][dim] residual stream
    void* xn = nullptr;       // [2][rows][max(dim, q_dim)] normalised input / attention output (hi, lo)
    void* q = nullptr;        // [2][rows][q_dim]
    void* gate = nullptr;     // [2][rows][hidden]
};

// one of the two halves (K, V) of a layer's pages as {d, token in page, kv head, page}; a box is 128 keys of one head
bool encode_pages(PrefillCtx* c, CUtensorMap* map, CUtensorMapDataType dt, const char* pool, int half, int hd, int page_tokens, int kv_heads, int num_pages) {
    const uint64_t head = (uint64_t)page_tokens * hd * 2, page = 2 * kv_heads * head;
    return encode_rows_4d(c->encode, map, dt, pool + half * kv_heads * head, hd, page_tokens, kv_heads, num_pages, (uint64_t)hd * 2, head, page);
}

// the few-rows GEMM: w in 128-row boxes, x = the [NB][K] activation block (hi rows, then lo rows)
template <int NB, class Epi>
cudaError_t sk_launch_t(cd_model* m, const CUtensorMap& w, const CUtensorMap& x, int N, int K, int ns, bool bf16,
                        const Epi& epi, int kslices) {
    auto kern = pf_skinny_kernel<NB, Epi>;
    static bool attr_set = false;  // per instantiation
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SkTile<NB>::smem(SkTile<NB>::STAGES_ALONE));
        if (e != cudaSuccess) return e;
        attr_set = true;
    }
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((N + 127) / 128, kslices);
    const int nst = (int)(lc.gridDim.x * lc.gridDim.y) <= m->sm_count ? SkTile<NB>::STAGES_ALONE : SkTile<NB>::STAGES_SHARED;
    lc.blockDim = dim3(PF_THREADS);
    lc.dynamicSmemBytes = SkTile<NB>::smem(nst);
    lc.stream = m->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // the kernel fetches weights before it waits for its predecessor
    at[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = at;
    lc.numAttrs = m->pdl ? 1 : 0;
    m->launches++;
    return cudaLaunchKernelEx(&lc, kern, w, x, N, K, ns, nst, make_idesc(NB, bf16), &m->st->error, epi);
}
template <class Epi>
cudaError_t sk_launch(cd_model* m, bool split, const CUtensorMap& w, const CUtensorMap& x, int N, int K, int ns, bool bf16,
                      const Epi& epi, int kslices = 1) {
    return split ? sk_launch_t<32>(m, w, x, N, K, ns, bf16, epi, kslices) : sk_launch_t<16>(m, w, x, N, K, ns, bf16, epi, kslices);
}

// weights, LM head and K pages: maps built once per model
int ensure_weight_maps(cd_model* m, PrefillCtx* c, CUtensorMapDataType dt, CUtensorMapDataType kdt) {
    if (!c->k_pages.empty()) return CD_OK;
    const cd_config& cf = m->cfg;
    const int D = cf.dim, Q = cf.q_dim, KV = cf.kv_dim, H = cf.hidden;
    c->k_pages.resize(cf.nlayers); c->v_pages.resize(cf.nlayers);
    c->sk_qkv.resize(cf.nlayers); c->sk_o.resize(cf.nlayers); c->sk_13.resize(cf.nlayers); c->sk_2.resize(cf.nlayers);
    bool ok = encode_2d(c->encode, &c->sk_head, dt, m->lm_head, D, m->v_loc, (uint64_t)D * 2, 128);
    auto pages = [&](int l) {
        return encode_pages(c, &c->k_pages[l], kdt, (const char*)m->layers[l].kv, 0, cf.hd, m->page_tokens, cf.kv_heads, m->num_pages) &&
               encode_pages(c, &c->v_pages[l], kdt, (const char*)m->layers[l].kv, 1, cf.hd, m->page_tokens, cf.kv_heads, m->num_pages);
    };
    if (m->opt.weight_dtype == CD_DTYPE_FP8_E4M3) {
        const size_t n_qkv = (size_t)(Q + 2 * KV) * D, n_o = (size_t)D * Q, n_13 = (size_t)2 * H * D, n_2 = (size_t)D * H;
        if (cudaMalloc(&c->f8_qkv, n_qkv * 2) != cudaSuccess || cudaMalloc(&c->f8_o, n_o * 2) != cudaSuccess ||
            cudaMalloc(&c->f8_13, n_13 * 2) != cudaSuccess || cudaMalloc(&c->f8_2, n_2 * 2) != cudaSuccess) {
            c->k_pages.clear();
            return fail(m, CD_ERR_CUDA, "prompt-pass buffers for the widened FP8 matrices");
        }
        for (int l = 0; l < cf.nlayers && ok; ++l) {
            ok = ok && pages(l);
        }
        if (!ok) { c->k_pages.clear(); return fail(m, CD_ERR_CUDA, "cuTensorMapEncodeTiled failed for a weight matrix"); }
        return CD_OK;
    }
    for (int l = 0; l < cf.nlayers && ok; ++l) {
        const cd_layer_dev& L = m->layers[l];
        ok = ok && encode_2d(c->encode, &c->sk_qkv[l], dt, L.wqkv, D, Q + 2 * KV, (uint64_t)D * 2, 128);
        ok = ok && encode_2d(c->encode, &c->sk_o[l], dt, L.wo, Q, D, (uint64_t)Q * 2, 128);
        ok = ok && encode_2d(c->encode, &c->sk_13[l], dt, L.w13, D, 2 * H, (uint64_t)D * 2, 128);
        ok = ok && encode_2d(c->encode, &c->sk_2[l], dt, L.w2, H, D, (uint64_t)H * 2, 128);
        ok = ok && pages(l);
    }
    if (!ok) { c->k_pages.clear(); return fail(m, CD_ERR_CUDA, "cuTensorMapEncodeTiled failed for a weight matrix"); }
    return CD_OK;
}

// the context of a model the tensor-core passes can serve, or CD_ERR_UNSUPPORTED
int get_ctx(cd_model* m, PrefillCtx** out, bool fp8_ok, bool tp_ok = false) {
    const cd_config& cf = m->cfg;
    const int dt = m->opt.weight_dtype;
    if (dt != CD_DTYPE_BF16 && dt != CD_DTYPE_F16 && !(fp8_ok && dt == CD_DTYPE_FP8_E4M3)) return CD_ERR_UNSUPPORTED;
    // tensor parallel: the prompt pass only (the ranks' partial products meet in the link region's buffers)
    if (m->tp_world > 1 && (!tp_ok || m->tp_pf_rows == 0 || dt == CD_DTYPE_FP8_E4M3)) return CD_ERR_UNSUPPORTED;
    if (cf.dim % 32 || cf.q_dim % 32 || cf.hidden % 16 || (cf.hd != 64 && cf.hd != 128)) return CD_ERR_UNSUPPORTED;
    if (m->page_tokens > 128 || 128 % m->page_tokens) return CD_ERR_UNSUPPORTED;
    PrefillCtx* c = (PrefillCtx*)m->prefill_ctx;
    if (!c) {
        c = new PrefillCtx();
        if (!(c->encode = encode_tiled_fn())) {
            delete c;
            return fail(m, CD_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
        }
        m->prefill_ctx = c;
    }
    *out = c;
    return CD_OK;
}

// T16: the 16-bit type of the weights and of the linears' activation operands; KT: the type of the KV
// cache, which the attention GEMMs' other operands (q, the probabilities, V transposed) share.
template <typename T16, typename KT>
int run(cd_model* m, PrefillCtx* c, size_t n, bool split) {
    const cd_config& cf = m->cfg;
    const bool bf16 = std::is_same<T16, __nv_bfloat16>::value, kbf16 = std::is_same<KT, __nv_bfloat16>::value;
    const CUtensorMapDataType dt = bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    const CUtensorMapDataType kdt = kbf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    const int D = cf.dim, Q = cf.q_dim, KV = cf.kv_dim, H = cf.hidden, hd = cf.hd;
    const int pos0 = (int)m->len, M = (int)n;
    auto cuda_fail = [&](const char* what, cudaError_t e) { return fail(m, CD_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e)); };

    int rc = ensure_weight_maps(m, c, dt, kdt);
    if (rc) return rc;
    // ---- workspace
    const size_t rows = round_up(n, PF_BM);
    if (rows > c->rows) {
        for (void* ptr : {(void*)c->x, c->xn, c->q, c->gate}) if (ptr) cudaFree(ptr);
        c->x = nullptr; c->xn = c->q = c->gate = nullptr;
        const size_t r = rows;
        c->rows = 0;
        struct { void** ptr; size_t bytes; } want[] = {
            {(void**)&c->x, r * D * 4}, {&c->xn, 2 * r * (size_t)std::max(D, Q) * 2}, {&c->q, 2 * r * (size_t)Q * 2}, {&c->gate, 2 * r * (size_t)H * 2}};
        for (auto& w : want) {
            cudaError_t e = cudaMalloc(w.ptr, w.bytes);
            if (e == cudaSuccess) e = cudaMemsetAsync(*w.ptr, 0, w.bytes, m->stream);
            if (e != cudaSuccess) return cuda_fail("prefill workspace", e);
        }
        c->rows = r;
    }
    const size_t R = c->rows;
    // hi matrices first, lo matrices (split mode) in the second half of each buffer
    T16* xn = (T16*)c->xn; KT* qb = (KT*)c->q; T16* gate = (T16*)c->gate;
    T16* xn_lo = split ? xn + R * (size_t)std::max(D, Q) : nullptr;
    KT* q_lo = split ? qb + R * (size_t)Q : nullptr;
    T16* gate_lo = split ? gate + R * (size_t)H : nullptr;
    CUtensorMap a_q[2];
    const bool ok = encode_2d(c->encode, &a_q[0], kdt, qb, Q, R, (uint64_t)Q * 2, PF_BM) &&
                    (!split || encode_2d(c->encode, &a_q[1], kdt, q_lo, Q, R, (uint64_t)Q * 2, PF_BM));
    if (!ok) return fail(m, CD_ERR_CUDA, "cuTensorMapEncodeTiled failed for an activation buffer");

    cudaError_t e;
#define PF_TRY(what, x) do { e = (x); if (e != cudaSuccess) return cuda_fail(what, e); } while (0)
    pf_embed_kernel<T16><<<M, 256, 0, m->stream>>>((const T16*)m->embed, m->prompt_dev, c->x, D);
    m->launches++;
    // tensor parallel: Wo and W2 are split along their input, so their products are partial sums that the ranks exchange
    // through two alternating buffers of the link region (prefill.cuh, tp_pf_reduce_kernel)
    const bool tpar = m->tp_world > 1;
    const size_t pf_flags = TpRegion::pf_flags_off(m->tp_world, D, m->tp_nb), pf_bufs = TpRegion::pf_buf_off(m->tp_world, D, m->tp_nb);
    if (tpar && rows > m->tp_pf_rows) return fail(m, CD_ERR_CAPACITY, "prompt chunk longer than the tensor-parallel partial-sum buffers");
    auto tp_buf = [&]() { return reinterpret_cast<float*>(m->link_region + pf_bufs + (size_t)((m->tp_pf_seq + 1) & 1u) * m->tp_pf_rows * D * 4); };
    auto tp_allreduce = [&]() {
        m->tp_pf_seq += 1;
        const int buf = (int)(m->tp_pf_seq & 1u);
        tp_pf_publish_kernel<<<1, 32, 0, m->stream>>>(m->tp, pf_flags, buf, m->tp_pf_seq);
        tp_pf_reduce_kernel<<<m->sm_count * 4, 256, 0, m->stream>>>(m->tp, pf_flags, pf_bufs, buf, m->tp_pf_seq, c->x, M, m->tp_pf_rows, m->alpha,
                                                                   &m->st->error);
        m->launches += 2;
        return cudaGetLastError();
    };
    PfGemm g = {};
    g.err = &m->st->error;
    const PfAttn attn{M, pos0, 0, 1, cf.gqa_ratio, m->page_tokens, split ? 1 : 0, (float)(1.4426950408889634 / std::sqrt((double)hd)), nullptr, &m->st->error};
    const bool fp8 = m->opt.weight_dtype == CD_DTYPE_FP8_E4M3;
    auto quantised = [&](PfGemm& p, const void* rows, int K) {  // the GEMM's output columns take the FP8 row scales
        if (!fp8) return;
        p.qrows = (const unsigned char*)rows; p.qstride = Wfmt<Fp8Row>::row_stride(K); p.qscale_off = Wfmt<Fp8Row>::scale_off(K);
    };
    for (int l = 0; l < cf.nlayers; ++l) {
        const cd_layer_dev& L = m->layers[l];
        if (fp8) {  // this layer's e4m3 values as 16-bit matrices (exact); the previous layer's GEMMs are done with the buffers (stream order)
            const int wb = m->sm_count * 8;
            pf_widen_fp8_kernel<T16><<<wb, 256, 0, m->stream>>>((const unsigned char*)L.wqkv, Wfmt<Fp8Row>::row_stride(D), (T16*)c->f8_qkv, Q + 2 * KV, D);
            pf_widen_fp8_kernel<T16><<<wb, 256, 0, m->stream>>>((const unsigned char*)L.wo, Wfmt<Fp8Row>::row_stride(Q), (T16*)c->f8_o, D, Q);
            pf_widen_fp8_kernel<T16><<<wb, 256, 0, m->stream>>>((const unsigned char*)L.w13, Wfmt<Fp8Row>::row_stride(D), (T16*)c->f8_13, 2 * H, D);
            pf_widen_fp8_kernel<T16><<<wb, 256, 0, m->stream>>>((const unsigned char*)L.w2, Wfmt<Fp8Row>::row_stride(H), (T16*)c->f8_2, D, H);
            m->launches += 4;
        }
        pf_rmsnorm_kernel<T16><<<M, 256, 0, m->stream>>>(c->x, L.gamma1, xn, xn_lo, D);
        m->launches++;
        {   // q, k, v = xn Wqkv with RoPE; k and v into the pages
            PfGemm p = g; p.M = M; p.N = Q + 2 * KV; p.K = D;
            quantised(p, L.wqkv, D);
            PfEpiQKV<KT> epi{qb, q_lo, (KT*)L.kv, m->page_table, m->rope, Q, KV, hd, cf.kv_heads, m->page_tokens, pos0};
            PF_TRY("qkv gemm", (pf_launch(m, c->encode, xn, xn_lo, fp8 ? c->f8_qkv : L.wqkv, Q + 2 * KV, p, bf16, epi)));
        }
        const PaOut<T16> attn_out{xn, xn_lo, Q, hd};
        if (hd == 128) PF_TRY("attention", (pa_launch<KT, 128, 128, false>(m, a_q, split, c->k_pages[l], c->v_pages[l], attn, cf.heads, attn_out)));
        else PF_TRY("attention", (pa_launch<KT, 64, 64, false>(m, a_q, split, c->k_pages[l], c->v_pages[l], attn, cf.heads, attn_out)));
        {   // x2 = x + alpha * (attn Wo)
            PfGemm p = g; p.M = M; p.N = D; p.K = Q;
            quantised(p, L.wo, Q);
            if (tpar) {
                PF_TRY("wo gemm", (pf_launch(m, c->encode, xn, xn_lo, fp8 ? c->f8_o : L.wo, D, p, bf16, PfEpiPartial{tp_buf(), D})));
                PF_TRY("wo all-reduce", tp_allreduce());
            } else {
                PF_TRY("wo gemm", (pf_launch(m, c->encode, xn, xn_lo, fp8 ? c->f8_o : L.wo, D, p, bf16, PfEpiResidual{c->x, D, m->alpha})));
            }
        }
        pf_rmsnorm_kernel<T16><<<M, 256, 0, m->stream>>>(c->x, L.gamma2, xn, xn_lo, D);
        m->launches++;
        {   // gate = act(x2n W1) * (x2n W3)
            PfGemm p = g; p.M = M; p.N = 2 * H; p.K = D;
            quantised(p, L.w13, D);
            PF_TRY("w13 gemm", (pf_launch(m, c->encode, xn, xn_lo, fp8 ? c->f8_13 : L.w13, 2 * H, p, bf16, PfEpiGate<T16>{gate, gate_lo, H, m->opt.activation})));
        }
        {   // x = x2 + alpha * (gate W2^T)
            PfGemm p = g; p.M = M; p.N = D; p.K = H;
            quantised(p, L.w2, H);
            if (tpar) {
                PF_TRY("w2 gemm", (pf_launch(m, c->encode, gate, gate_lo, fp8 ? c->f8_2 : L.w2, D, p, bf16, PfEpiPartial{tp_buf(), D})));
                PF_TRY("w2 all-reduce", tp_allreduce());
            } else {
                PF_TRY("w2 gemm", (pf_launch(m, c->encode, gate, gate_lo, fp8 ? c->f8_2 : L.w2, D, p, bf16, PfEpiResidual{c->x, D, m->alpha})));
            }
        }
    }
    // the last prompt position's hidden state, where the LM-head GEMV expects it
    PF_TRY("copy last row", cudaMemcpyAsync(m->x_a, c->x + (size_t)(M - 1) * D, (size_t)D * 4, cudaMemcpyDeviceToDevice, m->stream));
#undef PF_TRY
    return CD_OK;
}

// ---------------------------------------------------------------- several samples per step
// `--samples N` sharing a prompt (inference.rs:255-297 runs them one after the other): all N
// continuations advance together, one token each per step, so every weight byte is read once
// per step for all of them.  The linears are the prompt-pass GEMMs with one row per sample;
// attention, head reductions and samplers are the single-sample kernels, run per sample on that
// sample's state, so each sample's draws are those of its own sequential loop.
template <typename T16, typename KT>
int run_samples(cd_model* m, PrefillCtx* c, const uint32_t* first, int ns, size_t nsteps, int mode, int top_k, float t, float softcap,
                uint64_t* rng, uint32_t* out_ids, bool split) {
    const cd_config& cf = m->cfg;
    const bool bf16 = std::is_same<T16, __nv_bfloat16>::value;
    const CUtensorMapDataType dt = bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    const CUtensorMapDataType kdt = std::is_same<KT, __nv_bfloat16>::value ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    const int D = cf.dim, Q = cf.q_dim, KV = cf.kv_dim, H = cf.hidden, hd = cf.hd, V = m->v_loc, NB = m->nblocks;
    const int Vp = (V + 31) & ~31;  // row stride of the logits: the GEMM epilogue writes whole 32-column chunks
    const int pps = m->pages_per_seq, pt = m->page_tokens, len0 = (int)m->len, ring_ld = cf.seq + 1;
    auto cuda_fail = [&](const char* what, cudaError_t e) { return fail(m, CD_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e)); };
    int rc = ensure_weight_maps(m, c, dt, kdt);
    if (rc) return rc;
    cudaError_t e;
#define PF_TRY(what, x) do { e = (x); if (e != cudaSuccess) return cuda_fail(what, e); } while (0)
    if (ns > c->s_cap) {
        if (c->s_arena) cudaFree(c->s_arena);
        c->s_arena = nullptr; c->s_cap = 0;
        const size_t S = SK_ROWS, W = (size_t)std::max(D, Q);  // blocks of 16 rows: hi parts, then lo parts
        size_t off = 0;
        auto carve = [&](size_t bytes) { const size_t o = off; off = (off + bytes + 255) / 256 * 256; return o; };
        const size_t o_x = carve(S * D * 4), o_q = carve(S * Q * 4), o_logits = carve(S * Vp * 4);
        const size_t o_pacc = carve(S * cf.heads * m->nsplit * hd * 4), o_pml = carve(S * cf.heads * m->nsplit * 2 * 4);
        const size_t o_cnt = carve(S * cf.heads * 4), o_hcnt = carve(S * 4);
        const size_t o_bv = carve(S * NB * 4), o_bi = carve(S * NB * 4), o_tv = carve(S * NB * CD_MAX_GPU_TOPK * 4), o_ti = carve(S * NB * CD_MAX_GPU_TOPK * 4);
        const size_t o_mx = carve(S * NB * 4), o_sm = carve(S * NB * 4), o_tok = carve(S * 64), o_ring = carve(S * ring_ld * 4);
        const size_t o_xn = carve(2 * S * W * 2), o_gate = carve(2 * S * H * 2), o_st = carve(S * sizeof(DevState));
        const size_t o_ks = carve(8 * S * D * 4);
        PF_TRY("sample workspace", cudaMalloc((void**)&c->s_arena, off));
        PF_TRY("sample workspace", cudaMemsetAsync(c->s_arena, 0, off, m->stream));
        char* b = c->s_arena;
        c->sx = (float*)(b + o_x); c->sq = (float*)(b + o_q); c->slogits = (float*)(b + o_logits);
        c->spart_acc = (float*)(b + o_pacc); c->spart_ml = (float*)(b + o_pml); c->scounters = (unsigned int*)(b + o_cnt);
        c->shead_counters = (unsigned int*)(b + o_hcnt); c->sblock_vals = (float*)(b + o_bv); c->sblock_idxs = (uint32_t*)(b + o_bi);
        c->stopk_vals = (float*)(b + o_tv); c->stopk_idxs = (uint32_t*)(b + o_ti); c->smaxes = (float*)(b + o_mx); c->ssums = (float*)(b + o_sm);
        c->sout_token = (uint32_t*)(b + o_tok); c->sring = (uint32_t*)(b + o_ring); c->sxn = b + o_xn; c->sgate = b + o_gate;
        c->sst = (DevState*)(b + o_st);
        c->sksum = (float*)(b + o_ks);
        c->s_cap = (int)S;
    }
    const size_t S = (size_t)c->s_cap, W = (size_t)std::max(D, Q);
    T16* xn = (T16*)c->sxn; T16* gate = (T16*)c->sgate;
    // the lo block starts 16 rows into the buffer, in rows of whatever width the buffer currently holds
    T16* xn_lo = split ? xn + S * (size_t)D : nullptr;
    T16* attn_lo = split ? xn + S * (size_t)Q : nullptr;
    T16* gate_lo = split ? gate + S * (size_t)H : nullptr;
    // one map per activation buffer: rows 0-15 the hi parts, rows 16-31 the lo parts
    const uint32_t xrows = split ? 2 * SK_ROWS : SK_ROWS;
    CUtensorMap a_xn, a_attn, a_gate;
    const bool ok = encode_2d(c->encode, &a_xn, dt, xn, D, xrows, (uint64_t)D * 2, xrows) && encode_2d(c->encode, &a_attn, dt, xn, Q, xrows, (uint64_t)Q * 2, xrows) &&
                    encode_2d(c->encode, &a_gate, dt, gate, H, xrows, (uint64_t)H * 2, xrows);
    if (!ok) return fail(m, CD_ERR_CUDA, "cuTensorMapEncodeTiled failed for an activation buffer");

    // page tables: prompt pages that are full are shared, the page the prompt ends in is copied, later pages are the sample's own
    std::vector<int> table((size_t)ns * pps);
    for (int s = 0; s < ns; ++s)
        for (int j = 0; j < pps; ++j) table[(size_t)s * pps + j] = (s == 0 || (j + 1) * pt <= len0) ? j : s * pps + j;
    PF_TRY("page tables", cudaMemcpyAsync(m->page_table, table.data(), table.size() * 4, cudaMemcpyHostToDevice, m->stream));
    PF_TRY("page tables", cudaStreamSynchronize(m->stream));  // the host vector goes away
    if (len0 % pt) {
        const int jp = len0 / pt;
        const size_t page_bytes = (size_t)2 * cf.kv_heads * pt * hd * sizeof(KT);
        for (int l = 0; l < cf.nlayers; ++l)
            for (int s = 1; s < ns; ++s)
                PF_TRY("prompt page copy", cudaMemcpyAsync((char*)m->layers[l].kv + ((size_t)s * pps + jp) * page_bytes,
                                                           (char*)m->layers[l].kv + (size_t)jp * page_bytes, page_bytes, cudaMemcpyDeviceToDevice, m->stream));
    }
    for (int s = 0; s < ns; ++s) {
        begin_loop_kernel<<<1, 1, 0, m->stream>>>(c->sst + s, len0, first[s], rng ? rng[s] : 0ull);
        m->launches++;
    }
    PF_TRY("sample states", cudaGetLastError());
    PF_TRY("event", cudaEventRecord(m->ev0, m->stream));

    const float scale = 1.0f / std::sqrt((float)hd);
    const float inv_t = 1.0f / std::max(t, 1.17549435e-38f);  // decode.rs:174
    const int shared_tokens = len0 / pt * pt;
    const SaBlocks blocks{cf.gqa_ratio, ns};
    // one step of all samples; everything that changes from step to step is read on the device, except the
    // attention's slices, which select the captured graph
    auto enqueue_step = [&](const SaSplit& cut) -> int {
        pf_embed_samples_kernel<T16><<<ns, 256, 0, m->stream>>>((const T16*)m->embed, c->sst, c->sx, D, m->full_cfg.vocab);
        m->launches++;
        // Wo and W2 have few output rows: they are cut along K into `ks` slices and the following
        // RMSNorm kernel adds the slices' partial sums (in slice order) into the residual stream
        const int ks = std::max(1, std::min(8, m->sm_count / ((D + 127) / 128)));
        const int nthreads = std::min(1024, std::max(256, D / 4 / 32 * 32));
        auto fold = [&](const float* gamma) {
            return launch_chain(m, pf_reduce_rmsnorm_kernel<T16>, dim3(ns), dim3(nthreads), 0, c->sx, (const float*)c->sksum, ks, m->alpha, gamma, xn, xn_lo, D);
        };
        for (int l = 0; l < cf.nlayers; ++l) {
            const cd_layer_dev& L = m->layers[l];
            if (l == 0) {
                pf_rmsnorm_kernel<T16><<<ns, 256, 0, m->stream>>>(c->sx, L.gamma1, xn, xn_lo, D);
                m->launches++;
            } else {
                PF_TRY("norm", fold(L.gamma1));
            }
            {
                SkEpiQKV<KT> epi{c->sq, (KT*)L.kv, m->page_table, m->rope, c->sst, Q, KV, hd, cf.kv_heads, pt, pps};
                PF_TRY("qkv gemm", sk_launch(m, split, c->sk_qkv[l], a_xn, Q + 2 * KV, D, ns, bf16, epi));
            }
            const SampleAttn at{c->sq, m->page_table, c->sst, c->spart_acc, c->spart_ml, c->scounters, cf.kv_heads, pt, pps, m->nsplit, shared_tokens, blocks, cut, scale};
            const dim3 agrid(cf.kv_heads, cut.shared + cut.own, blocks.count());
            PF_TRY("attention", hd == 128 ? launch_chain(m, sample_attn_kernel<KT, T16, 128>, agrid, dim3(SA_THREADS), 0, at, (const KT*)L.kv, xn, attn_lo)
                                          : launch_chain(m, sample_attn_kernel<KT, T16, 64>, agrid, dim3(SA_THREADS), 0, at, (const KT*)L.kv, xn, attn_lo));
            PF_TRY("wo gemm", sk_launch(m, split, c->sk_o[l], a_attn, D, Q, ns, bf16, SkEpiPartial{c->sksum, D}, ks));
            PF_TRY("norm", fold(L.gamma2));
            PF_TRY("w13 gemm", sk_launch(m, split, c->sk_13[l], a_xn, 2 * H, D, ns, bf16, SkEpiGate<T16>{gate, gate_lo, H, m->opt.activation}));
            PF_TRY("w2 gemm", sk_launch(m, split, c->sk_2[l], a_gate, D, H, ns, bf16, SkEpiPartial{c->sksum, D}, ks));
        }
        PF_TRY("norm", fold(m->gamma_final));
        PF_TRY("head gemm", sk_launch(m, split, c->sk_head, a_xn, V, D, ns, bf16, SkEpiStore{c->slogits, Vp}));
        // each sample's own reductions and draw, on its own state; one launch covers all samples
        if (mode == 0) {
            head_argmax_kernel<<<dim3(NB, ns), 256, 0, m->stream>>>(c->slogits, V, c->sblock_vals, c->sblock_idxs, c->shead_counters, c->sout_token, c->sst, c->sring, 1, 0,
                                                                   TpLink{}, (size_t)Vp, (size_t)NB, (size_t)16, (size_t)ring_ld);
            m->launches++;
        } else if (mode == 1) {
            const size_t cs = (size_t)NB * CD_MAX_GPU_TOPK;
            head_topk_kernel<<<dim3(NB, ns), 256, 0, m->stream>>>(c->slogits, V, top_k, c->stopk_vals, c->stopk_idxs, (size_t)Vp, cs);
            sample_topk_kernel<<<ns, 1024, 0, m->stream>>>(c->stopk_vals, c->stopk_idxs, NB * top_k, top_k, t, softcap, c->sst, c->sring, cs, (size_t)ring_ld);
            m->launches += 2;
        } else {
            head_stats_kernel<<<dim3(NB, ns), 256, 0, m->stream>>>(c->slogits, V, inv_t, softcap, c->smaxes, c->ssums, (size_t)Vp, (size_t)NB);
            sample_fullvocab_kernel<<<ns, 256, 0, m->stream>>>(c->slogits, cf.vocab, c->smaxes, c->ssums, NB, t, softcap, c->sst, c->sring, (size_t)Vp, (size_t)NB,
                                                           (size_t)ring_ld);
            m->launches += 2;
        }
        PF_TRY("step launch", cudaGetLastError());
        return CD_OK;
    };
    // graphs of a step are kept per cut of the attention for as long as the request parameters stay the same
    const SampleGraphKey key{ns, mode, top_k, t, softcap, split ? 1 : 0, len0};
    if (!(key == c->s_key)) {
        for (auto& kv : c->s_graphs) cudaGraphExecDestroy(kv.second);
        c->s_graphs.clear();
        c->s_key = key;
    }
    for (size_t step = 0; step < nsteps; ++step) {
        const int attn_len = len0 + (int)step + 1;
        const SaSplit cut = sa_split(shared_tokens, attn_len, blocks, cf.kv_heads, m->nsplit, m->sm_count);
        if (!m->opt.use_graph) {
            if ((rc = enqueue_step(cut))) return rc;
            continue;
        }
        auto it = c->s_graphs.find(cut.id());
        if (it == c->s_graphs.end()) {
            cudaGraph_t graph = nullptr;
            const uint64_t before = m->launches;
            PF_TRY("graph capture", cudaStreamBeginCapture(m->stream, cudaStreamCaptureModeThreadLocal));
            rc = enqueue_step(cut);
            const cudaError_t e2 = cudaStreamEndCapture(m->stream, &graph);
            if (rc || e2 != cudaSuccess) {
                if (graph) cudaGraphDestroy(graph);
                return rc ? rc : cuda_fail("graph capture", e2);
            }
            cudaGraphExec_t exec = nullptr;
            e = cudaGraphInstantiate(&exec, graph, 0);
            cudaGraphDestroy(graph);
            if (e != cudaSuccess) return cuda_fail("graph instantiate", e);
            c->s_graph_nodes = m->launches - before;
            m->launches = before;
            it = c->s_graphs.emplace(cut.id(), exec).first;
        }
        PF_TRY("graph launch", cudaGraphLaunch(it->second, m->stream));
        m->launches += c->s_graph_nodes;
    }
    PF_TRY("event", cudaEventRecord(m->ev1, m->stream));
    std::vector<DevState> hst(ns);
    std::vector<uint32_t> hring((size_t)ns * ring_ld);
    PF_TRY("read back", cudaMemcpyAsync(hst.data(), c->sst, (size_t)ns * sizeof(DevState), cudaMemcpyDeviceToHost, m->stream));
    PF_TRY("read back", cudaMemcpyAsync(hring.data(), c->sring, hring.size() * 4, cudaMemcpyDeviceToHost, m->stream));
    PF_TRY("read back", cudaMemcpyAsync(m->h_state, m->st, sizeof(DevState), cudaMemcpyDeviceToHost, m->stream));
    PF_TRY("sync", cudaStreamSynchronize(m->stream));
    PF_TRY("event", cudaEventElapsedTime(&m->last_ms, m->ev0, m->ev1));
#undef PF_TRY
    for (int s = 0; s < ns; ++s) {
        memcpy(out_ids + (size_t)s * nsteps, hring.data() + (size_t)s * ring_ld, nsteps * 4);
        if (rng) rng[s] = hst[s].rng;
        if (hst[s].error) {
            cudaMemsetAsync(&c->sst[s].error, 0, sizeof(int32_t), m->stream);
            return device_wait_failed(m, hst[s].error, " during the multi-sample decode");
        }
    }
    if (m->h_state->error) return device_wait_failed(m, m->h_state->error, " during the multi-sample decode");
    return CD_OK;
}

}  // namespace

int decode_samples(cd_model* m, const uint32_t* first, int ns, size_t nsteps, int mode, int top_k, float t, float softcap, uint64_t* rng,
                   uint32_t* out_ids) {
    PrefillCtx* c = nullptr;
    int rc = get_ctx(m, &c, false);
    if (rc) return rc;
    const char* pm = getenv("CD_PREFILL");
    const bool split = !(pm && !strcmp(pm, "fast"));
    if (m->opt.weight_dtype == CD_DTYPE_F16) return run_samples<__half, __half>(m, c, first, ns, nsteps, mode, top_k, t, softcap, rng, out_ids, split);
    return m->kv_dtype == CD_DTYPE_F16 ? run_samples<__nv_bfloat16, __half>(m, c, first, ns, nsteps, mode, top_k, t, softcap, rng, out_ids, split)
                                       : run_samples<__nv_bfloat16, __nv_bfloat16>(m, c, first, ns, nsteps, mode, top_k, t, softcap, rng, out_ids, split);
}

int prefill_batched(cd_model* m, size_t n) {
    PrefillCtx* c = nullptr;
    int rc = get_ctx(m, &c, true, true);
    if (rc) return rc;
    const int dt = m->opt.weight_dtype;
    // CD_PREFILL=fast: one 16-bit rounding of every GEMM input (about 1 % of the logit range at 5B);
    // default: hi + lo pairs, which keeps the prompt pass within the decode path's distance of the oracle
    const char* mode = getenv("CD_PREFILL");
    const bool split = !(mode && !strcmp(mode, "fast"));
    if (dt == CD_DTYPE_F16) return run<__half, __half>(m, c, n, split);
    // bf16 and FP8 linears: bf16 activations and head; the cache is fp16 or bf16
    return m->kv_dtype == CD_DTYPE_F16 ? run<__nv_bfloat16, __half>(m, c, n, split) : run<__nv_bfloat16, __nv_bfloat16>(m, c, n, split);
}

const float* prefill_hidden_row(const cd_model* m, size_t i) {
    return static_cast<const PrefillCtx*>(m->prefill_ctx)->x + i * (size_t)m->cfg.dim;
}

void prefill_release(cd_model* m) {
    PrefillCtx* c = (PrefillCtx*)m->prefill_ctx;
    if (!c) return;
    for (auto& kv : c->s_graphs) cudaGraphExecDestroy(kv.second);
    for (void* ptr : {(void*)c->x, c->xn, c->q, c->gate, (void*)c->s_arena, c->f8_qkv, c->f8_o, c->f8_13, c->f8_2}) if (ptr) cudaFree(ptr);
    delete c;
    m->prefill_ctx = nullptr;
}

}  // namespace cd
