// Launching the persistent decode kernel; each storage type is instantiated in a file of its own (mega_*.cu), so that they
// compile side by side.
#pragma once
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "step.cuh"
#include "mega_launch.h"

namespace {
using namespace cd;

// ------------------------------------------------------------------ persistent kernel launch
template <typename WT, typename LT, typename KT, int ND, int NH, bool TPAR, bool GROUPED>
cudaError_t launch_mega_t(cd_model* m, int input_embed, int want_logits) {
    constexpr MegaRows Q = std::is_same<LT, Int4G32>::value ? MEGA_INT4 : std::is_same<LT, Fp8Row>::value ? MEGA_FP8 : MEGA_PLAIN;
    constexpr int RD = mega_stage_rows(ND, Q), RH = mega_stage_rows(NH, Q), RO = mega_head_rows(ND, Q);
    constexpr int NO = Q != MEGA_PLAIN ? 2 * ND : ND;  // a quantised chunk is twice as many elements as one of the head's
    const cd_config& c = m->cfg;
    auto kern = decode_mega_kernel<WT, LT, KT, ND, RD, NH, RH, NO, RO, TPAR, GROUPED>;
    // every CTA owns rows of every matrix: what tells a CTA that another one is done with a vector is that one's next rows
    const int grid = TPAR ? m->sm_count : std::min({m->sm_count, c.dim, c.hidden, (c.q_dim + 2 * c.kv_dim) / 2});
    const size_t stage_cap = mega_stage_bytes(ND, NH, Q, Wfmt<LT>::row_stride(std::max(c.dim, c.q_dim)), Wfmt<LT>::row_stride(c.hidden), (size_t)c.dim * sizeof(WT));
    int max_rows = 0;
    for (int n : {c.q_dim + 2 * c.kv_dim, c.dim, 2 * c.hidden, want_logits ? m->v_loc : 0}) max_rows = std::max(max_rows, n / grid + 2);
    const int xs_dim = TPAR ? std::max(c.q_dim, c.dim) : std::max({c.q_dim, c.dim, c.hidden});
    // (the residual entries are the CTA's rows of Wo and W2, not of the LM head: with 128 k rows of it those are 866 a CTA)
    const int rows_cap = (max_rows + 3) & ~3, resid_cap = (c.dim / grid + 2 + 3) & ~3;
    size_t off = 0;
    auto carve = [&](size_t bytes) { const size_t o = off; off += (bytes + 15) / 16 * 16; return o; };
    const size_t xs_off = carve((size_t)xs_dim * 4), partial_off = carve((size_t)rows_cap * (GEMV_CONSUMERS / 32) * 4), resid_off = carve((size_t)2 * resid_cap * 4),
                 pt_off = carve((size_t)m->pages_per_seq * 4), layers_off = carve((size_t)c.nlayers * sizeof(MegaLayer)), bars_off = carve(2 * 16 * 8);
    // One GPU: all that a CTA can have (with 220 KB, as the kernels per operator use, hidden 11968 to 12288 had four stages, not six;
    // 6 layers of 3648 x 11968, 40 positions, 493 and 458 us).  But eight chunks of W2's rows a thread spill 200 to 360 bytes of
    // registers a thread, which the L1 holds as long as shared memory takes no more than 196 KB (60 KB of L1, 28 KB behind that): 5
    // layers of dim 4096, 1000 positions, here and per operator: hidden 13312 (195 KB) 520 and 562 us, 13824 (202 KB) 574 and 567 us.
    const size_t budget = TPAR || m->opt.test_ring_kb > 0 ? (size_t)m->ring_kb * 1024 : NH == 8 ? (size_t)195 * 1024 : m->smem_per_block;
    // (MegaShared as the compiler laid it out: with sizeof in its place a ring that just fits asked for 96 bytes too many)
    static const size_t fixed = [&] {
        cudaFuncAttributes fa;
        return cudaFuncGetAttributes(&fa, kern) == cudaSuccess ? (size_t)fa.sharedSizeBytes : sizeof(MegaShared) + 1024;
    }();
    // (a ring of two stages loses to the kernels per operator: FP8, 5 layers of 4096 x 16384, 200 positions, 541 and 424 us)
    if (fixed + off + (TPAR ? 2 : 4) * stage_cap > budget) return cudaErrorNotSupported;
    const int nstages = (int)std::min<size_t>(16, (budget - fixed - off) / stage_cap) & ~1;  // even: slots alternate between the two consumer groups
    const size_t ring = (size_t)nstages * stage_cap, smem = ring + off;
    cudaError_t e = allow_shared_memory((const void*)kern);
    if (e != cudaSuccess) return e;
    MegaParams p;
    p.layers = (const MegaLayer*)m->mega_layers;
    p.embed = m->embed; p.lm_head = m->lm_head; p.gamma_final = m->gamma_final;
    p.x_a = m->x_a; p.x_b = m->x_b; p.q = m->q; p.gate = m->gate; p.logits = m->logits; p.norm_final = m->norm_final;
    {
        unsigned long long* t = (unsigned long long*)m->mega_tagged;
        p.tx_a = t; p.tx_b = p.tx_a + c.dim; p.tq = p.tx_b + c.dim; p.tkv = p.tq + c.q_dim; p.tgate = p.tkv + 2 * c.kv_dim; p.tparts = p.tgate + c.hidden;
    }
    p.part_acc = m->part_acc; p.part_ml = m->part_ml; p.grid_counter = m->grid_counter;
    p.st = m->st; p.page_table = m->page_table; p.rope = m->rope;
    p.dim = c.dim; p.hidden = c.hidden; p.heads = c.heads; p.kv_heads = c.kv_heads; p.hd = c.hd; p.nlayers = c.nlayers;
    p.vocab = m->v_loc; p.embed_rows = m->full_cfg.vocab; p.q_dim = c.q_dim; p.kv_dim = c.kv_dim; p.gqa = c.gqa_ratio; p.page_tokens = m->page_tokens;
    p.activation = m->opt.activation; p.alpha = m->alpha; p.attn_scale = 1.0f / std::sqrt((float)c.hd);
    p.trace = m->mega_trace;
    p.npages = m->pages_per_seq;
    p.tile_tokens = mega_tile_tokens(m->page_tokens, (size_t)c.hd * sizeof(KT), stage_cap);
    p.wait_ns = m->wait_ns;
    p.tp = m->tp;  // world <= 1 on one GPU
    p.tp.wait_ns = m->wait_ns;
    p.off_xs = ring + xs_off; p.off_partial = ring + partial_off; p.off_resid = ring + resid_off; p.off_pt = ring + pt_off; p.off_layers = ring + layers_off;
    p.off_bars = ring + bars_off;
    p.nstages = nstages; p.stage_cap = (uint32_t)stage_cap; p.rows_cap = rows_cap; p.resid_cap = resid_cap; p.input_embed = input_embed; p.want_logits = want_logits;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(grid);
    lc.blockDim = dim3(MEGA_THREADS);
    lc.dynamicSmemBytes = smem;
    lc.stream = m->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;  // all CTAs resident: they wait for one another
    at[0].val.cooperative = 1;
    lc.attrs = at;
    lc.numAttrs = 1;
    e = cudaLaunchKernelEx(&lc, kern, p);
    count_launch(m);
    return e;
}

template <typename WT, typename LT, typename KT, bool TPAR, bool GROUPED>
cudaError_t launch_mega_tp(cd_model* m, int input_embed, int want_logits) {
    switch (m->mega_nd * 10 + m->mega_nh) {
        case 11: return launch_mega_t<WT, LT, KT, 1, 1, TPAR, GROUPED>(m, input_embed, want_logits);
        case 12: return launch_mega_t<WT, LT, KT, 1, 2, TPAR, GROUPED>(m, input_embed, want_logits);
        case 14: if constexpr (!TPAR) return launch_mega_t<WT, LT, KT, 1, 4, TPAR, GROUPED>(m, input_embed, want_logits); else break;
        case 13: if constexpr (Wfmt<LT>::QUANT) return launch_mega_t<WT, LT, KT, 1, 3, TPAR, GROUPED>(m, input_embed, want_logits); else break;
        case 24: return launch_mega_t<WT, LT, KT, 2, 4, TPAR, GROUPED>(m, input_embed, want_logits);
        case 26: if constexpr (!Wfmt<LT>::QUANT) return launch_mega_t<WT, LT, KT, 2, 6, TPAR, GROUPED>(m, input_embed, want_logits); else break;
        case 28: if constexpr (!TPAR && !Wfmt<LT>::QUANT) return launch_mega_t<WT, LT, KT, 2, 8, TPAR, GROUPED>(m, input_embed, want_logits); else break;
        default: break;
    }
    return cudaErrorInvalidConfiguration;
}
}  // namespace

namespace cd {

template <typename WT, typename LT, typename KT>
cudaError_t launch_mega(cd_model* m, int input_embed, int want_logits) {
    if constexpr (!std::is_same<WT, float>::value && !Wfmt<LT>::QUANT) {  // the tensor-parallel form exists for the 16-bit storage types
        if (m->tp_world > 1) return launch_mega_tp<WT, LT, KT, true, false>(m, input_embed, want_logits);
    }
    if constexpr (std::is_same<KT, __half>::value) {
        if (m->cfg.gqa_ratio > 2) return launch_mega_tp<WT, LT, KT, false, true>(m, input_embed, want_logits);
    }
    return launch_mega_tp<WT, LT, KT, false, false>(m, input_embed, want_logits);
}

}  // namespace cd
