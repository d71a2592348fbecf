// One persistent kernel per decoded token.
//
// The multi-kernel path pays a fixed 4-6 us at each of its 5 x nlayers kernel boundaries
// (drain, launch, ring refill) during which HBM idles.  Here one cooperative grid of one
// CTA per SM walks the whole token.  Its producers stream, layer after layer and
// through one shared-memory ring of 1-D bulk copies, everything this CTA will read from
// HBM in the order it will need it: its rows of the q|k|v matrix, the K/V tiles of the
// cached positions its attention work covers, its rows of Wo, W1|W3 and W2 - and never
// stops at an operator boundary, because none of that depends on this token's activations
// (the one K/V row that does, the current position's, reaches the consumers as tagged words).  Sixteen consumer warps run the operators in order; a vector
// that the next operator needs whole (five times per layer) reaches every CTA as tagged words,
// which it polls for (tag_store below).  While consumers wait for them the ring keeps filling,
// so HBM stays busy.
//
// Phases of a layer (same arithmetic and epilogues as the stand-alone kernels):
//   1 RMSNorm + q|k|v GEMV + RoPE + KV append
//   2 attention: every kv head belongs to a few CTAs, each of which takes a contiguous
//     run of tiles of cached positions out of the ring (already resident: they were
//     requested while phase 1 ran), keeps a running softmax per warp or team of
//     warps, merges them in shared memory and stores ONE partial (max, sum, weighted V)
//     per q head
//   3 every CTA merges the few partials of every head (fixed order: deterministic, no
//     atomics, nobody waits for a "last arriver"), then Wo GEMV + scaled residual
//   4 RMSNorm + W1|W3 GEMV + gate
//   5 W2 GEMV + scaled residual
// then the final RMSNorm + LM head into the logits buffer; the per-block head reductions
// and samplers run as the small kernels they already are.
//
// Tensor parallel (TpLink::world > 1): every rank runs this kernel on its shard (its heads, its FFN columns,
// its LM-head rows).  The Wo and W2 phases push their partial vectors into every rank's inbox from the
// epilogue, and the phase that follows takes its input from the inbox - it polls (bounded by time) until
// all ranks' words are there and adds them in rank order - so the exchange needs no grid barrier of its
// own: behind Wo and W2 a CTA-local barrier is enough, three grid barriers per layer remain.
//
// Every wait (mbarrier, grid barrier) is bounded: on expiry the CTA records an error in
// DevState::error, stops working and leaves, and so does every other CTA when its own
// wait runs out.  No reference counterpart (the reference encodes 15 dispatches per layer,
// lib.rs:513-634).
#pragma once
#include <type_traits>

#include "kernels.cuh"

namespace cd {

struct MegaLayer {
    const void *wqkv, *wo, *w13, *w2;
    const float *gamma1, *gamma2;
    void* kv;
};

constexpr int MEGA_MAX_PARTS = 64;  // partial attention results per head the buffers hold
constexpr int MEGA_CPH_CAP = 8;     // CTAs that share a kv head: every CTA merges that many partials per head before Wo
constexpr int MEGA_MAX_GQA = 8;     // q heads per kv head: 1 or 2 (attention_phase), 4 or 8 (attention_grouped)

struct MegaParams {
    const MegaLayer* layers;  // device array [nlayers]
    const void* embed;
    const void* lm_head;
    const float* gamma_final;
    float *x_a, *x_b, *q, *gate, *logits, *norm_final;
    float *part_acc, *part_ml;         // [heads][MEGA_MAX_PARTS][hd], [heads][MEGA_MAX_PARTS][2]
    unsigned long long* grid_counter;  // monotonic: arrivals at the grid barrier (tensor parallel), CTAs started (one GPU)
    DevState* st;
    const int* page_table;
    const float2* rope;
    int dim, hidden, heads, kv_heads, hd, nlayers, vocab, q_dim, kv_dim, gqa, page_tokens, activation;
    int embed_rows;       // rows of the embedding table (vocab above is the LM-head rows this rank holds)
    float alpha, attn_scale;
    int nstages;
    uint32_t stage_cap;   // bytes per ring stage
    int rows_cap;         // rows a CTA may own in any phase
    int resid_cap;        // of them, rows of the residual stream
    int input_embed;      // 1: x = embed[st->token]; 0: x already in x_a
    int want_logits;
    int npages;                 // page-table entries of the sequence
    int tile_tokens;            // cached positions per attention tile (divides page_tokens; a K tile fits one ring stage)
    unsigned long long wait_ns; // bound of a grid-barrier wait
    unsigned long long* trace;  // optional [2][1 + 10 * nlayers + 1] globaltimer stamps of CTA 0 and the last CTA: start, two per phase of a layer, end
    TpLink tp;                  // tensor parallel (world > 1): the dimensions above are this rank's shard
    // byte offsets in dynamic shared memory, behind the ring: widest input vector, [rows_cap][8] partial sums, [2][resid_cap] residual
    // entries, page table, [nlayers] layer table, barriers.  (Offsets as kernel parameters and the rest of the CTA's scratch as
    // static shared memory cost no registers; with a pointer each the GEMV loops spilled, and at 640 threads a CTA's spills
    // do not fit the L1 that the ring leaves.)
    uint32_t off_xs, off_partial, off_resid, off_pt, off_layers, off_bars;
    // one GPU: the vectors between phases as tagged words (tag_store); tparts: [heads][MEGA_CPH_CAP][hd + 2], max and sum last
    unsigned long long *tx_a, *tx_b, *tq, *tkv, *tgate, *tparts;
};

// Wo / W2 epilogue: x_out = res + alpha y on one GPU; tensor parallel, the rank's partial y goes to every rank's
// inbox instead (EpiPush) and the phase that consumes it adds the residual.
static __device__ __noinline__ void push_partial(const TpLink& tp, int ar_out, int unit, float y) {
    const unsigned int seq = __ldcg(&tp.st->ar_base) + (unsigned int)ar_out;
    const size_t at = ((size_t)(seq % 3u) * tp.world + tp.rank) * tp.dim + unit;
    const float v = tp_sanitize(y);
    for (int r = 0; r < tp.world; ++r) reinterpret_cast<float*>(tp.peers[r])[at] = v;
}
struct EpiPushPartial {  // Wo / W2 under tensor parallelism: the rank's partial row to every rank's inbox as all-reduce ar_out
    const TpLink* tp;
    int ar_out;
    __device__ void operator()(int unit, const float (&y)[1]) const { push_partial(*tp, ar_out, unit, y[0]); }
};

// Two groups of eight consumer warps take alternate ring stages: a stage's latency chain
// (shared-memory loads, FMA chain, shuffle reduction) is long, and only with two stages
// in progress do the consumers drain the ring clearly faster than HBM fills it, which is
// what lets them catch up after every barrier.
constexpr int MEGA_GROUPS = 2;
constexpr int MEGA_CONSUMERS = MEGA_GROUPS * GEMV_CONSUMERS;
// + the producers, one working thread each: one alone took 0.3 us per stage (its wait, its copy, the walk), 54 GB/s per SM at
// 16 KB stages and less at smaller ones.  Twenty warps take no more registers than seventeen.
constexpr int MEGA_PRODUCERS = 4;
constexpr int MEGA_THREADS = MEGA_CONSUMERS + 32 * MEGA_PRODUCERS;
constexpr int MEGA_TEAMS = MEGA_CONSUMERS / 128;
constexpr int MEGA_TEAM_SMEM = 128 * 8 + 64;  // floats per team: lane-group accumulators, then (max, sum) pairs
// ---- who computes which part of the attention
// A kv head belongs to `cph` consecutive CTAs (as many as fit, at most one per tile and at most
// MEGA_CPH_CAP); CTA j of them takes tiles [j * ntiles / cph, (j + 1) * ntiles / cph) and
// produces partial j of every q head of that kv head.  With more kv heads than CTAs each CTA
// walks heads blockIdx.x, blockIdx.x + gridDim.x, ... on its own (cph = 1).
struct AttnPlan {
    int cph;          // CTAs (= partials) per kv head
    int first, step;  // this CTA's kv heads: first, first + step, ... (first < 0: none)
    int part;         // this CTA's partial index within its head
    int t0, t1;       // its tiles
};
struct MegaShared {
    float accs[MEGA_TEAMS][MEGA_TEAM_SMEM];  // attention: lane-group accumulators, then (max, sum) pairs
    float tparts[MEGA_TEAMS][2][128 + 2];    // per team and q head: weighted V, max, sum
    float q[MEGA_MAX_GQA * 128];             // q of the kv head's q heads
    uint4 row[2 * 128 / 4];                  // this position's K and V row as cached
    float2 rope[64];                         // (cos, sin) of this position
    float red[64];
    AttnPlan plan;
    int2 rows[5];                            // this CTA's rows of q|k|v, the residual stream, gate|up; [4] the head
    size_t kv_at;                            // this position's K row of kv head 0 in a layer's pages (elements)
    unsigned long long launch;               // one GPU: launches of this model ahead of this one
    int abort;
};
__device__ inline MegaShared& mega_shared() {
    __shared__ MegaShared sh;
    return sh;
}
__device__ inline unsigned char* mega_dyn() {
    extern __shared__ __align__(128) unsigned char smraw[];
    return smraw;
}
__device__ inline bool mega_aborted() { return *const_cast<const volatile int*>(&mega_shared().abort) != 0; }

__device__ inline void mega_bar() { asm volatile("bar.sync 1, 512;" ::: "memory"); }
__device__ inline void group_bar(int grp) { asm volatile("bar.sync %0, 256;" ::"r"(4 + grp) : "memory"); }
__device__ inline void team_bar(int team) { asm volatile("bar.sync %0, 128;" ::"r"(8 + team) : "memory"); }
__device__ inline float group_sum(float v, float* red, int grp) {
    const int lane = threadIdx.x & 31, warp = (threadIdx.x & 255) >> 5;
    v = warp_sum(v);
    group_bar(grp);
    if (lane == 0) red[warp] = v;
    group_bar(grp);
    float t = 0.0f;
#pragma unroll
    for (int i = 0; i < GEMV_CONSUMERS / 32; ++i) t += red[i];
    return t;
}
// mbarrier wait that gives up after budget_ns, or at once when the CTA's abort flag is up: the waits of a CTA that is
// leaving (its ring may never be filled or drained again) must not each run for the seconds mbar_wait allows
__device__ inline bool mbar_wait_or_abort(uint32_t bar, uint32_t parity, const int* abort_flag, unsigned long long budget_ns) {
    unsigned long long t0 = 0;
    for (int i = 0;; ++i) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
        if (abort_flag != nullptr && *reinterpret_cast<const volatile int*>(abort_flag) != 0) return false;
        if ((i & 15) == 15) {
            const unsigned long long now = global_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > budget_ns) return false;
        }
    }
}
__device__ inline void mbar_arrive_n(uint32_t bar, uint32_t n) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(bar), "r"(n) : "memory");
}

struct Ring {
    uint32_t base, full0, empty0, stage_cap;
    int nstages;
    // the next stage's slot and the parity of its turn, kept by increments: a division per stage was a third of the
    // consumers' latency per stage (producer and consumers count the same sequence)
    int slot;
    uint32_t turn;
    __device__ void advance(int n) {
        for (slot += n; slot >= nstages; slot -= nstages) turn ^= 1u;
    }
};

// rows [r0, r1) of an [N, K] matrix owned by this CTA
__device__ inline void cta_rows(int N, int unit, int& r0, int& r1) {
    const int nunits = N / unit;
    r0 = (int)((long long)blockIdx.x * nunits / gridDim.x) * unit;
    r1 = (int)((long long)(blockIdx.x + 1) * nunits / gridDim.x) * unit;
}

__device__ inline AttnPlan attn_plan(int kv_heads, int ntiles) {
    AttnPlan a;
    const int G = gridDim.x, c = blockIdx.x;
    if (kv_heads <= G) {
        a.cph = max(1, min(min(G / kv_heads, ntiles), MEGA_CPH_CAP));
        a.first = c < kv_heads * a.cph ? c / a.cph : -1;
        a.step = kv_heads;  // one head only
        a.part = c % a.cph;
    } else {
        a.cph = 1;
        a.first = c;
        a.step = G;
        a.part = 0;
    }
    a.t0 = (int)((long long)a.part * ntiles / a.cph);
    a.t1 = (int)((long long)(a.part + 1) * ntiles / a.cph);
    return a;
}

// ---- the token's stream: everything this CTA reads from HBM for one token, stage by stage, in the
// order the consumers use it: its rows of q|k|v, the K and V tiles of its attention work (one stage each, K before V),
// its rows of Wo, W1|W3 and W2, layer after layer, then of the LM head.  f(src, bytes, is_kv) is called once per ring
// stage; false stops the walk.  (One call of f: its wait loop inlined per segment was a quarter of the kernel's code.)
template <int RD, int RH, int RO, class F>
__device__ inline bool walk_token_stream(const MegaParams& p, const MegaLayer* layers, const int* pt, uint32_t rb_d, uint32_t rb_q, uint32_t rb_h, uint32_t rb_o, uint32_t kes, F& f) {
    const MegaShared& sh = mega_shared();
    const AttnPlan plan = sh.plan;
    const int T = p.tile_tokens, tpp = p.page_tokens / T;  // tiles per page
    const size_t head_bytes = (size_t)p.page_tokens * p.hd * kes, page_bytes = (size_t)2 * p.kv_heads * head_bytes, v_off = (size_t)p.kv_heads * head_bytes;
    const uint32_t tile_bytes = (uint32_t)T * p.hd * kes;
    for (int l = 0; l <= p.nlayers; ++l) {
        if (l == p.nlayers && !p.want_logits) break;
        const MegaLayer& L = layers[min(l, p.nlayers - 1)];
        for (int seg = 0; seg < (l < p.nlayers ? 5 : 1); ++seg) {
            const bool kv = l < p.nlayers && seg == 1;
            const char* base = nullptr;
            uint32_t step = tile_bytes, left = 0;  // bytes per stage, bytes of the whole segment
            int n, h = plan.first, pg = 0, sub = 0, t = plan.t0;
            if (kv) {
                n = 2 * (h < 0 ? 0 : (plan.t1 - plan.t0) * ((p.kv_heads - h + plan.step - 1) / plan.step));
                pg = t / tpp; sub = t % tpp;
            } else {
                const bool head = l == p.nlayers;
                const int2 r = sh.rows[head ? 4 : seg == 0 ? 0 : seg == 3 ? 2 : 1];
                const uint32_t rb = head ? rb_o : seg == 0 || seg == 3 ? rb_d : seg == 2 ? rb_q : rb_h;
                const int R = head ? RO : seg == 4 ? RH : RD;
                base = reinterpret_cast<const char*>(head ? p.lm_head : seg == 0 ? L.wqkv : seg == 2 ? L.wo : seg == 3 ? L.w13 : L.w2) + (size_t)r.x * rb;
                n = (r.y - r.x + R - 1) / R;
                step = (uint32_t)R * rb;
                left = (uint32_t)(r.y - r.x) * rb;
            }
            for (int i = 0; i < n; ++i) {
                const char* src = base;
                uint32_t bytes = step;
                if (kv) {  // page and offset advance by increments instead of a division per tile
                    src = reinterpret_cast<const char*>(L.kv) + (size_t)h * head_bytes + (size_t)pt[pg] * page_bytes + (size_t)sub * tile_bytes + ((i & 1) ? v_off : 0);
                    if (i & 1) {
                        if (++sub == tpp) { sub = 0; ++pg; }
                        if (++t == plan.t1) { h += plan.step; t = plan.t0; pg = t / tpp; sub = t % tpp; }
                    }
                } else {
                    bytes = min(step, left);
                    base += step;
                    left -= bytes;
                }
                if (!f(src, bytes, kv)) return false;
            }
        }
    }
    return true;
}

// ---- tensor parallel: the CTA's input vector x = res + alpha * (sum over the ranks, in rank order, of all-reduce
// in_reduce), gathered from this rank's inbox into shared memory (xg), every thread a few float4 positions; both
// consumer groups then take their slices from there, CTA 0 keeps the vector in x_out.  Out of line: one copy for
// all phases, and none of it in the instruction stream of a single-GPU token.
static __device__ __noinline__ void gather_input(const TpLink& tin, int K, float* xg, int* err) {
    const unsigned int seq = __ldcg(&tin.st->ar_base) + (unsigned int)tin.in_reduce;
    float* base = reinterpret_cast<float*>(tin.peers[tin.rank]);
    const float* inbox = base + (size_t)(seq % 3u) * tin.world * tin.dim;
    // re-arm the slot two all-reduces ahead (nobody reads or writes it now), split over the CTAs
    uint4* rearm = reinterpret_cast<uint4*>(base + (size_t)((seq + 2u) % 3u) * tin.world * tin.dim);
    const int n4 = tin.world * tin.dim / 4;
    for (int j = blockIdx.x * MEGA_CONSUMERS + threadIdx.x; j < n4; j += gridDim.x * MEGA_CONSUMERS)
        rearm[j] = make_uint4(TP_SENTINEL, TP_SENTINEL, TP_SENTINEL, TP_SENTINEL);
    for (int q4 = threadIdx.x; q4 < K / 4; q4 += MEGA_CONSUMERS) {
        float4 a;  // summed in fixed rank order: identical on every rank
        if (!tp_gather4(inbox, tin.world, tin.dim, (size_t)q4 * 4, a, tin.st, tin.wait_ns)) {
            atomicCAS(err, 0, DEV_ERR_TP_WAIT);
            mega_shared().abort = 1;
        }
        const float4 r4 = __ldcg(reinterpret_cast<const float4*>(tin.res + (size_t)q4 * 4));
        const float4 v = make_float4(r4.x + tin.alpha * a.x, r4.y + tin.alpha * a.y, r4.z + tin.alpha * a.z, r4.w + tin.alpha * a.w);
        *reinterpret_cast<float4*>(xg + (size_t)q4 * 4) = v;
        if (blockIdx.x == 0) *reinterpret_cast<float4*>(tin.x_out + (size_t)q4 * 4) = v;
    }
    mega_bar();
}

// ---- tensor parallel, first layer: the token's input vector (the embedding row of st->token, which CTA 0 also
// stores as fp32 in x_a, or x_a itself) into shared memory, so that every phase of such a kernel reads its input there
template <typename WT>
__device__ __noinline__ void stage_first_input(const MegaParams& p, float* xs) {
    constexpr int EPC = Elem<WT>::EPC;
    if (p.input_embed) {
        const WT* row = reinterpret_cast<const WT*>(p.embed) + (size_t)checked_token(__ldcg(&p.st->token), p.embed_rows, &p.st->error) * p.dim;
        for (int c = threadIdx.x; c < p.dim / EPC; c += MEGA_CONSUMERS) {
            float f[EPC];
            Elem<WT>::unpack(ldg_stream(reinterpret_cast<const char*>(row) + (size_t)c * 16), f);
#pragma unroll
            for (int e = 0; e < EPC; e += 4) {
                const float4 v = make_float4(f[e], f[e + 1], f[e + 2], f[e + 3]);
                *reinterpret_cast<float4*>(xs + (size_t)c * EPC + e) = v;
                if (blockIdx.x == 0) *reinterpret_cast<float4*>(p.x_a + (size_t)c * EPC + e) = v;
            }
        }
    } else {
        for (int q4 = threadIdx.x; q4 < p.dim / 4; q4 += MEGA_CONSUMERS)
            *reinterpret_cast<float4*>(xs + (size_t)q4 * 4) = __ldcg(reinterpret_cast<const float4*>(p.x_a + (size_t)q4 * 4));
    }
    mega_bar();
}

template <typename LT> struct RowChunks {  // this thread's 16-byte chunks of a stage's rows
    uint32_t base, row_bytes;
    int nchunks;
    __device__ uint4 operator()(int j, int i) const {
        const int c = (threadIdx.x & 255) + i * GEMV_CONSUMERS;
        return c < nchunks ? lds128(base + (uint32_t)j * row_bytes + (uint32_t)c * 16u) : make_uint4(0, 0, 0, 0);
    }
};
// ---- the input slice a thread holds (chunks tid, tid + 256, ... of the vector, the same in both groups), and the rows of
// a stage times it
template <typename LT, int NITER> struct Slices {
    static constexpr int EPC = Wfmt<LT>::EPC;
    float x[NITER][EPC];
    __device__ void set(int i, int e, float4 v) { x[i][e] = v.x; x[i][e + 1] = v.y; x[i][e + 2] = v.z; x[i][e + 3] = v.w; }
    // chunk i of row j of the stage at `base`; all of them are in registers when release() hands the stage back
    template <int R, class Release> __device__ void rows(uint32_t base, uint32_t row_bytes, int K, const Release& release, float (&acc)[R]) const {
        const RowChunks<LT> load{base, row_bytes, K / EPC};
        uint4 w[R][NITER];
#pragma unroll
        for (int j = 0; j < R; ++j)
#pragma unroll
            for (int i = 0; i < NITER; ++i) w[j][i] = load(j, i);
        release();
#pragma unroll
        for (int j = 0; j < R; ++j) {
            float a = 0.0f;
#pragma unroll
            for (int i = 0; i < NITER; ++i) a = Wfmt<LT>::dot(w[j][i], 0u, x[i], a);
            acc[j] = a;
        }
    }
};
// Quantised rows on the tensor cores (mma.m16n8k16; with an fp32 FMA per weight the decoder was bound by issue slots).  Weights
// widen to fp16 exactly; inputs are fp16 pairs hi + lo, rounded to nearest, of x times a power of two that brings the largest of
// the vector to 2^14: off by at most 2^-23 of x (three of four fp32 values are exact), or by 2^-39 of the largest where that is
// more.  Products are exact, sums fp32.  Chunks stay where they are in the row: lane (g, t) = lane / 4, lane % 4 puts its own
// weights of two matrix rows into rows g and g + 8 of A: quad g holds chunk g % 4 of rows j + g / 4 and j + 2 + g / 4.  Column
// 2 c of B is the hi, 2 c + 1 the lo part of chunk c's inputs, so that element (g, 2 (g % 4)) + (g, 2 (g % 4) + 1), which lane
// t = g % 4 holds, is the sum over quad g's chunk; the others are not used.  256 weights per MMA; two MMAs for hi and lo over
// eight chunks of two rows (128 weights each) took 15.4 us for the 90 MB of the 5B model's W1|W3 in FP8, HBM 14 us.
struct QuantLane {
    static __device__ int warp() { return (threadIdx.x & 255) >> 5; }
    static __device__ int g() { return (threadIdx.x & 31) >> 2; }
    static __device__ int t() { return threadIdx.x & 3; }
    // the quad's sums of an MMA's result d, rows j .. j + 3 (or two of them), into acc: lanes that hold none add zero
    template <int R> static __device__ void take(int j, float lower, float upper, float (&acc)[R]) {
        const bool mine = t() == (g() & 3), second = g() >= 4;
        acc[j] = mine && !second ? lower : 0.0f;
        acc[j + 1] = mine && second ? lower : 0.0f;
        if (R > 2) {
            acc[R > 2 ? j + 2 : 0] = mine && !second ? upper : 0.0f;
            acc[R > 2 ? j + 3 : 0] = mine && second ? upper : 0.0f;
        }
    }
    // the hi (even columns) or lo part of two inputs
    static __device__ uint32_t part(float a, float b) {
        const uint32_t hi = Mma16<__half>::part(a, b), lo = Mma16<__half>::part(a, b);
        return g() & 1 ? lo : hi;
    }
};
// FP8: a chunk is 64 bytes, 16 a lane
template <int NITER> struct Slices<Fp8Row, NITER> {
    static constexpr int STEPS = 2 * NITER;
    uint32_t x[STEPS][8];
    __device__ static int lane_chunk(int i, int c) { return ((i * (GEMV_CONSUMERS / 32) + QuantLane::warp()) * 4 + c) * 4 + QuantLane::t(); }
    __device__ void fill(const float* xs, float inv, float up, int K) {
#pragma unroll
        for (int i = 0; i < STEPS; ++i) {
            const int at = 16 * lane_chunk(i, QuantLane::g() >> 1);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float4 v = at < K ? *reinterpret_cast<const float4*>(xs + at + 4 * e) : make_float4(0.f, 0.f, 0.f, 0.f);
                x[i][2 * e] = QuantLane::part(v.x * inv * up, v.y * inv * up);
                x[i][2 * e + 1] = QuantLane::part(v.z * inv * up, v.w * inv * up);
            }
        }
    }
    __device__ static uint32_t widen(uint32_t two) {
        const __half2 h(__nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)two, __NV_E4M3));
        return *reinterpret_cast<const uint32_t*>(&h);
    }
    template <int R, class Release> __device__ void rows(uint32_t base, uint32_t row_bytes, int K, const Release& release, float (&acc)[R]) const {
        static_assert(R == 2 || R == 4, "two or four rows");
        float d[2][4] = {};
#pragma unroll
        for (int i = 0; i < STEPS; ++i) {
            const int c = lane_chunk(i, QuantLane::g() & 3);
            const uint32_t at = base + (uint32_t)(QuantLane::g() >> 2) * row_bytes + (uint32_t)c * 16u;
            uint4 w0 = make_uint4(0, 0, 0, 0), w1 = w0;
            if (16 * c < K) {
                w0 = lds128(at);
                if (R == 4) w1 = lds128(at + 2u * row_bytes);
            }
            const uint32_t u[4] = {w0.x, w0.y, w0.z, w0.w}, v[4] = {w1.x, w1.y, w1.z, w1.w};
#pragma unroll
            for (int k = 0; k < 4; ++k)
                Mma16<__half>::mma(d[k & 1], {widen(u[k] & 0xffffu), R == 4 ? widen(v[k] & 0xffffu) : 0u, widen(u[k] >> 16), R == 4 ? widen(v[k] >> 16) : 0u}, x[i][2 * k],
                                   x[i][2 * k + 1]);
        }
        release();
        QuantLane::take<R>(0, (d[0][0] + d[0][1]) + (d[1][0] + d[1][1]), (d[0][2] + d[0][3]) + (d[1][2] + d[1][3]), acc);
    }
};
// INT4 (groups of 32 with one fp16 scale): a chunk is a group, 4 bytes a lane; its sum times the group's scale in fp32.  A pair
// of nibbles n = q + 8 is masked out of its word into the mantissas of a pair of fp16 1024.0 (1024 + n, or 1024 + 16 n where it
// lies four bits up) and becomes q, exactly, with one more operation.  As the pair of subnormals that the mask alone gives (and the
// offset off the sums) that operation is saved, but an MMA aligns its products by their operands' exponents, and a subnormal's
// leading zeros count as digits: the FFN of one layer was off by 5e-6 to 1.2e-5 of its norm where fp32 FMAs leave 2.5e-6 to 8e-6
// (dims 256 to 1024, even and heavy-tailed inputs); with q the two are equal to 0.4 %.  Bound by issue slots: the 50 MB
// of the 5B model's W1|W3 take 16.4 us (14.6 as subnormals; 18.0 with a step's loads right ahead of their use), W2 10.6.
template <int NITER> struct Slices<Int4G32, NITER> {
    // Steps whose words are loaded ahead of the first one's product.  NEAR: a warp takes 16 groups at a time and quad c four
    // neighbours, whose scales are one load, in an order of its own, so that the words of the four quads lie in different banks
    // (W1|W3, with subnormals, 14.8 us, 16.2 without).  Longer rows take groups one by one: W2's 11008 inputs are not a whole
    // number of sixteens a warp, and the registers do not last (12.9 us against 10.5).
    static constexpr int STEPS = 4 * NITER, BATCH = 4, NEAR = NITER == 1 ? 4 : 1;
    uint32_t x[STEPS][4];
    __device__ static int first_group(int i, int c) { return ((i / NEAR * (GEMV_CONSUMERS / 32) + QuantLane::warp()) * 4 + c) * NEAR; }
    __device__ static int group_of(int i, int c) { return first_group(i, c) + ((i + c) & (NEAR - 1)); }
    __device__ void fill(const float* xs, float inv, float up, int K) {
#pragma unroll
        for (int i = 0; i < STEPS; ++i) {
            const int at = group_of(i, QuantLane::g() >> 1) * 32 + 8 * QuantLane::t();
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
            if (at < K) { a = *reinterpret_cast<const float4*>(xs + at); b = *reinterpret_cast<const float4*>(xs + at + 4); }
            x[i][0] = QuantLane::part(a.x * inv * up, a.y * inv * up);
            x[i][1] = QuantLane::part(a.z * inv * up, a.w * inv * up);
            x[i][2] = QuantLane::part(b.x * inv * up, b.y * inv * up);
            x[i][3] = QuantLane::part(b.z * inv * up, b.w * inv * up);
        }
    }
    // the pair of nibbles in bits 0-3 or 4-7 of the halves of a word: as fp16 1024 + n or 1024 + 16 n, and from there n - 8, exactly
    __device__ static uint32_t low(uint32_t w) {
        const uint32_t b = (w & 0x000F000Fu) | 0x64006400u;
        const __half2 q = __hsub2(*reinterpret_cast<const __half2*>(&b), __float2half2_rn(1032.0f));
        return *reinterpret_cast<const uint32_t*>(&q);
    }
    __device__ static uint32_t high(uint32_t w) {
        const uint32_t b = (w & 0x00F000F0u) | 0x64006400u;
        const __half2 q = __hfma2(*reinterpret_cast<const __half2*>(&b), __float2half2_rn(0.0625f), __float2half2_rn(-72.0f));
        return *reinterpret_cast<const uint32_t*>(&q);
    }
    template <int R, class Release> __device__ void rows(uint32_t base, uint32_t row_bytes, int K, const Release& release, float (&acc)[R]) const {
        static_assert(R == 2 || R % 4 == 0, "two rows, or fours");
        constexpr int SETS = (R + 3) / 4, P = R == 2 ? 1 : 2;  // of four rows; lane's rows of a set
        const int ngroups = K / 32, quad = QuantLane::g() & 3;
        const uint32_t row = base + (uint32_t)(QuantLane::g() >> 2) * row_bytes, scale = row + Wfmt<Int4G32>::scale_off(K);
        float sum[SETS][2] = {};
#pragma unroll
        for (int i0 = 0; i0 < STEPS; i0 += BATCH) {
            if (i0 > 0 && first_group(i0, 0) >= ngroups) break;  // the whole warp's groups lie behind the row
            uint32_t w[BATCH][SETS][2] = {};
            unsigned short s[BATCH][SETS][2] = {};
            uint2 s4[SETS][2] = {};
            if (NEAR == 4 && first_group(i0, quad) < ngroups) {
#pragma unroll
                for (int j = 0; j < SETS; ++j)
#pragma unroll
                    for (int k = 0; k < P; ++k)
                        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(s4[j][k].x), "=r"(s4[j][k].y)
                                     : "r"(scale + (uint32_t)(4 * j + 2 * k) * row_bytes + (uint32_t)first_group(i0, quad) * 2u));
            }
#pragma unroll
            for (int i = 0; i < BATCH; ++i) {
                const int group = group_of(i0 + i, quad);
                if (group < ngroups) {
#pragma unroll
                    for (int j = 0; j < SETS; ++j)
#pragma unroll
                        for (int k = 0; k < P; ++k) {
                            const uint32_t off = (uint32_t)(4 * j + 2 * k) * row_bytes;
                            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w[i][j][k]) : "r"(row + off + (uint32_t)group * 16u + 4u * QuantLane::t()));
                            if (NEAR == 1) asm volatile("ld.shared.u16 %0, [%1];" : "=h"(s[i][j][k]) : "r"(scale + off + (uint32_t)group * 2u));
                        }
                }
            }
#pragma unroll
            for (int i = 0; i < BATCH; ++i) {
                const uint32_t(&b)[4] = x[i0 + i];
                const uint32_t pick = 0x0010u + 0x0022u * (uint32_t)((i + quad) & 3);  // NEAR: this step's half of the four
                const bool in = group_of(i0 + i, quad) < ngroups;
                auto scale_of = [&](int j, int k) {
                    const uint32_t bits = NEAR == 1 ? s[i][j][k] : in ? __byte_perm(s4[j][k].x, s4[j][k].y, pick) : 0u;
                    return __half2float(__ushort_as_half((unsigned short)bits));
                };
#pragma unroll
                for (int j = 0; j < SETS; ++j) {
                    float d[4] = {0.f, 0.f, 0.f, 0.f};
                    const uint32_t u = w[i][j][0], v = P == 2 ? w[i][j][1] : 0u;
                    Mma16<__half>::mma(d, {low(u), P == 2 ? low(v) : 0u, high(u), P == 2 ? high(v) : 0u}, b[0], b[1]);
                    Mma16<__half>::mma(d, {low(u >> 8), P == 2 ? low(v >> 8) : 0u, high(u >> 8), P == 2 ? high(v >> 8) : 0u}, b[2], b[3]);
                    sum[j][0] = fmaf(d[0] + d[1], scale_of(j, 0), sum[j][0]);
                    if (P == 2) sum[j][1] = fmaf(d[2] + d[3], scale_of(j, 1), sum[j][1]);
                }
            }
        }
        release();
#pragma unroll
        for (int j = 0; j < SETS; ++j) QuantLane::take<R>(4 * j, sum[j][0], sum[j][1], acc);
    }
};

// ---- consumer side of one GEMV phase: this CTA's rows [r0, r1) out of the ring times the input slices, times `unscale` (a power
// of two, applied behind the row's scale: their product may be subnormal); a partial sum per row and warp of a group
template <typename LT, int NITER, int R>
__device__ inline void stream_partials(Ring& ring, const Slices<LT, NITER>& x, float unscale, int r0, int r1, int K, const MegaParams& p) {
    using F = Wfmt<LT>;
    float* partial = reinterpret_cast<float*>(mega_dyn() + p.off_partial);
    constexpr int NW = GEMV_CONSUMERS / 32;
    const int grp = threadIdx.x >> 8, tid = threadIdx.x & 255, lane = tid & 31, warp = tid >> 5;
    const uint32_t row_bytes = F::row_stride(K);
    const int ngroups = (r1 - r0 + R - 1) / R;

    // Ring slots are owned by groups for the whole GEMV phase: group = (global stage number) & 1,
    // and the ring has an even number of slots, so the successive uses of one slot are all
    // consumed, in order, by the same group.  (A parity wait can only tell adjacent phases of
    // an mbarrier apart; a group that skipped another group's use of a slot could mistake
    // an old phase for the one it wants.)
    const int g0 = (grp - ring.slot) & 1;
    Ring at = ring;
    at.advance(g0);
    for (int g = g0; g < ngroups; g += MEGA_GROUPS, at.advance(MEGA_GROUPS)) {
        const int s = at.slot;
        if (!mbar_wait(ring.full0 + 8u * s, at.turn)) {
            atomicCAS(&p.st->error, 0, DEV_ERR_FULL_WAIT);
            mega_shared().abort = 1;  // every consumer still meets at the barrier below, then all leave together
            break;
        }
        const uint32_t base = ring.base + (uint32_t)s * ring.stage_cap;
        float scale[R];
#pragma unroll
        for (int j = 0; j < R; ++j) {
            scale[j] = 1.0f;
            if (F::ROW_SCALE) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(scale[j]) : "r"(base + (uint32_t)j * row_bytes + F::scale_off(K)) : "memory");
        }
        float acc[R];
        x.template rows<R>(
            base, row_bytes, K,
            [&]() {
                __syncwarp();
                if (lane == 0) mbar_arrive_n(ring.empty0 + 8u * s, 2);  // a stage expects 16 arrivals: eight warps of one group, twice each
            },
            acc);
        if (F::ROW_SCALE) {
#pragma unroll
            for (int j = 0; j < R; ++j) acc[j] = acc[j] * scale[j] * unscale;
        } else if (F::QUANT) {
#pragma unroll
            for (int j = 0; j < R; ++j) acc[j] *= unscale;
        }
        int rr;
        const float tot = warp_reduce_rows<R>(acc, lane, rr);
        const int row = g * R + rr;
        if ((lane & (32 / R - 1)) == 0 && row < r1 - r0) partial[row * NW + warp] = tot;
    }
    ring.advance(ngroups);
}
// row r of the phase: the sums of its group's warps
__device__ inline float row_sum(const float* partial, int r) {
    float t = 0.0f;
#pragma unroll
    for (int w = 0; w < GEMV_CONSUMERS / 32; ++w) t += partial[r * (GEMV_CONSUMERS / 32) + w];
    return t;
}

// ---- one GEMV phase of the tensor-parallel form.  The input vector comes from `x` (fp32, L2-only loads), from
// `x_smem` (this CTA's shared memory).
template <typename WT, int NITER, int R, int UNIT, bool NORM, class Epi>
__device__ inline bool consume_gemv(Ring& ring, const float* x, const float* x_smem, const float* gamma, float* norm_out, int N, int K,
                                    const MegaParams& p, const Epi& epi) {
    constexpr int EPC = Elem<WT>::EPC;
    const int grp = threadIdx.x >> 8, tid = threadIdx.x & 255;
    const int nchunks = K / EPC;
    float* red = mega_shared().red + grp * 32;
    int r0, r1;
    cta_rows(N, UNIT, r0, r1);

    Slices<WT, NITER> slices;
    float(&xr)[NITER][EPC] = slices.x;
    float gm[NORM ? NITER : 1][NORM ? EPC : 1];  // gamma, requested together with x: one memory latency for both
    if (NORM) {
#pragma unroll
        for (int i = 0; i < NITER; ++i) {
            const int c = tid + i * GEMV_CONSUMERS;
#pragma unroll
            for (int e = 0; e < EPC; e += 4) {
                const float4 g = c < nchunks ? *reinterpret_cast<const float4*>(gamma + (size_t)c * EPC + e) : make_float4(0.f, 0.f, 0.f, 0.f);
                gm[NORM ? i : 0][NORM ? e : 0] = g.x; gm[NORM ? i : 0][NORM ? e + 1 : 0] = g.y;
                gm[NORM ? i : 0][NORM ? e + 2 : 0] = g.z; gm[NORM ? i : 0][NORM ? e + 3 : 0] = g.w;
            }
        }
    }
    float ss = 0.0f;
#pragma unroll
    for (int i = 0; i < NITER; ++i) {
        const int c = tid + i * GEMV_CONSUMERS;
#pragma unroll
        for (int e = 0; e < EPC; e += 4) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (c < nchunks) {
                if (x_smem != nullptr) v = *reinterpret_cast<const float4*>(x_smem + (size_t)c * EPC + e);
                else v = __ldcg(reinterpret_cast<const float4*>(x + (size_t)c * EPC + e));
            }
            xr[i][e] = v.x; xr[i][e + 1] = v.y; xr[i][e + 2] = v.z; xr[i][e + 3] = v.w;
            ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
        }
    }
    if (NORM) {
        const float tot = group_sum(ss, red, grp);
        const float inv = 1.0f / sqrtf(tot * (1.0f / (float)K) + RMS_EPS);
#pragma unroll
        for (int i = 0; i < NITER; ++i) {
            const int c = tid + i * GEMV_CONSUMERS;
            if (c < nchunks) {
#pragma unroll
                for (int e = 0; e < EPC; e += 4) {
                    xr[i][e] = xr[i][e] * inv * gm[NORM ? i : 0][NORM ? e : 0];
                    xr[i][e + 1] = xr[i][e + 1] * inv * gm[NORM ? i : 0][NORM ? e + 1 : 0];
                    xr[i][e + 2] = xr[i][e + 2] * inv * gm[NORM ? i : 0][NORM ? e + 2 : 0];
                    xr[i][e + 3] = xr[i][e + 3] * inv * gm[NORM ? i : 0][NORM ? e + 3 : 0];
                    if (norm_out != nullptr && blockIdx.x == 0 && grp == 0)
                        *reinterpret_cast<float4*>(norm_out + (size_t)c * EPC + e) =
                            make_float4(xr[i][e], xr[i][e + 1], xr[i][e + 2], xr[i][e + 3]);
                }
            }
        }
    }
    stream_partials<WT, NITER, R>(ring, slices, 1.0f, r0, r1, K, p);
    mega_bar();
    if (mega_aborted()) return false;
    const float* partial = reinterpret_cast<const float*>(mega_dyn() + p.off_partial);
    const int u0 = r0 / UNIT, nu = (r1 - r0) / UNIT;
#pragma unroll 1
    for (int u = threadIdx.x; u < nu; u += MEGA_CONSUMERS) {
        float y[UNIT];
#pragma unroll
        for (int k = 0; k < UNIT; ++k) y[k] = row_sum(partial, u * UNIT + k);
        epi(u0 + u, y);
    }
    return true;
}

// ---- one GPU: vectors between phases travel as tagged words.  A word is a 64-bit pair (value, tag), written by one
// relaxed store and read by relaxed loads, so a reader knows from the word itself that it holds this layer's value: no
// fence, no counter, no barrier, and the poll that sees the last word already has the data in registers.  A buffer is
// written once per layer; its readers of layer l are done before any CTA can write layer l + 1, because every CTA owns
// rows of every matrix and a CTA's rows of the next phase are stored only after it has read its whole input.
// (Against a grid barrier per phase - release reduction, acquire polls, then the loads: 2.8-3.0 us and the loads - a token of
// the 5B model takes 2.12 instead of 2.25 ms, of a 0.6B model of 24 layers 0.74 instead of 0.91 ms.)
__device__ inline void tag_store(unsigned long long* p, float v, uint32_t tag) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"((unsigned long long)tag << 32 | __float_as_uint(v)) : "memory");
}
__device__ inline void tag_load2(const unsigned long long* p, unsigned long long& a, unsigned long long& b) {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ inline float tag_value(unsigned long long w) { return __uint_as_float((uint32_t)w); }

// Polls the pairs of words at src[0 .. N - 1] until all carry `tag`.  False when the time is up or another CTA has
// already failed (the CTA's abort flag is raised then).
template <int N>
__device__ inline bool tag_poll(const unsigned long long* const (&src)[N], uint32_t tag, unsigned long long (&w)[N][2], const MegaParams& p) {
    unsigned long long t0 = 0;
#pragma unroll 1
    for (int i = 1;; ++i) {
#pragma unroll
        for (int b = 0; b < N; ++b) tag_load2(src[b], w[b][0], w[b][1]);
        bool all = true;
#pragma unroll
        for (int b = 0; b < N; ++b) all = all && (uint32_t)(w[b][0] >> 32) == tag && (uint32_t)(w[b][1] >> 32) == tag;
        if (all) return true;
        if ((i & 63) == 0) {
            const unsigned long long now = global_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > p.wait_ns || dev_failed(p.st) || mega_aborted()) break;
        }
    }
    atomicCAS(&p.st->error, 0, 3);
    mega_shared().abort = 1;
    return false;
}

// Where an input vector goes: times gamma (when given) into xs, and its entries at this CTA's rows of the residual stream
// as they are into resid (when given; two arrays take turns, since the epilogue of the phase before may still read the other).
struct InputTo {
    float *xs, *resid;
    const float* gamma;
    int2 rows;  // this CTA's rows of the residual stream
    __device__ float2 scale(int i) const { return gamma != nullptr ? *reinterpret_cast<const float2*>(gamma + i) : make_float2(1.0f, 1.0f); }
    __device__ void put(int i, float2 v, float2 g) const {
        *reinterpret_cast<float2*>(xs + i) = make_float2(v.x * g.x, v.y * g.y);
        if (resid != nullptr) {
            if (i >= rows.x && i < rows.y) resid[i - rows.x] = v.x;
            if (i + 1 >= rows.x && i + 1 < rows.y) resid[i + 1 - rows.x] = v.y;
        }
    }
};
// A whole vector from its tagged words; returns this thread's share of the sum of squares, and the largest magnitude it put.
__device__ inline float2 gather_tagged(const unsigned long long* src, uint32_t tag, int K, const InputTo& to, const MegaParams& p) {
    constexpr int B = 4;
    const int n = K / 2;
    float ss = 0.0f, mx = 0.0f;
#pragma unroll 1
    for (int c0 = threadIdx.x; c0 < n; c0 += MEGA_CONSUMERS * B) {
        const unsigned long long* at[B];
        unsigned long long w[B][2];
        float2 g[B];
#pragma unroll
        for (int b = 0; b < B; ++b) {
            const int c = c0 + b * MEGA_CONSUMERS < n ? c0 + b * MEGA_CONSUMERS : c0;
            at[b] = src + 2 * c;
            g[b] = to.scale(2 * c);  // ahead of the polls: its latency passes while the input arrives
        }
        if (!tag_poll<B>(at, tag, w, p)) break;
#pragma unroll
        for (int b = 0; b < B; ++b)
            if (c0 + b * MEGA_CONSUMERS < n) {
                const float2 v = make_float2(tag_value(w[b][0]), tag_value(w[b][1]));
                to.put(2 * (c0 + b * MEGA_CONSUMERS), v, g[b]);
                ss = fmaf(v.x, v.x, fmaf(v.y, v.y, ss));
                mx = fmaxf(mx, fmaxf(fabsf(v.x * g[b].x), fabsf(v.y * g[b].y)));
            }
    }
    return make_float2(ss, mx);
}
// the first layer's: the embedding row of the current token, or x_a as the host left it
template <typename WT> __device__ inline float2 gather_first(const MegaParams& p, const InputTo& to) {
    const WT* row = reinterpret_cast<const WT*>(p.embed) + (p.input_embed ? (size_t)checked_token(__ldcg(&p.st->token), p.embed_rows, &p.st->error) * p.dim : 0);
    float ss = 0.0f, mx = 0.0f;
#pragma unroll 1
    for (int i = 2 * threadIdx.x; i < p.dim; i += 2 * MEGA_CONSUMERS) {
        const float2 v = p.input_embed ? make_float2(Elem<WT>::to_f32(row[i]), Elem<WT>::to_f32(row[i + 1])) : __ldcg(reinterpret_cast<const float2*>(p.x_a + i));
        const float2 g = to.scale(i);
        to.put(i, v, g);
        ss = fmaf(v.x, v.x, fmaf(v.y, v.y, ss));
        mx = fmaxf(mx, fmaxf(fabsf(v.x * g.x), fabsf(v.y * g.y)));
    }
    return make_float2(ss, mx);
}

// The phases of one GPU share their code: a layer's instructions run once per layer and CTA, and five inlined copies of
// the GEMV waited for the instruction cache (about 0.5 us at the start of every phase of a small model).
enum { PH_QKV = 0, PH_WO = 1, PH_W13 = 2, PH_W2 = 3, PH_HEAD = 4 };

// the rows of a phase: input slices out of xs, times inv (1 / root mean square, or 1), then times the power of two `up` of quantised
// rows (one after the other: their product overflows where the vector is zero or tiny); the rows' results times unscale
template <typename LT, int NITER, int R>
__device__ inline void tagged_rows(Ring& ring, const MegaParams& p, float inv, float up, float unscale, float* norm_out, const int2& rows, int K) {
    const float* xs = reinterpret_cast<const float*>(mega_dyn() + p.off_xs);
    Slices<LT, NITER> x;
    if constexpr (Wfmt<LT>::QUANT) {
        x.fill(xs, inv, up, K);
    } else {
        constexpr int EPC = Wfmt<LT>::EPC;
        const int tid = threadIdx.x & 255, nchunks = K / EPC;
#pragma unroll
        for (int i = 0; i < NITER; ++i) {
            const int c = tid + i * GEMV_CONSUMERS;
#pragma unroll
            for (int e = 0; e < EPC; e += 4) {
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (c < nchunks) v = *reinterpret_cast<const float4*>(xs + (size_t)c * EPC + e);
                v.x *= inv; v.y *= inv; v.z *= inv; v.w *= inv;
                if (norm_out != nullptr && blockIdx.x == 0 && threadIdx.x < 256 && c < nchunks) *reinterpret_cast<float4*>(norm_out + (size_t)c * EPC + e) = v;
                x.set(i, e, v);
            }
        }
    }
    stream_partials<LT, NITER, R>(ring, x, unscale, rows.x, rows.y, K, p);
}

// the epilogue of a phase on this CTA's rows (arithmetic of EpiQKV, EpiGate, EpiResidual, EpiStore)
template <typename KT>
__device__ inline void tagged_epilogue(const MegaParams& p, int ph, bool last_layer, void* kv, uint32_t tag) {
    const MegaShared& sh = mega_shared();
    const float* partial = reinterpret_cast<const float*>(mega_dyn() + p.off_partial);
    const float* resid = reinterpret_cast<const float*>(mega_dyn() + p.off_resid);
    const int2 rows = sh.rows[ph == PH_W2 ? PH_WO : ph];
    if (ph == PH_QKV || ph == PH_W13) {  // pairs of rows
#pragma unroll 1
        for (int j = 2 * threadIdx.x; j < rows.y - rows.x; j += 2 * MEGA_CONSUMERS) {
            const int r = rows.x + j;
            float e = row_sum(partial, j), o = row_sum(partial, j + 1);
            if (ph == PH_W13) {
                tag_store(p.tgate + (r >> 1), gate_value(e, o, p.activation), tag);
                continue;
            }
            const int d = r & (p.hd - 1);  // (hd is 64 or 128)
            if (r < p.q_dim + p.kv_dim) {
                const float2 cs = sh.rope[d >> 1];
                const float a = e * cs.x - o * cs.y, b = o * cs.x + e * cs.y;
                e = a;
                o = b;
            }
            unsigned long long* dst = p.tq + r;
            if (r >= p.q_dim) {  // tkv: this position's K then V as cached (rounded), for the CTAs that attend to it in this layer
                const int rk = r - p.q_dim, v = rk >= p.kv_dim, head = (v ? rk - p.kv_dim : rk) >> (p.hd == 128 ? 7 : 6);
                const KT ek = Elem<KT>::from_f32(e), ok = Elem<KT>::from_f32(o);
                KT* page = reinterpret_cast<KT*>(kv) + sh.kv_at + (size_t)(v * p.kv_heads + head) * p.page_tokens * p.hd + d;
                page[0] = ek;
                page[1] = ok;
                e = Elem<KT>::to_f32(ek);
                o = Elem<KT>::to_f32(ok);
                dst = p.tkv + rk;
            }
            tag_store(dst, e, tag);
            tag_store(dst + 1, o, tag);
        }
    } else {
#pragma unroll 1
        for (int j = threadIdx.x; j < rows.y - rows.x; j += MEGA_CONSUMERS) {
            const int r = rows.x + j;
            const float y = row_sum(partial, j);
            if (ph == PH_HEAD) {
                p.logits[r] = y;
            } else {
                const float v = resid[(ph == PH_W2 ? p.resid_cap : 0) + j] + p.alpha * y;
                tag_store((ph == PH_W2 ? p.tx_a : p.tx_b) + r, v, tag);
                if (ph == PH_W2 && last_layer) p.x_a[r] = v;
            }
        }
    }
}

// ---- grid barrier for the consumer threads of all CTAs (arrival k of this launch).  One thread
// per CTA adds to a monotonic counter with release semantics (a reduction, not an atomic with a
// result: no round trip) and polls it with acquire loads until all CTAs of this arrival are in;
// the wait is bounded by time.
__device__ inline bool grid_barrier(unsigned long long* counter, unsigned long long target, unsigned long long wait_ns, int* err) {
    mega_bar();  // every consumer's global writes of the phase are issued
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(counter), "l"(1ull) : "memory");
        bool ok = false;
        unsigned long long t0 = 0;
        for (int i = 0;; ++i) {
            unsigned long long v;
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(counter) : "memory");
            if (v >= target) { ok = true; break; }
            if ((i & 63) == 63) {
                const unsigned long long now = global_ns();
                if (t0 == 0) t0 = now;
                else if (now - t0 > wait_ns) break;
            }
        }
        if (!ok) {
            atomicCAS(err, 0, 3);
            mega_shared().abort = 1;
        }
    }
    mega_bar();
    return !mega_aborted();
}

// q of the kv head's q heads and, where the CTA holds the newest tile, this position's K and V row (as cached) from the
// tagged words into shared memory: every lane group needs the same values.
template <typename KT>
__device__ inline bool attention_inputs(const MegaParams& p, int h, bool newest, uint32_t tag) {
    MegaShared& sh = mega_shared();
    const int nq = p.gqa * p.hd / 2, t = threadIdx.x;  // pairs of q, at most one per thread
    const bool want_q = t < nq, want_row = newest && t < p.hd;  // pair t of the row: K's pairs, then V's
    float mx = 0.0f;
    if (want_q || want_row) {
        const unsigned long long* const q = p.tq + (size_t)h * p.gqa * p.hd + 2 * t;
        const unsigned long long* const row = p.tkv + h * p.hd + (t < p.hd / 2 ? 2 * t : p.kv_dim + 2 * t - p.hd);
        const unsigned long long* const at[2] = {want_q ? q : row, want_row ? row : q};
        unsigned long long w[2][2];
        if (tag_poll<2>(at, tag, w, p)) {
            if (want_q) {
                const float2 v = make_float2(tag_value(w[0][0]), tag_value(w[0][1]));
                *reinterpret_cast<float2*>(sh.q + 2 * t) = v;
                mx = fmaxf(fabsf(v.x), fabsf(v.y));
            }
            if (want_row) {
                KT* kv = reinterpret_cast<KT*>(sh.row);
                kv[2 * t] = Elem<KT>::from_f32(tag_value(w[1][0]));
                kv[2 * t + 1] = Elem<KT>::from_f32(tag_value(w[1][1]));
            }
        }
    }
    if (p.gqa > 2) {  // the largest magnitude per warp
        mx = warp_max(mx);
        if ((t & 31) == 0) sh.red[t >> 5] = mx;
    }
    mega_bar();
    return !mega_aborted();
}

// ---- attention phase with 4 or 8 q heads per kv head and an fp16 cache.  Scores are a product with M = heads: rows 0-7 of
// mma.m16n8k16 hold the heads' q rounded to fp16 (times a power of two that brings the largest to 2^14), rows 8-15 the
// remainders (together within 2^-23 of q, as above), so one instruction gives both parts of eight positions' scores and no shuffle sums them up (the general
// phase below spends 40 instructions per position and head on that: 15.6 us per layer of a 1B model at 2000 positions, 9.1 us
// here; a token of it 0.88 ms, 0.91 ms with a kernel per operator).  A warp takes eight positions of a tile; its probabilities go through 128
// bytes of shared memory to lanes that hold 16 bytes of a V row each, for four heads.  Warps 0-7 and 8-15 take alternate
// tiles (4 heads), or heads 0-3 and 4-7 of every tile (8 heads).  q and the newest row arrive, partials leave as tagged words.
template <class Tick>
__device__ inline bool attention_grouped(Ring& ring, const MegaParams& p, int attn_len, uint32_t tag, const Tick& input_is_in) {
    constexpr float NEG = -3.402823466e+38f;
    constexpr int NH = 4;  // heads a warp accumulates
    MegaShared& sh = mega_shared();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, set = warp >> 3, g = lane >> 2, t = lane & 3;
    const int HD = p.hd, T = p.tile_tokens, ntiles = (attn_len + T - 1) / T, pos = attn_len - 1, CH = HD / 8;  // CH: 16-byte chunks of a row
    const bool by_head = p.gqa > NH;
    const int h0 = by_head ? NH * set : 0;  // this warp's heads among the kv head's
    const uint32_t row_bytes = (uint32_t)HD * 2u;
    float* probs_all = &sh.tparts[0][0][0];
    float* probs = probs_all + warp * 8 * NH;  // [8 positions][NH]
    const AttnPlan plan = sh.plan;
    bool ok = true;
    if (plan.first < 0) { input_is_in(); return !mega_aborted(); }
    for (int h = plan.first; h < p.kv_heads && ok; h += plan.step) {
        if (!attention_inputs<__half>(p, h, plan.t1 == ntiles, tag)) { ok = false; break; }
        if (h == plan.first) input_is_in();
        float mx = 0.0f;
#pragma unroll
        for (int i = 0; i < MEGA_CONSUMERS / 32; ++i) mx = fmaxf(mx, sh.red[i]);
        const int e = (int)(__float_as_uint(mx) >> 23), f = e == 255 ? 127 : min(253, max(1, 268 - e));
        const float up = __uint_as_float((uint32_t)f << 23), down = __uint_as_float((uint32_t)(254 - f) << 23) * p.attn_scale;
        // step s = 2 j + b: elements 4 b .. 4 b + 3 of chunk 4 j + t
        uint32_t qa[8][4];
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            const int d = (4 * (s >> 1) + t) * 8 + 4 * (s & 1);
            const bool live = g < p.gqa && d < HD;
            float4 v = live ? *reinterpret_cast<const float4*>(sh.q + g * HD + d) : make_float4(0.f, 0.f, 0.f, 0.f);
            v.x *= up; v.y *= up; v.z *= up; v.w *= up;
#pragma unroll
            for (int k = 0; k < 2; ++k) {  // hi, lo
                qa[s][k] = Mma16<__half>::part(v.x, v.y);
                qa[s][2 + k] = Mma16<__half>::part(v.z, v.w);
            }
        }
        float acc[NH][8], m = NEG, lsum = 0.0f;  // m, lsum: of head h0 + g (lsum of this lane's positions), meaningful for g < NH
#pragma unroll
        for (int q = 0; q < NH; ++q)
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[q][i] = 0.0f;
        const int ncta_tiles = plan.t1 - plan.t0;
        Ring at = ring;
        for (int idx = 0; idx < ncta_tiles; ++idx) {
            const int tile = plan.t0 + idx;
            const int slot_k = at.slot;
            const uint32_t turn_k = at.turn;
            at.advance(1);
            const int slot_v = at.slot;
            const uint32_t turn_v = at.turn;
            at.advance(1);
            if (!mbar_wait(ring.full0 + 8u * slot_k, turn_k) || !mbar_wait(ring.full0 + 8u * slot_v, turn_v)) {
                atomicCAS(&p.st->error, 0, DEV_ERR_FULL_WAIT);
                sh.abort = 1;
                ok = false;
                break;
            }
            const int w0 = (warp & 7) * 8;  // first position of this warp in the tile
            if ((by_head || (idx & 1) == set) && w0 < T && tile * T + w0 < attn_len) {  // (uniform in the warp)
                const uint32_t kbase = ring.base + (uint32_t)slot_k * ring.stage_cap, vbase = ring.base + (uint32_t)slot_v * ring.stage_cap;
                float c[4] = {0.f, 0.f, 0.f, 0.f}, c2[4] = {0.f, 0.f, 0.f, 0.f};
                const int kpos = tile * T + w0 + g;
                const bool klive = w0 + g < T && kpos < attn_len;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (4 * j < CH) {
                        const int ch = 4 * j + t;
                        uint4 k = make_uint4(0, 0, 0, 0);
                        if (klive) k = kpos == pos ? sh.row[ch] : lds128(kbase + (uint32_t)(w0 + g) * row_bytes + (uint32_t)ch * 16u);
                        Mma16<__half>::mma(c, qa[2 * j], k.x, k.y);
                        Mma16<__half>::mma(c2, qa[2 * j + 1], k.z, k.w);
                    }
                }
                // scores of head g at positions 2 t and 2 t + 1; this warp's heads move to g = 0 .. NH - 1
                float s0 = ((c[0] + c2[0]) + (c[2] + c2[2])) * down, s1 = ((c[1] + c2[1]) + (c[3] + c2[3])) * down;
                if (by_head) {
                    s0 = __shfl_sync(0xffffffffu, s0, ((g + h0) & 7) * 4 + t);
                    s1 = __shfl_sync(0xffffffffu, s1, ((g + h0) & 7) * 4 + t);
                }
                const int p0 = w0 + 2 * t;
                if (p0 >= T || tile * T + p0 >= attn_len) s0 = NEG;
                if (p0 + 1 >= T || tile * T + p0 + 1 >= attn_len) s1 = NEG;
                float top = fmaxf(s0, s1);
                top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
                top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
                const float mnew = fmaxf(m, top), corr = expf(m - mnew);
                const float e0 = s0 > NEG ? expf(s0 - mnew) : 0.0f, e1 = s1 > NEG ? expf(s1 - mnew) : 0.0f;
                lsum = lsum * corr + e0 + e1;
                m = mnew;
                __syncwarp();
                if (g < NH) {
                    probs[(2 * t) * NH + g] = e0;
                    probs[(2 * t + 1) * NH + g] = e1;
                }
                __syncwarp();
#pragma unroll
                for (int q = 0; q < NH; ++q) {
                    const float cq = __shfl_sync(0xffffffffu, corr, 4 * q);
#pragma unroll
                    for (int i = 0; i < 8; ++i) acc[q][i] *= cq;
                }
                const int ch = lane & (CH - 1), side = 32 / CH;  // positions side by side
#pragma unroll 2
                for (int r = lane / CH; r < 8; r += side) {
                    const int vpos = tile * T + w0 + r;
                    uint4 v = make_uint4(0, 0, 0, 0);
                    if (w0 + r < T && vpos < attn_len) v = vpos == pos ? sh.row[CH + ch] : lds128(vbase + (uint32_t)(w0 + r) * row_bytes + (uint32_t)ch * 16u);
                    const float4 pr = *reinterpret_cast<const float4*>(probs + r * NH);
                    float x[8];
                    Elem<__half>::unpack(v, x);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        acc[0][i] = fmaf(pr.x, x[i], acc[0][i]);
                        acc[1][i] = fmaf(pr.y, x[i], acc[1][i]);
                        acc[2][i] = fmaf(pr.z, x[i], acc[2][i]);
                        acc[3][i] = fmaf(pr.w, x[i], acc[3][i]);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(ring.empty0 + 8u * slot_k);
                mbar_arrive(ring.empty0 + 8u * slot_v);
            }
        }
        // ---- merge: the warps' maxima, then every warp's sums relative to the CTA's, added in two halves of eight warps
        lsum += __shfl_xor_sync(0xffffffffu, lsum, 1);
        lsum += __shfl_xor_sync(0xffffffffu, lsum, 2);
        float* ls = probs_all + 16 * 8 * NH;  // [16 warps][NH] sums of the probabilities, then their maxima
        float* mxs = ls + 16 * NH;
        if (t == 0 && g < NH) mxs[warp * NH + g] = m;
        mega_bar();
        if (mega_aborted()) ok = false;
        ring.advance(2 * ncta_tiles);
        if (!ok) break;
        const int first = by_head ? 8 * set : 0, last = by_head ? first + 8 : 16;  // warps with the same heads
        float M = NEG;
        if (g < NH)
            for (int w = first; w < last; ++w) M = fmaxf(M, mxs[w * NH + g]);
        const float wgt = m > NEG ? expf(m - M) : 0.0f;
        lsum *= wgt;
        // slots: [8][NH][128] weighted V
        float* slots = &sh.accs[0][0];
#pragma unroll
        for (int q = 0; q < NH; ++q) {
            const float wq = __shfl_sync(0xffffffffu, wgt, 4 * q);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float v = acc[q][i] * wq;
                v += __shfl_xor_sync(0xffffffffu, v, 16);
                if (CH == 8) v += __shfl_xor_sync(0xffffffffu, v, 8);
                acc[q][i] = v;
            }
        }
        if (t == 0 && g < NH) ls[warp * NH + g] = lsum;
        const bool second = by_head ? (warp & 4) != 0 : set != 0;           // which half of the warps writes first
        float* mine = slots + (by_head ? set * 4 + (warp & 3) : warp & 7) * NH * 128;
        if (second && lane < CH)
#pragma unroll
            for (int q = 0; q < NH; ++q)
#pragma unroll
                for (int i = 0; i < 8; i += 4) *reinterpret_cast<float4*>(mine + q * 128 + lane * 8 + i) = make_float4(acc[q][i], acc[q][i + 1], acc[q][i + 2], acc[q][i + 3]);
        mega_bar();
        if (!second && lane < CH)
#pragma unroll
            for (int q = 0; q < NH; ++q)
#pragma unroll
                for (int i = 0; i < 8; i += 4) {
                    float4* at = reinterpret_cast<float4*>(mine + q * 128 + lane * 8 + i);
                    const float4 o = *at;
                    *at = make_float4(acc[q][i] + o.x, acc[q][i + 1] + o.y, acc[q][i + 2] + o.z, acc[q][i + 3] + o.w);
                }
        mega_bar();
        for (int i = threadIdx.x; i < p.gqa * HD; i += MEGA_CONSUMERS) {
            const int q = i / HD, d = i & (HD - 1);
            const int s0 = by_head ? 4 * (q / NH) : 0, s1 = by_head ? s0 + 4 : 8, wa = by_head ? 8 * (q / NH) : 0, wb = by_head ? wa + 8 : 16;
            float a = 0.0f;
            for (int s = s0; s < s1; ++s) a += slots[(s * NH + q % NH) * 128 + d];
            unsigned long long* o = p.tparts + ((size_t)(h * p.gqa + q) * MEGA_CPH_CAP + plan.part) * (HD + 2);
            tag_store(o + d, a, tag);
            if (d < 2) {
                float r = NEG;
                if (d == 0) for (int w = wa; w < wb; ++w) r = fmaxf(r, mxs[w * NH + q % NH]);
                else { r = 0.0f; for (int w = wa; w < wb; ++w) r += ls[w * NH + q % NH]; }
                tag_store(o + HD + d, r, tag);
            }
        }
        mega_bar();  // the slots are free for the next head
    }
    return ok && !mega_aborted();
}

// ---- attention phase (sdpa_causal, lib.rs:1426-1489, for the tiles of this CTA).  All sixteen warps
// work on every tile, in four teams of four warps that divide its positions; GQ is the number of q heads per kv head (a
// template parameter, so that one head's state costs no registers when there is one).  LPT lanes hold one cached position's row as 16-byte chunks, 128 / LPT
// positions side by side, UNR deep, with a running (max, sum, weighted V) per lane group and q head.  A warp copies its
// rows of a tile to registers, releases the two ring slots (every warp arrives once on each) and computes while the next
// tile lands; nothing but the ring's barriers orders the warps until the merge at the end.
// TAG: q and the new position's row arrive, and the CTA's partials leave, as tagged words.
template <typename KT, int GQ, bool TAG, class Tick>
__device__ inline bool attention_phase(Ring& ring, const MegaParams& p, const void* kv_pool, int attn_len, uint32_t tag, const Tick& input_is_in) {
    MegaShared& sh = mega_shared();
    constexpr int EPC = Elem<KT>::EPC;
    constexpr int UNR = 2;
    constexpr float NEG = -3.402823466e+38f;
    const int tid = threadIdx.x, team = tid >> 7, tt = tid & 127, lane = tid & 31;
    const int HD = p.hd, LPT = HD / EPC, NG = 128 / LPT;
    const int g = tt / LPT, l = tt % LPT;
    const int T = p.tile_tokens, ntiles = (attn_len + T - 1) / T, pos = attn_len - 1;
    const uint32_t row_bytes = (uint32_t)HD * sizeof(KT);
    const size_t head_stride = (size_t)p.page_tokens * HD, page_stride = (size_t)2 * p.kv_heads * head_stride;
    const KT* pool = reinterpret_cast<const KT*>(kv_pool);
    float* accs = sh.accs[team];  // [NG][HD] lane-group accumulators of this team
    float* gm = accs + 128 * 8;    // [NG] max, then [NG] sum
    float* gl = gm + 32;
    bool ok = true;
    const AttnPlan plan = sh.plan;
    if (plan.first >= 0) {
        const int t0 = plan.t0, t1 = plan.t1;
        const int ncta_tiles = t1 - t0;
        for (int h = plan.first; h < p.kv_heads && ok; h += plan.step) {
            if constexpr (TAG) {
                if (!attention_inputs<KT>(p, h, t1 == ntiles, tag)) { ok = false; break; }
                if (h == plan.first) input_is_in();
            }
            float qf[GQ][EPC], acc[GQ][EPC], m[GQ], lsum[GQ];
#pragma unroll
            for (int qi = 0; qi < GQ; ++qi) {
                m[qi] = NEG;
                lsum[qi] = 0.0f;
#pragma unroll
                for (int e = 0; e < EPC; ++e) acc[qi][e] = 0.0f;
#pragma unroll
                for (int e = 0; e < EPC; e += 4) {
                    const float4 v = TAG ? *reinterpret_cast<const float4*>(sh.q + qi * HD + l * EPC + e)
                                         : __ldcg(reinterpret_cast<const float4*>(p.q + (size_t)(h * GQ + qi) * HD + l * EPC + e));
                    qf[qi][e] = v.x; qf[qi][e + 1] = v.y; qf[qi][e + 2] = v.z; qf[qi][e + 3] = v.w;
                }
            }
            const int TQ = max(1, T / MEGA_TEAMS);  // positions of a tile per team
            Ring at = ring;
            for (int idx = 0; idx < ncta_tiles; ++idx) {
                if (!ok) break;  // this warp only: the others learn it from the abort flag behind the barrier below
                const int tile = t0 + idx;
                const int slot_k = at.slot;
                const uint32_t turn_k = at.turn;
                at.advance(1);
                const int slot_v = at.slot;
                const uint32_t turn_v = at.turn;
                at.advance(1);
                if (!mbar_wait(ring.full0 + 8u * slot_k, turn_k) || !mbar_wait(ring.full0 + 8u * slot_v, turn_v)) {
                    atomicCAS(&p.st->error, 0, DEV_ERR_FULL_WAIT);
                    sh.abort = 1;
                    ok = false;
                    break;
                }
                const uint32_t kbase = ring.base + (uint32_t)slot_k * ring.stage_cap, vbase = ring.base + (uint32_t)slot_v * ring.stage_cap;
                for (int tb = 0; tb < TQ; tb += NG * UNR) {  // bounds are uniform across the warp (shuffles inside)
                    uint4 kw[UNR], vw[UNR];
                    bool live[UNR];
#pragma unroll
                    for (int u = 0; u < UNR; ++u) {
                        const int tq = tb + g + u * NG, ti = team * TQ + tq, tok = tile * T + ti;
                        kw[u] = make_uint4(0, 0, 0, 0);
                        vw[u] = make_uint4(0, 0, 0, 0);
                        live[u] = tq < TQ && ti < T && tok < attn_len;
                        if (live[u]) {
                            if (tok == pos) {  // this token's own row was written after the tile was requested: read it from global memory
                                if constexpr (TAG) {
                                    kw[u] = sh.row[l];
                                    vw[u] = sh.row[LPT + l];
                                } else {
                                    const int* pt = reinterpret_cast<const int*>(mega_dyn() + p.off_pt);
                                    const int page = pt[tok / p.page_tokens], off = tok % p.page_tokens;
                                    const KT* kp = pool + (size_t)page * page_stride + (size_t)h * head_stride + (size_t)off * HD + l * EPC;
                                    kw[u] = ldg_stream_coherent(kp);
                                    vw[u] = ldg_stream_coherent(kp + (size_t)p.kv_heads * head_stride);
                                }
                            } else {
                                kw[u] = lds128(kbase + (uint32_t)ti * row_bytes + (uint32_t)l * 16u);
                                vw[u] = lds128(vbase + (uint32_t)ti * row_bytes + (uint32_t)l * 16u);
                            }
                        }
                    }
                    if (tb + NG * UNR >= TQ) {  // the warp's last rows of the tile are in registers: the slots may be refilled
                        __syncwarp();
                        if (lane == 0) {
                            mbar_arrive(ring.empty0 + 8u * slot_k);
                            mbar_arrive(ring.empty0 + 8u * slot_v);
                        }
                    }
#pragma unroll
                    for (int qi = 0; qi < GQ; ++qi) {
                        float sc[UNR];
                        float mnew = m[qi];
#pragma unroll
                        for (int u = 0; u < UNR; ++u) {
                            float f[EPC];
                            Elem<KT>::unpack(kw[u], f);
                            float d = 0.0f;
#pragma unroll
                            for (int e = 0; e < EPC; ++e) d = fmaf(qf[qi][e], f[e], d);
                            for (int o = LPT / 2; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
                            sc[u] = live[u] ? d * p.attn_scale : NEG;
                            mnew = fmaxf(mnew, sc[u]);
                        }
                        if (mnew > NEG) {
                            const float corr = expf(m[qi] - mnew);
                            lsum[qi] *= corr;
#pragma unroll
                            for (int e = 0; e < EPC; ++e) acc[qi][e] *= corr;
#pragma unroll
                            for (int u = 0; u < UNR; ++u) {
                                if (live[u]) {
                                    const float pr = expf(sc[u] - mnew);
                                    lsum[qi] += pr;
                                    float f[EPC];
                                    Elem<KT>::unpack(vw[u], f);
#pragma unroll
                                    for (int e = 0; e < EPC; ++e) acc[qi][e] = fmaf(pr, f[e], acc[qi][e]);
                                }
                            }
                            m[qi] = mnew;
                        }
                    }
                }
            }
            mega_bar();  // every warp is through its tiles (or has given up)
            if (mega_aborted()) ok = false;
            ring.advance(2 * ncta_tiles);
            if (!ok) break;
            // ---- merge: lane groups of a team, then the teams; team 0 stores this CTA's partial of every q head
#pragma unroll
            for (int qi = 0; qi < GQ; ++qi) {  // unrolled: a run-time index would put the per-head state in local memory
#pragma unroll
                for (int e = 0; e < EPC; ++e) accs[g * HD + l * EPC + e] = acc[qi][e];
                if (l == 0) { gm[g] = m[qi]; gl[g] = lsum[qi]; }
                team_bar(team);
                float* mine = sh.tparts[team][qi];
                if (tt < HD) {
                    float M = NEG;
                    for (int gg = 0; gg < NG; ++gg) M = fmaxf(M, gm[gg]);
                    float L = 0.0f, a = 0.0f;
                    for (int gg = 0; gg < NG; ++gg) {
                        if (gl[gg] > 0.0f) {
                            const float wgt = expf(gm[gg] - M);
                            L += gl[gg] * wgt;
                            a += accs[gg * HD + tt] * wgt;
                        }
                    }
                    mine[tt] = a;
                    if (tt == 0) { mine[128] = M; mine[129] = L; }
                }
                team_bar(team);
            }
            mega_bar();
            if (team < GQ && tt < HD) {  // team k merges the teams' results of q head k
                float M = NEG;
                for (int k = 0; k < MEGA_TEAMS; ++k) {
                    const float* tp = sh.tparts[k][team];
                    if (tp[129] > 0.0f) M = fmaxf(M, tp[128]);
                }
                float L = 0.0f, a = 0.0f;
                for (int k = 0; k < MEGA_TEAMS; ++k) {
                    const float* tp = sh.tparts[k][team];
                    if (tp[129] > 0.0f) {
                        const float wgt = expf(tp[128] - M);
                        L += tp[129] * wgt;
                        a += tp[tt] * wgt;
                    }
                }
                if constexpr (TAG) {
                    unsigned long long* o = p.tparts + ((size_t)(h * GQ + team) * MEGA_CPH_CAP + plan.part) * (HD + 2);
                    tag_store(o + tt, a, tag);
                    if (tt < 2) tag_store(o + HD + tt, tt ? L : M, tag);
                } else {
                    const size_t slot = (size_t)(h * GQ + team) * MEGA_MAX_PARTS + plan.part;
                    p.part_acc[slot * HD + tt] = a;
                    if (tt == 0) {
                        p.part_ml[slot * 2 + 0] = M;
                        p.part_ml[slot * 2 + 1] = L;
                    }
                }
            }
            mega_bar();  // the teams' partials are free for the next head
        }
    } else if constexpr (TAG) {
        input_is_in();
    }
    return ok && !mega_aborted();
}

// ---- after the barrier behind the attention phase: every CTA merges the partials of every head
// (fixed order) into the attention vector, in its own shared memory
__device__ inline void merge_attention(const MegaParams& p, float* xs) {
    constexpr float NEG = -3.402823466e+38f;
    const int HD = p.hd, cph = mega_shared().plan.cph;
    for (int c = threadIdx.x; c < p.q_dim / 4; c += MEGA_CONSUMERS) {  // four consecutive dimensions of one head
        const int hq = (c * 4) / HD, d = (c * 4) % HD;
        const float2* ml = reinterpret_cast<const float2*>(p.part_ml) + (size_t)hq * MEGA_MAX_PARTS;
        const float* pa = p.part_acc + (size_t)hq * MEGA_MAX_PARTS * HD + d;
        // one pass with a running maximum, so that the loads of all partials are independent of each other
        float M = NEG, L = 0.0f;
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
        for (int k = 0; k < cph; ++k) {
            const float2 v = __ldcg(ml + k);
            const float4 a = __ldcg(reinterpret_cast<const float4*>(pa + (size_t)k * HD));
            if (v.y > 0.0f) {
                const float Mn = fmaxf(M, v.x);
                const float corr = expf(M - Mn), wgt = expf(v.x - Mn);
                L = L * corr + v.y * wgt;
                o.x = o.x * corr + a.x * wgt; o.y = o.y * corr + a.y * wgt; o.z = o.z * corr + a.z * wgt; o.w = o.w * corr + a.w * wgt;
                M = Mn;
            }
        }
        const float inv = L > 0.0f ? 1.0f / L : 0.0f;
        *reinterpret_cast<float4*>(xs + (size_t)c * 4) = make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
    }
    mega_bar();
}

// the same from tagged partials, as the input of the Wo phase
__device__ inline float2 gather_merged(const MegaParams& p, uint32_t tag) {
    constexpr float NEG = -3.402823466e+38f;
    constexpr int B = 4;  // partials in flight
    float mx = 0.0f;
    float* xs = reinterpret_cast<float*>(mega_dyn() + p.off_xs);
    const int HD = p.hd, cph = mega_shared().plan.cph;
#pragma unroll 1
    for (int c = threadIdx.x; c < p.q_dim / 4; c += MEGA_CONSUMERS) {
        const int hq = (c * 4) / HD, d = (c * 4) % HD;
        const unsigned long long* base = p.tparts + (size_t)hq * MEGA_CPH_CAP * (HD + 2);
        float M = NEG, L = 0.0f;
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
        for (int k0 = 0; k0 < cph; k0 += B) {
            const unsigned long long* at[3 * B];
            unsigned long long w[3 * B][2];
#pragma unroll
            for (int k = 0; k < B; ++k) {
                const unsigned long long* part = base + (k0 + k < cph ? k0 + k : k0) * (HD + 2);
                at[3 * k] = part + d;
                at[3 * k + 1] = part + d + 2;
                at[3 * k + 2] = part + HD;
            }
            if (!tag_poll<3 * B>(at, tag, w, p)) break;
#pragma unroll
            for (int k = 0; k < B; ++k) {
                const float m1 = tag_value(w[3 * k + 2][0]), l1 = tag_value(w[3 * k + 2][1]);
                if (k0 + k < cph && l1 > 0.0f) {
                    const float Mn = fmaxf(M, m1);
                    const float corr = expf(M - Mn), wgt = expf(m1 - Mn);
                    L = L * corr + l1 * wgt;
                    o.x = o.x * corr + tag_value(w[3 * k][0]) * wgt; o.y = o.y * corr + tag_value(w[3 * k][1]) * wgt;
                    o.z = o.z * corr + tag_value(w[3 * k + 1][0]) * wgt; o.w = o.w * corr + tag_value(w[3 * k + 1][1]) * wgt;
                    M = Mn;
                }
            }
        }
        const float inv = L > 0.0f ? 1.0f / L : 0.0f;
        o = make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
        *reinterpret_cast<float4*>(xs + (size_t)c * 4) = o;
        mx = fmaxf(fmaxf(mx, fmaxf(fabsf(o.x), fabsf(o.y))), fmaxf(fabsf(o.z), fabsf(o.w)));
    }
    return make_float2(0.0f, mx);
}

// TPAR: the tensor-parallel form (a kernel of its own, so that none of it weighs on the single-GPU token)
// WT: storage of the embedding and the LM head, LT: row format of the linears, KT: of the cache; N, R: chunks a thread takes of
// a row and rows of a stage, at K = dim or q_dim (D), K = hidden (H), and the head's (O); GROUPED: more than two q
// heads per kv head (kernels of their own, like TPAR)
template <typename WT, typename LT, typename KT, int ND, int RD, int NH, int RH, int NO, int RO, bool TPAR, bool GROUPED>
__global__ void __launch_bounds__(MEGA_THREADS, 1) decode_mega_kernel(const __grid_constant__ MegaParams p) {
    constexpr int NW = GEMV_CONSUMERS / 32;
    MegaShared& sh = mega_shared();
    float* const xs = reinterpret_cast<float*>(mega_dyn() + p.off_xs);
    int* const pt_s = reinterpret_cast<int*>(mega_dyn() + p.off_pt);
    MegaLayer* const layers_s = reinterpret_cast<MegaLayer*>(mega_dyn() + p.off_layers);
    Ring ring;
    ring.base = smem_addr(mega_dyn());
    ring.full0 = ring.base + p.off_bars;
    ring.empty0 = ring.full0 + 8u * p.nstages;
    ring.stage_cap = p.stage_cap;
    ring.nstages = p.nstages;
    ring.slot = 0;
    ring.turn = 0;
    int* const err = &p.st->error;
    const int tid = threadIdx.x, warp = tid >> 5;

    if (tid == 0) {
        for (int s = 0; s < p.nstages; ++s) {
            mbar_init(ring.full0 + 8u * s, 1);
            mbar_init(ring.empty0 + 8u * s, 2 * NW);  // the GEMV group's eight warps twice, or all sixteen warps of the attention phase
        }
        mbar_fence_init();
        sh.abort = 0;
    }
    const int attn_len = __ldcg(&p.st->pos) + 1;  // written by the previous token's last kernel
    for (int i = tid; i < p.npages; i += MEGA_THREADS) pt_s[i] = p.page_table[i];
    for (int i = tid; i < p.nlayers * (int)(sizeof(MegaLayer) / 8); i += MEGA_THREADS)
        reinterpret_cast<unsigned long long*>(layers_s)[i] = reinterpret_cast<const unsigned long long*>(p.layers)[i];
    if (tid < 4) {
        int r0, r1;
        cta_rows(tid == 0 ? p.q_dim + 2 * p.kv_dim : tid == 1 ? p.dim : tid == 2 ? 2 * p.hidden : p.vocab, tid == 0 || tid == 2 ? 2 : 1, r0, r1);
        sh.rows[tid == 3 ? PH_HEAD : tid] = make_int2(r0, r1);
    }
    if (tid == 32) sh.plan = attn_plan(p.kv_heads, (attn_len + p.tile_tokens - 1) / p.tile_tokens);
    if (tid == 64) {
        const int page = p.page_table[(attn_len - 1) / p.page_tokens], off = (attn_len - 1) % p.page_tokens;
        sh.kv_at = ((size_t)page * 2 * p.kv_heads * p.page_tokens + off) * p.hd;
    }
    // every CTA of a launch adds one, however it ends, and the next launch starts behind the last of them
    if (!TPAR && tid == 96) sh.launch = atomicAdd(p.grid_counter, 1ull) / gridDim.x;
    if (tid < p.hd / 2) sh.rope[tid] = p.rope[(size_t)(attn_len - 1) * (p.hd / 2) + tid];
    __syncthreads();

    if (warp >= MEGA_CONSUMERS / 32) {  // ---- producers: fill the ring, stage after stage, as slots come free; each every fourth stage
        if ((tid & 31) == 0) {
            const uint64_t policy = l2_evict_first_policy();
            uint64_t kv_policy;
            asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(kv_policy));
            const int mine = warp - MEGA_CONSUMERS / 32;
            // A slot's successive stages may belong to different producers.  A parity wait tells adjacent turns apart: a producer
            // that is done with its stage n - np knows the stages up to n - np - nstages read, and so, with np <= nstages, the
            // slot's turn before last.
            const int np = min(MEGA_PRODUCERS, ring.nstages);  // 2 or 4 (nstages is even)
            if (mine >= np) return;
            int n = 0;
            uint32_t first = 1;  // the ring's first turn: every slot is free
            const unsigned long long producer_budget = p.wait_ns + 2000000000ull;
            auto put = [&](const char* src, uint32_t bytes, bool is_kv) {
                if ((n++ & (np - 1)) == mine) {
                    const uint32_t full = ring.full0 + 8u * ring.slot, empty = ring.empty0 + 8u * ring.slot;
                    // (a consumer that gave up raises the CTA's abort flag: the slot will not come free, and that is no error of its own)
                    if (!first && !mbar_wait_or_abort(empty, ring.turn ^ 1u, &sh.abort, producer_budget)) {
                        if (!mega_aborted()) atomicCAS(err, 0, DEV_ERR_EMPTY_WAIT);
                        return false;
                    }
                    mbar_arrive_expect_tx(full, bytes);
                    // (cached positions are read again by the next token: no evict-first)
                    bulk_g2s_stream(ring.base + (uint32_t)ring.slot * ring.stage_cap, src, bytes, full, is_kv ? kv_policy : policy);
                }
                if (++ring.slot == ring.nstages) { ring.slot = 0; ring.turn ^= 1u; first = 0; }
                return true;
            };
            walk_token_stream<RD, RH, RO>(p, layers_s, pt_s, Wfmt<LT>::row_stride(p.dim), Wfmt<LT>::row_stride(p.q_dim), Wfmt<LT>::row_stride(p.hidden),
                                          (uint32_t)p.dim * (uint32_t)sizeof(WT), (uint32_t)sizeof(KT), put);
        }
        return;
    }
    // ---- consumers
    unsigned long long* tr = nullptr;
    if (p.trace != nullptr && tid == 0 && (blockIdx.x == 0 || blockIdx.x == gridDim.x - 1))
        tr = p.trace + (blockIdx.x == 0 ? 0 : 1) * (size_t)(10 * p.nlayers + 2);
    auto stamp = [&]() {
        if (tr != nullptr) *tr++ = global_ns();
    };
    stamp();
    bool ok = true;
    if constexpr (!TPAR) {
        // layer l's words carry tag0 + l: no two launches share a tag, whether the earlier one got through or not
        const uint32_t tag0 = (uint32_t)sh.launch * (uint32_t)p.nlayers + 1u;
        float* const resid = reinterpret_cast<float*>(mega_dyn() + p.off_resid);
        const int phases = 4 * p.nlayers + (p.want_logits ? 1 : 0);
        for (int step = 0; step < phases; ++step) {
            const int l = step >> 2, ph = l < p.nlayers ? step & 3 : PH_HEAD;
            const MegaLayer& L = layers_s[min(l, p.nlayers - 1)];
            const uint32_t tag = tag0 + (uint32_t)l;
            float2 in;  // sum of squares, largest magnitude
            if (ph == PH_WO) {
                if constexpr (GROUPED) ok = attention_grouped(ring, p, attn_len, tag, stamp);
                else ok = p.gqa == 1 ? attention_phase<KT, 1, true>(ring, p, L.kv, attn_len, tag, stamp) : attention_phase<KT, 2, true>(ring, p, L.kv, attn_len, tag, stamp);
                stamp();
                if (!ok) break;
                in = gather_merged(p, tag);
            } else {
                const InputTo to{xs, ph == PH_QKV ? resid : ph == PH_W13 ? resid + p.resid_cap : nullptr,
                                 ph == PH_QKV ? L.gamma1 : ph == PH_W13 ? L.gamma2 : ph == PH_HEAD ? p.gamma_final : nullptr, sh.rows[PH_WO]};
                if (step == 0) in = gather_first<WT>(p, to);
                else in = gather_tagged(ph == PH_W13 ? p.tx_b : ph == PH_W2 ? p.tgate : p.tx_a, ph == PH_W13 || ph == PH_W2 ? tag : tag - 1u, ph == PH_W2 ? p.hidden : p.dim, to, p);
            }
            const bool norm = ph != PH_WO && ph != PH_W2;
            in.x = warp_sum(in.x);
            if (Wfmt<LT>::QUANT) in.y = warp_max(in.y);
            if ((tid & 31) == 0) { sh.red[warp] = in.x; sh.red[32 + warp] = in.y; }
            mega_bar();
            if (ph != PH_HEAD) stamp();
            float inv = 1.0f;
            if (norm) {
                float tot = 0.0f;
#pragma unroll
                for (int i = 0; i < MEGA_CONSUMERS / 32; ++i) tot += sh.red[i];
                inv = 1.0f / sqrtf(tot * (1.0f / (float)p.dim) + RMS_EPS);
            }
            if constexpr (Wfmt<LT>::QUANT) {
                float mx = 0.0f, up = 1.0f, unscale = 1.0f;
                if (ph != PH_HEAD) {  // the power of two that brings the largest input to [2^14, 2^15)
#pragma unroll
                    for (int i = 0; i < MEGA_CONSUMERS / 32; ++i) mx = fmaxf(mx, sh.red[32 + i]);
                    const int e = (int)(__float_as_uint(mx * inv) >> 23), f = e == 255 ? 127 : min(253, max(1, 268 - e));
                    up = __uint_as_float((uint32_t)f << 23);
                    unscale = __uint_as_float((uint32_t)(254 - f) << 23);
                }
                if (ph == PH_HEAD) tagged_rows<WT, NO, RO>(ring, p, inv, 1.0f, 1.0f, p.norm_final, sh.rows[ph], p.dim);
                else if (ph == PH_W2) tagged_rows<LT, NH, RH>(ring, p, inv, up, unscale, nullptr, sh.rows[PH_WO], p.hidden);
                else tagged_rows<LT, ND, RD>(ring, p, inv, up, unscale, nullptr, sh.rows[ph], ph == PH_WO ? p.q_dim : p.dim);
            } else {
                if (ph == PH_W2) tagged_rows<LT, NH, RH>(ring, p, inv, 1.0f, 1.0f, nullptr, sh.rows[PH_WO], p.hidden);
                else tagged_rows<LT, ND, RD>(ring, p, inv, 1.0f, 1.0f, ph == PH_HEAD ? p.norm_final : nullptr, sh.rows[ph], ph == PH_WO ? p.q_dim : p.dim);
            }
            mega_bar();
            if (mega_aborted()) { ok = false; break; }
            tagged_epilogue<KT>(p, ph, l + 1 == p.nlayers, L.kv, tag);
            if (ph != PH_HEAD) stamp();
        }
        stamp();
    } else {
        const unsigned long long epoch = __ldcg(&p.st->epoch);
        unsigned long long arrivals = epoch * 3ull * (unsigned long long)p.nlayers;  // barriers completed by earlier launches
        auto barrier = [&]() {
            arrivals += 1;
            return grid_barrier(p.grid_counter, arrivals * gridDim.x, p.wait_ns, err);
        };
        // behind a phase whose output travels through the ranks' inboxes the consumer's poll is the synchronisation: the CTA
        // only has to be done with its own shared memory
        auto exchange = [&]() {
            mega_bar();
            return !mega_aborted();
        };
        TpLink tin = p.tp;  // the all-reduced input of a phase, x = res + alpha * sum
        tin.alpha = p.alpha;
        for (int l = 0; l < p.nlayers && ok; ++l) {
            const MegaLayer L = layers_s[l];
            EpiQKV<KT> eq{p.q, reinterpret_cast<KT*>(L.kv), p.page_table, p.st, p.rope, p.q_dim, p.kv_dim, p.hd, p.kv_heads, p.page_tokens};
            // layers after the first: x = x2 + alpha * sum(W2 partials of the layer before), kept in x_a
            if (l == 0) stage_first_input<WT>(p, xs);
            else { tin.in_reduce = 2 * l; tin.res = p.x_b; tin.x_out = p.x_a; gather_input(tin, p.dim, xs, err); }
            ok = consume_gemv<WT, ND, RD, 2, true>(ring, nullptr, xs, L.gamma1, nullptr, p.q_dim + 2 * p.kv_dim, p.dim, p, eq);
            stamp();
            if (!ok || !(ok = barrier())) break;
            stamp();
            ok = p.gqa == 1 ? attention_phase<KT, 1, false>(ring, p, L.kv, attn_len, 0u, stamp) : attention_phase<KT, 2, false>(ring, p, L.kv, attn_len, 0u, stamp);
            stamp();
            if (!ok || !(ok = barrier())) break;
            stamp();
            merge_attention(p, xs);
            ok = consume_gemv<WT, ND, RD, 1, false>(ring, nullptr, xs, nullptr, nullptr, p.dim, p.q_dim, p, EpiPushPartial{&p.tp, 2 * l + 1});
            stamp();
            if (!ok || !(ok = exchange())) break;
            stamp();
            // x2 = x + alpha * sum(Wo partials), kept in x_b
            tin.in_reduce = 2 * l + 1; tin.res = p.x_a; tin.x_out = p.x_b;
            gather_input(tin, p.dim, xs, err);
            ok = consume_gemv<WT, ND, RD, 2, true>(ring, nullptr, xs, L.gamma2, nullptr, 2 * p.hidden, p.dim, p, EpiGate{p.gate, p.activation});
            stamp();
            if (!ok || !(ok = barrier())) break;
            stamp();
            ok = consume_gemv<WT, NH, RH, 1, false>(ring, p.gate, nullptr, nullptr, nullptr, p.dim, p.hidden, p, EpiPushPartial{&p.tp, 2 * l + 2});
            stamp();
            if (!ok || !(ok = exchange())) break;
            stamp();
        }
        if (ok && p.want_logits) {
            tin.in_reduce = 2 * p.nlayers; tin.res = p.x_b; tin.x_out = p.x_a;
            gather_input(tin, p.dim, xs, err);
            ok = consume_gemv<WT, ND, RD, 1, true>(ring, nullptr, xs, p.gamma_final, p.norm_final, p.vocab, p.dim, p, EpiStore{p.logits});
        }
        stamp();
        if (ok && tid == 0 && blockIdx.x == 0) p.st->epoch = epoch + 1;  // every CTA read it before its first barrier
    }
    if (!ok) {
        // leave only once copies that may still be in flight towards this CTA have landed: a copy lands within
        // microseconds, and a slot nobody filled never completes, so the wait for each is short
        for (int s = 0; s < p.nstages; ++s) mbar_wait_or_abort(ring.full0 + 8u * s, ring.turn, nullptr, 200000ull);
    }
}

}  // namespace cd
