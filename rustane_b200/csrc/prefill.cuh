// Batched prefill for sm_100a: every linear of the prompt pass is one tensor-core GEMM
//   C[M tokens, N features] = A[M, K] (activations, 16-bit) * B[N, K]^T (weights as stored for the GEMVs)
// issued with tcgen05.mma, accumulators in tensor memory, operands staged by TMA.
// The attention of the prompt between them is pf_attn_kernel (pf_attn.cuh).
// Math follows the naive forward (full_model.rs:336-437, layer.rs:1287-1431) restricted to
// the prompt positions; K and V land in the decode layout (pages).  There is no batched
// prompt pass in the reference's Metal decoder: it feeds prompt tokens one at a time
// (inference.rs:650-670).
//
// A tile of the output is 128 CG rows x `bn` columns, CG = 1 or 2 CTAs.  As a pair (cta_group::2) each CTA stages its own 128
// rows of A and half of the tile's rows of B, so B crosses L2 -> shared memory once for 256 rows; the even CTA issues the MMAs
// of both.  CTAs are persistent (tiles in turn, row tiles fastest: neighbours share a weight tile in L2) and keep two
// accumulators of 256 columns in tensor memory, so a tile's epilogue runs while the next tile is multiplied.
// Warp 0: TMA producer (one thread).  Warp 1: owns the tensor-memory allocation and issues the MMAs (one thread).  Warps
// 2-5: epilogue, each reading the 32 accumulator lanes tcgen05.ld lets it see (lanes 32 * (warp % 4) ...).
// Shared memory: a ring of stages, each a [128][64] A tile (two under SPLIT) and a [bn / CG][64] B tile of 16-bit elements in
// the 128-byte-swizzled K-major layout TMA writes and the MMA reads.
// What bounds it: the tensor pipe (at hi + lo operands 256 columns take 1024 clocks of MMA for 48 KB a CTA).  One tile a CTA, one
// accumulator and 256 columns a CTA of its own took 299, 173 and 96 us at 1024 rows x (22016, 12288 and, in the mean, 4096 features) of the 5B
// model; this form 230, 130 and 88 us = 1600 TFLOP/s issued in the first.  At few rows the chain of a tile's MMAs
// counts: with the loops of warps 0 and 1 in one thread each (their addresses not in uniform registers) a step of 64 along K took 890
// clocks, as whole warps with one elected thread 624 (37 x 4096 x 4096: 36 and 27 us).
// Every wait is bounded; on expiry the kernel records an error, skips its remaining
// work, still meets the final barrier and frees its tensor memory.
//
// Further down: pf_skinny_kernel, the same machinery with the operands swapped for at most 16
// activation rows (several samples decoding together), its epilogues, and the small kernels
// around both (embedding rows, RMSNorm to hi + lo 16-bit operands).
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace cd {

constexpr int PF_BM = 128, PF_BK = 64, PF_THREADS = 192;
enum { DEV_ERR_PF_FULL = 8, DEV_ERR_PF_EMPTY = 9, DEV_ERR_PF_ACCUM = 10 };

// SPLIT: the activation operand arrives as two 16-bit matrices hi + lo (lo = the rounding
// error of hi, itself rounded), both multiplied with the same weight tile into the same
// accumulator, so the product sees about 16 mantissa bits of the fp32 activation instead of 8.
constexpr uint32_t PF_A_BYTES = PF_BM * PF_BK * 2, PF_RING = 200 * 1024;
constexpr int PF_MAX_STAGES = 8, PF_MAX_BN = 256;
constexpr size_t PF_SMEM = PF_RING + 1024 /* alignment slack */ + 256 /* barriers */;

struct PfGemm {
    int M, N, K;
    int bn;  // columns of a tile: a multiple of 32, PF_MAX_BN at most
    int* err;
    // FP8 linears: B holds the e4m3 values widened to 16 bits; output column n is multiplied by the
    // row scale stored behind row n of the quantised matrix (Wfmt<Fp8Row>), nullptr otherwise
    const unsigned char* qrows;
    uint32_t qstride, qscale_off;
    // grouped problem (a mixture of experts): row tile y multiplies the B rows of group tile_group[y], `group_rows` apart;
    // a negative entry is a tile nobody needs.  nullptr: one matrix
    const int* tile_group;
    int group_rows;
};

// ------------------------------------------------------------------ PTX wrappers
__device__ inline void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
// one CTA of a pair: both of the pair's CTAs load into their own shared memory and count on the even CTA's barrier (no multicast)
__device__ inline void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t leader_bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(dst), "l"(map), "r"(leader_bar), "r"(c0), "r"(c1) : "memory");
}
template <int CG = 1> __device__ inline void tmem_alloc(uint32_t slot_smem, uint32_t ncols) {  // whole warp (of both CTAs of a pair)
    if constexpr (CG == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_smem), "r"(ncols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    } else {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_smem), "r"(ncols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
}
template <int CG = 1> __device__ inline void tmem_dealloc(uint32_t taddr, uint32_t ncols) {  // whole warp (of both CTAs of a pair)
    if constexpr (CG == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ inline void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ inline void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
template <int CG = 1> __device__ inline void umma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    if constexpr (CG == 1)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                     ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                     ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// arrives on bar (CG = 2: on the barrier at this offset of both CTAs) once every MMA issued so far has finished
template <int CG = 1> __device__ inline void umma_commit(uint32_t bar) {
    if constexpr (CG == 1)
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
    else
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ inline bool elect_one() {  // true in one thread of a converged warp
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ inline uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ inline uint32_t cluster_addr(uint32_t addr, uint32_t rank) {  // the same shared-memory offset in CTA `rank` of the cluster
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ inline void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ inline void mbar_arrive_cluster(uint32_t bar) { asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory"); }
// mbar_wait for a barrier that threads of the other CTA arrive on
__device__ inline bool mbar_wait_cluster(uint32_t bar, uint32_t parity, int limit = MBAR_WAIT_LIMIT) {
    for (int i = 0; i < limit; ++i) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}
__device__ inline void tmem_ld32(uint32_t taddr, float (&v)[32]) {  // this lane's 32 consecutive accumulator columns
    uint32_t r[32];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
// Shared-memory matrix descriptor of a K-major tile with 128-byte rows written by TMA with
// the 128-byte swizzle: 8-row groups are 1024 bytes apart; the leading-dimension field is
// not used for this layout; descriptor version 1 (sm_100); swizzle mode 2 (128 B).
__device__ inline uint64_t umma_desc(uint32_t tile_smem) {
    uint64_t d = (uint64_t)((tile_smem & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// ------------------------------------------------------------------ epilogues: (z, row, first column, 32 values)
template <typename T16> __device__ inline T16 pf_cast(float v);
template <> __device__ inline __nv_bfloat16 pf_cast<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ inline __half pf_cast<__half>(float v) { return __float2half_rn(v); }

struct PfEpiPartial {  // the product y, raw (tensor parallel: this rank's partial one, for the all-reduce that follows)
    float* y;
    int ld;
    int silu_cols = 0;  // the first columns go through silu
    __device__ void operator()(int row, int col, const float (&v)[32]) const {
        float4* p = reinterpret_cast<float4*>(y + (size_t)row * ld + col);
        if (col < silu_cols) {
#pragma unroll
            for (int i = 0; i < 32; ++i) reinterpret_cast<float*>(p)[i] = col + i < silu_cols ? __fdividef(v[i], 1.0f + __expf(-v[i])) : v[i];
            return;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) p[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    }
};

struct PfEpiResidual {  // x += alpha * y on the fp32 residual stream
    float* x;
    int ld;
    float alpha;
    __device__ void operator()(int row, int col, const float (&v)[32]) const {
        float4* p = reinterpret_cast<float4*>(x + (size_t)row * ld + col);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float4 t = __ldcg(p + i);
            t.x += alpha * v[4 * i]; t.y += alpha * v[4 * i + 1]; t.z += alpha * v[4 * i + 2]; t.w += alpha * v[4 * i + 3];
            p[i] = t;
        }
    }
};

// value -> hi (+ lo when a second matrix is kept)
template <typename T16> __device__ inline void pf_store(T16* hi, T16* lo, size_t at, float v) {
    const T16 h = pf_cast<T16>(v);
    hi[at] = h;
    if (lo != nullptr) lo[at] = pf_cast<T16>(v - Elem<T16>::to_f32(h));
}

// the same for N neighbouring values as 16-byte stores (N a multiple of 8, hi + at and lo + at on 16-byte boundaries)
template <typename T16, int N> __device__ inline void pf_store_run(T16* hi, T16* lo, size_t at, const float (&v)[N]) {
#pragma unroll
    for (int i = 0; i < N; i += 8) {
        uint32_t h[4], l[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const T16 a = pf_cast<T16>(v[i + 2 * k]), b = pf_cast<T16>(v[i + 2 * k + 1]);
            const T16 c = pf_cast<T16>(v[i + 2 * k] - Elem<T16>::to_f32(a)), d = pf_cast<T16>(v[i + 2 * k + 1] - Elem<T16>::to_f32(b));
            h[k] = (uint32_t)*reinterpret_cast<const unsigned short*>(&a) | (uint32_t)*reinterpret_cast<const unsigned short*>(&b) << 16;
            l[k] = (uint32_t)*reinterpret_cast<const unsigned short*>(&c) | (uint32_t)*reinterpret_cast<const unsigned short*>(&d) << 16;
        }
        *reinterpret_cast<uint4*>(hi + at + i) = make_uint4(h[0], h[1], h[2], h[3]);
        if (lo != nullptr) *reinterpret_cast<uint4*>(lo + at + i) = make_uint4(l[0], l[1], l[2], l[3]);
    }
}

template <typename T16> struct PfEpiGate {  // columns (2j, 2j+1) = (w1, w3) column j: gate[j] = act(y1) * y3
    T16* gate;
    T16* gate_lo;
    int ld, act;
    __device__ void operator()(int row, int col, const float (&v)[32]) const {
        const size_t at = (size_t)row * ld + (col >> 1);
        float g[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const float y1 = v[2 * j], y3 = v[2 * j + 1];
            float a;
            if (act == 1) {
                const float l = fmaxf(y1, 0.5f * y1);
                a = l * l;
            } else {
                a = y1 / (1.0f + expf(-y1));
            }
            g[j] = a * y3;
        }
        if (ld % 8 == 0) {
            pf_store_run(gate, gate_lo, at, g);
        } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) pf_store(gate, gate_lo, at + j, g[j]);
        }
    }
};

// RoPE on q and k; q to a [M, Q] buffer, k and v into the pages.  A thread's 32 columns lie inside one head (widths of 64 or
// 128), so every destination is a run of 64 bytes: 16-byte stores.  (Element by element the epilogue bound the GEMM: 311 us
// at 1024 x 12288 x 4096 where gate|up, 1.8 times the products, took 300; the 5B model's 1024-token prompt went from 30.5
// to 25.9 ms, 4096 tokens from 147 to 131 ms, with this and the same for the attention's output.)
template <typename T16> struct PfEpiQKV {
    T16* q;
    T16* q_lo;
    T16* kv_pool;
    const int* page_table;
    const float2* rope;
    int Q, KV, hd, kv_heads, page_tokens, pos0;
    __device__ void operator()(int row, int col, const float (&v)[32]) const {
        const int pos = pos0 + row;
        if (col < Q + KV) {
            float r[32];
            const float2* cs = rope + (size_t)pos * (hd >> 1) + ((col % hd) >> 1);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const float2 c = cs[j];
                r[2 * j] = v[2 * j] * c.x - v[2 * j + 1] * c.y;
                r[2 * j + 1] = v[2 * j + 1] * c.x + v[2 * j] * c.y;
            }
            if (col < Q) {
                pf_store_run(q, q_lo, (size_t)row * Q + col, r);
                return;
            }
            const int ck = col - Q, head = ck / hd, d = ck % hd;
            const int page = page_table[pos / page_tokens], off = pos % page_tokens;
            pf_store_run(kv_pool, (T16*)nullptr, ((((size_t)page * 2 + 0) * kv_heads + head) * page_tokens + off) * hd + d, r);
        } else {
            const int cv = col - Q - KV, head = cv / hd, d = cv % hd;
            const int page = page_table[pos / page_tokens], off = pos % page_tokens;
            pf_store_run(kv_pool, (T16*)nullptr, ((((size_t)page * 2 + 1) * kv_heads + head) * page_tokens + off) * hd + d, v);
        }
    }
};

// ------------------------------------------------------------------ the GEMM
template <int CG, bool SPLIT, class Epi>
__global__ void __launch_bounds__(PF_THREADS, 1)
pf_gemm_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_a_lo, const __grid_constant__ CUtensorMap tma_b,
               PfGemm p, uint32_t idesc, Epi epi) {
    constexpr uint32_t B_OFF = (SPLIT ? 2 : 1) * PF_A_BYTES;  // stage = A hi | A lo (SPLIT) | B
    extern __shared__ unsigned char pf_raw[];
    const uint32_t rank = CG == 2 ? cluster_rank() : 0u;
    const uint32_t stage = B_OFF + (uint32_t)(p.bn / CG) * PF_BK * 2;
    const int nst = min(PF_MAX_STAGES, (int)(PF_RING / stage));
    const int nkb = (p.K + PF_BK - 1) / PF_BK;
    const int tiles_m = (p.M + CG * PF_BM - 1) / (CG * PF_BM), tiles = tiles_m * ((p.N + p.bn - 1) / p.bn);

    const uint32_t ring = (smem_addr(pf_raw) + 1023u) & ~1023u;
    const uint32_t bars = ring + PF_RING;
    const uint32_t full0 = bars, empty0 = full0 + 8u * PF_MAX_STAGES, accum0 = empty0 + 8u * PF_MAX_STAGES, drained0 = accum0 + 16u, slot = drained0 + 16u;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < nst; ++s) {
            mbar_init(full0 + 8u * s, 1);
            mbar_init(empty0 + 8u * s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(accum0 + 8u * b, 1);
            mbar_init(drained0 + 8u * b, 4 * CG);  // one arrival per epilogue warp, those of both CTAs at the even one's
        }
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc<CG>(slot, 2 * PF_MAX_BN);
    tc_fence_before();
    __syncwarp();
    if constexpr (CG == 2) cluster_sync();
    else __syncthreads();
    tc_fence_after();
    uint32_t tmem_base;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(slot));
    pdl_wait();  // under programmatic dependent launch: the operands and what the epilogue updates are the previous kernels'
    pdl_launch_dependents();
    bool failed = false;
    // whole warps wait and loop, one elected thread issues: addresses and descriptors stay in uniform registers
    auto wait = [&](uint32_t bar, uint32_t parity, int code) {
        const bool ok = __all_sync(0xffffffffu, CG == 2 ? mbar_wait_cluster(bar, parity) : mbar_wait(bar, parity));
        if (!ok) {
            atomicExch(p.err, code);
            failed = true;
        }
        return ok;
    };
    // the walk over this unit's tiles, the same in every role: first row (of the unit), first column, first row of B
    auto at_tile = [&](int t, int& m0, int& n0, int& b0) {
        const int mt = t % tiles_m;
        m0 = mt * CG * PF_BM;
        n0 = b0 = t / tiles_m * p.bn;
        if (p.tile_group == nullptr) return true;
        const int g = __ldcg(p.tile_group + mt);
        b0 += g * p.group_rows;
        return g >= 0;
    };
    const int unit = blockIdx.x / CG, units = gridDim.x / CG;

    int s = 0, m0, n0, b0;
    uint32_t ph = 0;  // ring position and its turn
    auto next_stage = [&] {
        if (++s == nst) { s = 0; ph ^= 1u; }
    };
    if (warp == 0) {  // ---- TMA producer
        for (int t = unit; t < tiles && !failed; t += units) {
            if (!at_tile(t, m0, n0, b0)) continue;
            const int row = m0 + (int)rank * PF_BM, b_row = b0 + (int)rank * (p.bn / CG);
            for (int kb = 0; kb < nkb; ++kb, next_stage()) {
                if (!wait(empty0 + 8u * s, ph ^ 1u, DEV_ERR_PF_EMPTY)) break;
                if (elect_one()) {
                    const uint32_t a_dst = ring + s * stage, full = full0 + 8u * s;
                    if (rank == 0) mbar_arrive_expect_tx(full, CG * stage);
                    if constexpr (CG == 2) {
                        const uint32_t bar = cluster_addr(full, 0);
                        tma_load_2d_pair(a_dst, &tma_a, kb * PF_BK, row, bar);
                        if (SPLIT) tma_load_2d_pair(a_dst + PF_A_BYTES, &tma_a_lo, kb * PF_BK, row, bar);
                        tma_load_2d_pair(a_dst + B_OFF, &tma_b, kb * PF_BK, b_row, bar);
                    } else {
                        tma_load_2d(a_dst, &tma_a, kb * PF_BK, row, full);
                        if (SPLIT) tma_load_2d(a_dst + PF_A_BYTES, &tma_a_lo, kb * PF_BK, row, full);
                        tma_load_2d(a_dst + B_OFF, &tma_b, kb * PF_BK, b_row, full);
                    }
                }
                __syncwarp();
            }
        }
        // the last stages are read before this CTA leaves: nothing arrives on its barriers afterwards
        for (int k = 0; k < nst && !failed; ++k, next_stage()) wait(empty0 + 8u * s, ph ^ 1u, DEV_ERR_PF_EMPTY);
    } else if (warp == 1) {  // ---- MMA issuer
        int j = 0;
        for (int t = unit; rank == 0 && t < tiles && !failed && nkb > 0; t += units) {
            if (!at_tile(t, m0, n0, b0)) continue;
            const uint32_t buf = j & 1, acc = tmem_base + buf * PF_MAX_BN;
            if (!wait(drained0 + 8u * buf, ((j >> 1) & 1) ^ 1u, DEV_ERR_PF_ACCUM)) break;
            tc_fence_after();
            for (int kb = 0; kb < nkb; ++kb, next_stage()) {
                if (!wait(full0 + 8u * s, ph, DEV_ERR_PF_FULL)) break;
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t base = ring + s * stage;
                    const uint64_t adesc = umma_desc(base), ldesc = umma_desc(base + PF_A_BYTES), bdesc = umma_desc(base + B_OFF);
#pragma unroll
                    for (int k = 0; k < PF_BK / 16; ++k) {  // 16 elements = 32 bytes further along K inside the swizzle span
                        umma_f16<CG>(acc, adesc + 2u * k, bdesc + 2u * k, idesc, (kb | k) != 0);
                        if (SPLIT) umma_f16<CG>(acc, ldesc + 2u * k, bdesc + 2u * k, idesc, 1u);
                    }
                    umma_commit<CG>(empty0 + 8u * s);  // the stage may be refilled once these MMAs have read it
                    if (kb == nkb - 1) umma_commit<CG>(accum0 + 8u * buf);
                }
                __syncwarp();
            }
            ++j;
        }
    } else {  // ---- epilogue warps
        const int lane_base = (warp & 3) * 32;
        int j = 0;
        for (int t = unit; t < tiles && !failed; t += units) {
            if (!at_tile(t, m0, n0, b0)) continue;
            const uint32_t buf = j & 1, acc = tmem_base + buf * PF_MAX_BN + ((uint32_t)lane_base << 16);
            const int row = m0 + (int)rank * PF_BM + lane_base + lane;
            if (nkb > 0 && !wait(accum0 + 8u * buf, (j >> 1) & 1, DEV_ERR_PF_ACCUM)) break;
            tc_fence_after();
            const int chunks = min(p.bn, p.N - n0 + 31) / 32;
#pragma unroll 1
            for (int c = 0; c < chunks; ++c) {
                float v[32];
                if (nkb > 0) {
                    tmem_ld32(acc + (uint32_t)c * 32u, v);
                } else {
#pragma unroll
                    for (int i = 0; i < 32; ++i) v[i] = 0.0f;
                }
                if (c == chunks - 1) {  // the accumulator may be overwritten
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if constexpr (CG == 2) mbar_arrive_cluster(cluster_addr(drained0 + 8u * buf, 0));
                        else mbar_arrive(drained0 + 8u * buf);
                    }
                }
                if (p.qrows != nullptr) {
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        v[i] *= *reinterpret_cast<const float*>(p.qrows + (size_t)(n0 + c * 32 + i) * p.qstride + p.qscale_off);
                }
                if (row < p.M) epi(row, n0 + c * 32, v);
            }
            ++j;
        }
    }
    if (__any_sync(0xffffffffu, failed)) {  // give copies that may still be in flight time to land before the CTA leaves
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
    }
    tc_fence_before();
    if constexpr (CG == 2) cluster_sync();
    else __syncthreads();
    if (warp == 1) tmem_dealloc<CG>(tmem_base, 2 * PF_MAX_BN);
    if constexpr (CG == 2) cluster_sync();
}

// ------------------------------------------------------------------ the GEMM for a handful of rows
// Multi-sample decode has at most 16 activation rows, so the operands swap roles: the weight
// tile [128 features][64] is the M-side operand (every staged byte is useful) and the
// activations are the N side, [NB rows][64] with rows 0-15 the hi parts and rows 16-31 the lo
// parts of the samples (NB = 16 without the lo parts).  D[feature lane][row column] in tensor
// memory; an epilogue thread owns one feature and adds column j + 16 to column j.  One CTA per
// 128 features and K slice.  The kernel is a weight stream; what bounds it is what a CTA has in flight, and its start and
// end: eight 20 KB stages where every CTA has an SM of its own, five where two share one (a step of eight samples of
// the 5B model 2.96 ms with five everywhere, 2.80 ms so).  Requesting 24-96 MB of the next matrix into L2 behind a kernel's own
// loads made the step 5-8 % slower, four accumulators for a step's four MMAs changed nothing, and neither did
// cutting K among the CTAs of a cluster (192 CTAs instead of 96 for q|k|v) or into twice as many slices.
constexpr int SK_ROWS = 16;  // samples per call at most
template <int NB> struct SkTile {
    static constexpr uint32_t A_BYTES = 128 * PF_BK * 2, B_BYTES = NB * PF_BK * 2, STAGE = A_BYTES + 2048 * ((B_BYTES + 2047) / 2048);
    static constexpr int STAGES_ALONE = 8, STAGES_SHARED = 5;
    static constexpr size_t smem(int nst) { return (size_t)nst * STAGE + 1024 + 256; }
};

struct SkEpiPartial {  // this K slice's partial sums: part[slice][s][f] = y[s]
    float* part;
    int ld;
    __device__ void operator()(int f, bool valid, const float (&y)[SK_ROWS], int ns) const {
        if (!valid) return;
        float* p = part + (size_t)blockIdx.y * SK_ROWS * ld;
#pragma unroll
        for (int s = 0; s < SK_ROWS; ++s)
            if (s < ns) p[(size_t)s * ld + f] = y[s];
    }
};
struct SkEpiStore {  // out[s][f] = y[s]
    float* out;
    int ld;
    __device__ void operator()(int f, bool valid, const float (&y)[SK_ROWS], int ns) const {
        if (!valid) return;
#pragma unroll
        for (int s = 0; s < SK_ROWS; ++s)
            if (s < ns) out[(size_t)s * ld + f] = y[s];
    }
};
template <typename T16> struct SkEpiGate {  // features (2j, 2j+1) = (w1, w3) column j sit in neighbouring lanes
    T16* gate;
    T16* gate_lo;
    int ld, act;
    __device__ void operator()(int f, bool valid, const float (&y)[SK_ROWS], int ns) const {
#pragma unroll
        for (int s = 0; s < SK_ROWS; ++s) {
            if (s >= ns) break;  // uniform across the warp
            const float y3 = __shfl_xor_sync(0xffffffffu, y[s], 1);
            if (valid && !(f & 1)) {
                const float y1 = y[s];
                float a;
                if (act == 1) {
                    const float l = fmaxf(y1, 0.5f * y1);
                    a = l * l;
                } else {
                    a = y1 / (1.0f + expf(-y1));
                }
                pf_store(gate, gate_lo, (size_t)s * ld + (f >> 1), a * y3);
            }
        }
    }
};
template <typename T16> struct SkEpiQKV {  // RoPE pairs sit in neighbouring lanes; q fp32 per sample, k / v into the sample's page
    float* q;
    T16* kv_pool;
    const int* page_table;  // [samples][pages_per_seq]
    const float2* rope;
    const DevState* st;  // the samples' common position (read on the device: one captured graph serves every step)
    int Q, KV, hd, kv_heads, page_tokens, pages_per_seq;
    __device__ void operator()(int f, bool valid, const float (&y)[SK_ROWS], int ns) const {
        const int pos = __ldcg(&st->pos);
        const bool roped = f < Q + KV;
        float2 cs = make_float2(1.0f, 0.0f);
        if (valid && roped) cs = rope[(size_t)pos * (hd >> 1) + ((f % hd) >> 1)];
        const int kv01 = f < Q + KV ? 0 : 1;
        const int ck = f - Q - kv01 * KV, head = ck / hd, d = ck % hd;
#pragma unroll
        for (int s = 0; s < SK_ROWS; ++s) {
            if (s >= ns) break;  // uniform across the warp
            const float p = __shfl_xor_sync(0xffffffffu, y[s], 1);
            if (!valid) continue;
            float r = y[s];
            if (roped) r = (f & 1) ? y[s] * cs.x + p * cs.y : y[s] * cs.x - p * cs.y;
            if (f < Q) {
                q[(size_t)s * Q + f] = r;
            } else {
                const int page = page_table[(size_t)s * pages_per_seq + pos / page_tokens], off = pos % page_tokens;
                kv_pool[((((size_t)page * 2 + kv01) * kv_heads + head) * page_tokens + off) * hd + d] = pf_cast<T16>(r);
            }
        }
    }
};

template <int NB, class Epi>
__global__ void __launch_bounds__(PF_THREADS, 2)
pf_skinny_kernel(const __grid_constant__ CUtensorMap tma_w, const __grid_constant__ CUtensorMap tma_x, int N, int K, int ns, int nst, uint32_t idesc, int* err,
                 Epi epi) {
    using TL = SkTile<NB>;
    extern __shared__ unsigned char pf_raw[];
    const int n0 = blockIdx.x * 128;
    // blockIdx.y: which slice of K this CTA multiplies (a matrix with few rows is cut along K so that
    // enough CTAs stream it; the epilogue then stores a partial sum for the consumer to add up)
    const int nkb_all = (K + PF_BK - 1) / PF_BK, per = (nkb_all + (int)gridDim.y - 1) / (int)gridDim.y;
    const int kb_first = blockIdx.y * per, nkb = max(0, min(nkb_all, kb_first + per) - kb_first);
    const uint32_t tiles = (smem_addr(pf_raw) + 1023u) & ~1023u;
    const uint32_t bars = tiles + nst * TL::STAGE;
    const uint32_t full0 = bars, empty0 = bars + 8u * nst, accum = bars + 16u * nst, slot = accum + 8u;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < nst; ++s) {
            mbar_init(full0 + 8u * s, 1);
            mbar_init(empty0 + 8u * s, 1);
        }
        mbar_init(accum, 1);
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(slot, 32);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    uint32_t tmem_base;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(slot));
    bool failed = false;
    // whole warps wait and loop, one elected thread issues: with the loops in one thread a step took 890 clocks (see above), 16 KB a
    // CTA, which bound the kernel and not HBM (3.17 ms a step; 2.96)
    auto wait = [&](uint32_t bar, uint32_t parity, int code) {
        const bool ok = __all_sync(0xffffffffu, mbar_wait(bar, parity));
        if (!ok) {
            atomicExch(err, code);
            failed = true;
        }
        return ok;
    };
    if (warp == 0) {
        // Under programmatic dependent launch the first ring of weight tiles is requested before the previous kernel has
        // finished; the activations it produces are requested only after the wait.
        const int ahead = min(nst, nkb);
        if (elect_one()) {
            for (int kb = 0; kb < ahead; ++kb) {
                mbar_arrive_expect_tx(full0 + 8u * kb, TL::A_BYTES + TL::B_BYTES);
                tma_load_2d(tiles + kb * TL::STAGE, &tma_w, (kb_first + kb) * PF_BK, n0, full0 + 8u * kb);
            }
        }
        __syncwarp();
        pdl_wait();
        pdl_launch_dependents();
        if (elect_one()) {
            for (int kb = 0; kb < ahead; ++kb) tma_load_2d(tiles + kb * TL::STAGE + TL::A_BYTES, &tma_x, (kb_first + kb) * PF_BK, 0, full0 + 8u * kb);
        }
        __syncwarp();
        int s = 0, turn = 0;
        for (int kb = nst; kb < nkb; ++kb) {
            if (!wait(empty0 + 8u * s, turn, DEV_ERR_PF_EMPTY)) break;
            if (elect_one()) {
                const uint32_t a_dst = tiles + s * TL::STAGE;
                mbar_arrive_expect_tx(full0 + 8u * s, TL::A_BYTES + TL::B_BYTES);
                tma_load_2d(a_dst, &tma_w, (kb_first + kb) * PF_BK, n0, full0 + 8u * s);
                tma_load_2d(a_dst + TL::A_BYTES, &tma_x, (kb_first + kb) * PF_BK, 0, full0 + 8u * s);
            }
            __syncwarp();
            if (++s == nst) { s = 0; turn ^= 1; }
        }
    } else if (warp == 1) {
        int s = 0, turn = 0;
        for (int kb = 0; kb < nkb; ++kb) {
            if (!wait(full0 + 8u * s, turn, DEV_ERR_PF_FULL)) break;
            tc_fence_after();
            if (elect_one()) {
                const uint64_t adesc = umma_desc(tiles + s * TL::STAGE), bdesc = umma_desc(tiles + s * TL::STAGE + TL::A_BYTES);
#pragma unroll
                for (int k = 0; k < PF_BK / 16; ++k) umma_f16(tmem_base, adesc + 2u * k, bdesc + 2u * k, idesc, (kb | k) != 0);
                umma_commit(empty0 + 8u * s);
                if (kb == nkb - 1) umma_commit(accum);
            }
            __syncwarp();
            if (++s == nst) { s = 0; turn ^= 1; }
        }
    } else {
        const int lane_base = (warp & 3) * 32;
        const int f = n0 + lane_base + lane;
        pdl_wait();  // nothing is written before the previous kernel is complete
        if (nkb > 0 && !mbar_wait(accum, 0)) {
            atomicExch(err, DEV_ERR_PF_ACCUM);
            failed = true;
        }
        if (!failed) {
            tc_fence_after();
            float v[32];
            if (nkb > 0) {
                tmem_ld32(tmem_base + ((uint32_t)lane_base << 16), v);
            } else {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = 0.0f;
            }
            float y[SK_ROWS];
#pragma unroll
            for (int j = 0; j < SK_ROWS; ++j) y[j] = NB == 32 ? v[j] + v[j + 16] : v[j];
            epi(f, f < N, y, ns);
        }
    }
    if (__any_sync(0xffffffffu, failed)) {
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, 32);
}

// FP8 rows (Wfmt<Fp8Row>: K e4m3 bytes, then the row scale) to a [N][K] 16-bit matrix of the unscaled
// e4m3 values, which both 16-bit types hold exactly; the scale is applied to the GEMM's output column.
template <typename T16>
__global__ void __launch_bounds__(256) pf_widen_fp8_kernel(const unsigned char* __restrict__ rows, uint32_t stride, T16* __restrict__ out, int N, int K) {
    const size_t total = (size_t)N * (K / 4);
    for (size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x; j < total; j += (size_t)gridDim.x * blockDim.x) {
        const size_t r = j / (K / 4);
        const int c = (int)(j % (K / 4)) * 4;
        const uint32_t v = *reinterpret_cast<const uint32_t*>(rows + r * stride + c);
        const __half2 h01(__nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(v & 0xffffu), __NV_E4M3));
        const __half2 h23(__nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(v >> 16), __NV_E4M3));
        const float2 a = __half22float2(h01), b = __half22float2(h23);
        T16* o = out + r * K + c;
        o[0] = pf_cast<T16>(a.x); o[1] = pf_cast<T16>(a.y); o[2] = pf_cast<T16>(b.x); o[3] = pf_cast<T16>(b.y);
    }
}

// ------------------------------------------------------------------ small batched kernels
// token rows of the embedding table into the fp32 residual stream (cpu/embedding.rs:8-16)
template <typename WT>
__global__ void pf_embed_kernel(const WT* __restrict__ embed, const uint32_t* __restrict__ ids, float* __restrict__ x, int D) {
    const WT* row = embed + (size_t)ids[blockIdx.x] * D;
    for (int i = threadIdx.x; i < D; i += blockDim.x) x[(size_t)blockIdx.x * D + i] = Elem<WT>::to_f32(row[i]);
}

// the same with one token per sample, taken from the samples' device states
template <typename WT>
__global__ void pf_embed_samples_kernel(const WT* __restrict__ embed, DevState* __restrict__ st, float* __restrict__ x, int D, int vocab) {
    const WT* row = embed + (size_t)checked_token(st[blockIdx.x].token, vocab, &st[blockIdx.x].error) * D;
    for (int i = threadIdx.x; i < D; i += blockDim.x) x[(size_t)blockIdx.x * D + i] = Elem<WT>::to_f32(row[i]);
}

// x * rsqrt(mean(x^2) + eps) * gamma per row (cpu/rmsnorm.rs:149-183), written as 16-bit GEMM input
template <typename T16>
__global__ void __launch_bounds__(256) pf_rmsnorm_kernel(const float* __restrict__ x, const float* __restrict__ gamma, T16* __restrict__ out,
                                                         T16* __restrict__ out_lo, int D) {
    __shared__ float red[32];
    pdl_launch_dependents();  // a following weight-streaming kernel may start fetching; it waits before it reads `out`
    const float* row = x + (size_t)blockIdx.x * D;
    float ss = 0.0f;
    for (int i = threadIdx.x; i < D; i += blockDim.x) ss += row[i] * row[i];
    const float inv = 1.0f / sqrtf(block_sum(ss, red) * (1.0f / (float)D) + RMS_EPS);
    for (int i = threadIdx.x; i < D; i += blockDim.x) pf_store(out, out_lo, (size_t)blockIdx.x * D + i, row[i] * inv * gamma[i]);
}

// The same after folding in a linear that was cut along K: x += alpha * (sum of the slices' partial
// sums, in slice order), written back, then normalised.  One CTA of up to 1024 threads per row, four neighbouring entries a
// thread and turn, all slices' loads of a turn in flight: the kernel is one memory latency and two block-wide sums long.
template <typename T16>
__global__ void __launch_bounds__(1024) pf_reduce_rmsnorm_kernel(float* __restrict__ x, const float* __restrict__ part, int nslices, float alpha,
                                                                 const float* __restrict__ gamma, T16* __restrict__ out, T16* __restrict__ out_lo, int D) {
    __shared__ float red[32];
    constexpr int S = 8;  // slices at most
    pdl_wait();
    pdl_launch_dependents();
    float4* row = reinterpret_cast<float4*>(x + (size_t)blockIdx.x * D);
    const float4* p4 = reinterpret_cast<const float4*>(part + (size_t)blockIdx.x * D);
    const size_t slice = (size_t)SK_ROWS * D / 4;
    float ss = 0.0f;
    for (int i = threadIdx.x; i < D / 4; i += blockDim.x) {
        float4 v = __ldcg(row + i), p[S];
#pragma unroll
        for (int k = 0; k < S; ++k) p[k] = k < nslices ? __ldcg(p4 + k * slice + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < S; ++k) { a.x += p[k].x; a.y += p[k].y; a.z += p[k].z; a.w += p[k].w; }
        v.x += alpha * a.x; v.y += alpha * a.y; v.z += alpha * a.z; v.w += alpha * a.w;
        row[i] = v;
        ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    }
    const float inv = 1.0f / sqrtf(block_sum(ss, red) * (1.0f / (float)D) + RMS_EPS);
    for (int i = threadIdx.x; i < D / 4; i += blockDim.x) {  // (the entries this thread wrote)
        const float4 v = row[i], g = reinterpret_cast<const float4*>(gamma)[i];
        const float y[4] = {v.x * inv * g.x, v.y * inv * g.y, v.z * inv * g.z, v.w * inv * g.w};
        uint2 hi, lo;
        T16* h = reinterpret_cast<T16*>(&hi);
        T16* l = reinterpret_cast<T16*>(&lo);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            h[k] = pf_cast<T16>(y[k]);
            l[k] = pf_cast<T16>(y[k] - Elem<T16>::to_f32(h[k]));
        }
        reinterpret_cast<uint2*>(out + (size_t)blockIdx.x * D)[i] = hi;
        if (out_lo != nullptr) reinterpret_cast<uint2*>(out_lo + (size_t)blockIdx.x * D)[i] = lo;
    }
}

// ---------------------------------------------------------------------- tensor parallel: all-reduce of a [rows, dim] partial product
// After the row-sharded Wo / W2 GEMM every rank holds a partial y_r in one of its two buffers of the link region.
// tp_pf_publish_kernel tells every peer so (a sequence number into the peer's flag row, after a system-scope
// fence); tp_pf_reduce_kernel waits (bounded) until all ranks have published `seq`, then x += alpha * sum_r y_r
// with the ranks' buffers read over NVLink and added in rank order, so every rank keeps a bit-identical residual
// stream.  Two buffers alternate: a rank overwrites a buffer only after it has seen every rank publish the
// all-reduce in between, i.e. after every rank finished reading it.
static __global__ void tp_pf_publish_kernel(TpLink tp, size_t flags_off, int buf, unsigned int seq) {
    __threadfence_system();
    if ((int)threadIdx.x < tp.world)
        st_release_sys(reinterpret_cast<unsigned int*>(tp.peers[threadIdx.x] + flags_off) + buf * tp.world + tp.rank, seq);
}

static __global__ void __launch_bounds__(256)
tp_pf_reduce_kernel(TpLink tp, size_t flags_off, size_t buf_off, int buf, unsigned int seq, float* __restrict__ x, int rows, size_t buf_rows,
                    float alpha, int* err) {
    __shared__ int s_ok;
    if (threadIdx.x == 0) s_ok = 1;
    __syncthreads();
    if ((int)threadIdx.x < tp.world) {
        const unsigned int* f = reinterpret_cast<const unsigned int*>(tp.peers[tp.rank] + flags_off) + buf * tp.world + threadIdx.x;
        if (!tp_wait_flag(f, seq, tp.st, tp.wait_ns)) { atomicCAS(err, 0, DEV_ERR_TP_WAIT); s_ok = 0; }
    }
    __syncthreads();
    if (!s_ok) return;
    const size_t n4 = (size_t)rows * tp.dim / 4, off = buf_off + (size_t)buf * buf_rows * tp.dim * 4;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (size_t)gridDim.x * blockDim.x) {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int r = 0; r < tp.world; ++r) {  // rank order; L2-only loads: the buffers are rewritten every other all-reduce
            const float4 v = __ldcg(reinterpret_cast<const float4*>(tp.peers[r] + off) + i);
            a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
        }
        float4 t = reinterpret_cast<float4*>(x)[i];
        t.x += alpha * a.x; t.y += alpha * a.y; t.z += alpha * a.z; t.w += alpha * a.w;
        reinterpret_cast<float4*>(x)[i] = t;
    }
}

}  // namespace cd
