// Attention of a prompt in one kernel (tcgen05): scores, causal / windowed softmax and the product with V never leave the
// chip.  No batched counterpart in the reference (its decoder feeds prompt tokens one at a time, inference.rs:650-670); the
// math is sdpa_fwd.rs:36-46, :325-354 restricted to the visible keys.  The method is FlashAttention (Dao et al. 2022) in the form
// published for this architecture (FlashAttention-4): tiles of keys with a running softmax, two query tiles in turns, a reference
// that is seldom raised.
//
// One CTA = 256 query rows of one head, as two tiles of 128 that take turns: while one tile's softmax runs on its four
// warps, the tensor cores work on the other one.  Warps 0-3 / 4-7: softmax of tile 0 / 1, a query row per thread.
// Warp 8: TMA producer.  Warp 9: owns the tensor memory, issues the MMAs.  (Warps 10, 11 complete their warpgroup, whose
// registers go to the softmax: 12 warps of 168 at launch, 8 x 216 + 4 x 72 behind the split.)
// q and the probabilities enter the products as 16-bit hi + lo pairs against K and V as cached (two MMAs per product, about
// 22 mantissa bits with an fp16 cache); scores, softmax and the accumulators are fp32.  The probabilities are relative to a
// running reference that is raised only when a row's maximum has grown by more than 2^8, so the accumulator in tensor memory
// is rarely rescaled; the row's sum uses the same reference, and the division at the end cancels it.
//
// Tensor memory (512 columns): S of tile q at 128 q, O of tile q at 256 + 128 q.  A row's probabilities overwrite its scores
// (64 columns hi, 64 columns lo, two 16-bit values per column) and are the A operand of the second product from there.
// Shared memory: q hi + lo of both tiles, then a ring of three tiles of 128 keys (K, V, K, V, ...), all in the 128-byte
// swizzle; V is read as an MN-major operand, so nothing transposes it.
//
// What bounds it: the tensor pipe (per 128 x 128 scores at width 128: 4 x 512 clocks of MMA, against 1024 of exponentials
// and about as many of conversions per softmax warp).  Measured per layer of the 5B model (32 heads of 128, causal): 1024
// tokens 51 us, 4096 tokens 401 us = 343 TFLOP/s of scores and products as the model counts them, twice that issued.  The
// separate kernels it replaced (score GEMM, softmax, P V GEMM, transposed V) took 268 and 2170 us.
#pragma once
#include "prefill.cuh"

namespace cd {

constexpr int PA_KEYS = 128, PA_ROWS = 256, PA_THREADS = 384, PA_RING = 3;
constexpr int PA_REGS = 256 * 216 + 128 * 72;  // registers of the split: what a block has to hold at launch
enum { DEV_ERR_PA_WAIT = 11 };

struct PfAttn {
    int rows, pos0;          // query rows of this pass, position of the first
    int window;              // positions a query sees, itself included; 0: all
    int maps, group;         // query vectors per head (blockIdx.y = head * maps + map), heads per kv head
    int page_tokens;         // divides 128, or is a multiple of it
    int split;               // 1: q arrives as hi + lo, the probabilities are split likewise
    float scale_log2;        // score scale * log2(e)
    const float* slopes;     // distance bias per head (BIAS), subtracted as slope * (query position - key position)
    int* err;
};

template <int KD, int VD> struct PaSmem {
    static constexpr uint32_t Q_TILE = 128 * KD * 2, SLOT = PA_KEYS * (KD > VD ? KD : VD) * 2;
    static constexpr size_t BYTES = (size_t)4 * Q_TILE + (size_t)PA_RING * SLOT + 1024 /* alignment */ + 256 /* barriers */;
};

__device__ inline void tma_load_4d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
// A operand from tensor memory
__device__ inline void umma_f16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ inline void tmem_ld32_start(uint32_t taddr, float* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]),
                   "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]),
                   "=f"(v[16]), "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]),
                   "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
                 : "r"(taddr) : "memory");
}
__device__ inline void tmem_ld32_use(float* v) {  // the values may be read from here on (behind tcgen05.wait::ld)
    asm volatile("" : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]), "+f"(v[6]), "+f"(v[7]),
                      "+f"(v[8]), "+f"(v[9]), "+f"(v[10]), "+f"(v[11]), "+f"(v[12]), "+f"(v[13]), "+f"(v[14]), "+f"(v[15]),
                      "+f"(v[16]), "+f"(v[17]), "+f"(v[18]), "+f"(v[19]), "+f"(v[20]), "+f"(v[21]), "+f"(v[22]), "+f"(v[23]),
                      "+f"(v[24]), "+f"(v[25]), "+f"(v[26]), "+f"(v[27]), "+f"(v[28]), "+f"(v[29]), "+f"(v[30]), "+f"(v[31]));
}
// 128 columns with all four loads in flight
__device__ inline void tmem_ld128(uint32_t taddr, float (&v)[128]) {
#pragma unroll
    for (int c = 0; c < 4; ++c) tmem_ld32_start(taddr + 32u * c, v + 32 * c);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int c = 0; c < 4; ++c) tmem_ld32_use(v + 32 * c);
}
__device__ inline void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
                   "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
                   "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(taddr) : "memory");
}
__device__ inline void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// MN-major operand as TMA writes it: rows of 64 elements (128 bytes, swizzled) of the N extent, one row per step of K; 8 rows
// are 1024 bytes, the next 64 elements of N `n_block` bytes further
__device__ inline uint64_t umma_desc_mn(uint32_t tile_smem, uint32_t n_block) {
    uint64_t d = (uint64_t)((tile_smem & 0x3FFFFu) >> 4);
    d |= (uint64_t)(n_block >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
__device__ inline float exp2_fast(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// two fp32 values as packed 16-bit heads, and the packed remainders
template <typename T16> __device__ inline uint32_t pa_split(float a, float b, uint32_t& lo);
template <> __device__ inline uint32_t pa_split<__half>(float a, float b, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
    lo = *reinterpret_cast<const uint32_t*>(&l);
    return *reinterpret_cast<const uint32_t*>(&h);
}
template <> __device__ inline uint32_t pa_split<__nv_bfloat16>(float a, float b, uint32_t& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    const uint32_t u = *reinterpret_cast<const uint32_t*>(&h);
    const __nv_bfloat162 l = __floats2bfloat162_rn(a - __uint_as_float(u << 16), b - __uint_as_float(u & 0xffff0000u));
    lo = *reinterpret_cast<const uint32_t*>(&l);
    return u;
}

// Epilogue of the dense family: heads side by side in the [rows, heads * VD] operand of the output projection.
template <typename T16> struct PaOut {
    T16* out;
    T16* out_lo;
    int ld, hd;
    __device__ float factor(int, int, float, float l) const { return 1.0f / l; }
    __device__ void operator()(int z, int row, int col, const float (&v)[32]) const { pf_store_run(out, out_lo, (size_t)row * ld + z * hd + col, v); }
};

template <typename KT, int KD, int VD, bool BIAS, class Epi>
__global__ void __launch_bounds__(PA_THREADS, 1)
pf_attn_kernel(const __grid_constant__ CUtensorMap tma_q, const __grid_constant__ CUtensorMap tma_q_lo, const __grid_constant__ CUtensorMap tma_k,
               const __grid_constant__ CUtensorMap tma_v, const __grid_constant__ PfAttn p, uint32_t idesc_s, uint32_t idesc_o, Epi epi) {
    using SM = PaSmem<KD, VD>;
    constexpr uint32_t TM_O = 256;
    constexpr int KB = KD / 64, VB = VD / 64;
    extern __shared__ unsigned char pf_raw[];
    const uint32_t q_smem = (smem_addr(pf_raw) + 1023u) & ~1023u;  // [tile][hi, lo][KB][128][64]
    const uint32_t ring = q_smem + 4 * SM::Q_TILE;
    const uint32_t bars = ring + PA_RING * SM::SLOT;
    const uint32_t q_full = bars, full0 = bars + 8u, empty0 = full0 + 8u * PA_RING, s_full = empty0 + 8u * PA_RING, p_full = s_full + 16u, o_done = p_full + 16u,
                   slot = o_done + 16u;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int z = blockIdx.y, h = z / p.maps, map = z % p.maps, kvh = h / p.group;
    const int row0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * PA_ROWS;  // the rows with the most keys first
    // key tiles [jb, je) a query tile sees
    auto first_tile = [&](int q) { return p.window > 0 ? max(0, p.pos0 + row0 + 128 * q - p.window + 1) / PA_KEYS : 0; };
    auto last_tile = [&](int q) { return row0 + 128 * q >= p.rows ? 0 : (p.pos0 + min(p.rows, row0 + 128 * q + 128) - 1) / PA_KEYS + 1; };
    const int jb[2] = {first_tile(0), first_tile(1)}, je[2] = {last_tile(0), last_tile(1)};
    const int j0 = jb[0], j1 = max(je[0], je[1]);

    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        for (int s = 0; s < PA_RING; ++s) {
            mbar_init(full0 + 8u * s, 1);
            mbar_init(empty0 + 8u * s, 1);
        }
        for (int q = 0; q < 2; ++q) {
            mbar_init(s_full + 8u * q, 1);
            mbar_init(p_full + 8u * q, 4);  // one arrival per softmax warp
            mbar_init(o_done + 8u * q, 1);
        }
        mbar_fence_init();
    }
    if (warp == 9) tmem_alloc(slot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    uint32_t tmem;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(slot));
    bool failed = false;
    auto wait = [&](uint32_t bar, uint32_t parity) {  // one thread
        if (!failed && !mbar_wait(bar, parity)) {
            atomicCAS(p.err, 0, DEV_ERR_PA_WAIT);
            failed = true;
        }
        return !failed;
    };
    auto wait_warp = [&](uint32_t bar, uint32_t parity) {  // a whole warp, which goes on or gives up together
        if (!__all_sync(0xffffffffu, mbar_wait(bar, parity))) {
            atomicCAS(p.err, 0, DEV_ERR_PA_WAIT);
            failed = true;
        }
        return !failed;
    };

    if (warp >= 8) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
        if (warp == 8 && lane == 0) {  // ---- TMA producer: q of both tiles, then K and V tiles in turn
            mbar_arrive_expect_tx(q_full, (p.split ? 4u : 2u) * SM::Q_TILE);
            for (int q = 0; q < 2; ++q)
                for (int b = 0; b < KB; ++b) {
                    const uint32_t dst = q_smem + (uint32_t)q * 2u * SM::Q_TILE + (uint32_t)b * 16384u;
                    tma_load_2d(dst, &tma_q, z * KD + b * 64, row0 + 128 * q, q_full);
                    if (p.split) tma_load_2d(dst + SM::Q_TILE, &tma_q_lo, z * KD + b * 64, row0 + 128 * q, q_full);
                }
            int n = 0;
            for (int j = j0; j < j1 && !failed; ++j) {
                const int key = j * PA_KEYS, page = key / p.page_tokens, off = key % p.page_tokens;
                for (int v = 0; v < 2; ++v, ++n) {
                    const int s = n % PA_RING;
                    if (n >= PA_RING && !wait(empty0 + 8u * s, (n / PA_RING - 1) & 1)) break;
                    const uint32_t dst = ring + (uint32_t)s * SM::SLOT;
                    mbar_arrive_expect_tx(full0 + 8u * s, (uint32_t)PA_KEYS * (v ? VD : KD) * 2u);
                    if (v) for (int b = 0; b < VB; ++b) tma_load_4d(dst + (uint32_t)b * 16384u, &tma_v, b * 64, off, kvh, page, full0 + 8u * s);
                    else for (int b = 0; b < KB; ++b) tma_load_4d(dst + (uint32_t)b * 16384u, &tma_k, map * KD + b * 64, off, kvh, page, full0 + 8u * s);
                }
            }
        }
        if (warp == 9 && lane == 0 && wait(q_full, 0)) {  // ---- MMA issuer
            // stage 2 (j - j0) holds K of tile j, the next one V
            auto k_stage = [&](int j) { return 2 * (j - j0); };
            auto scores = [&](int q, int j) {  // S_q = q K_j^T
                const uint32_t qs = q_smem + (uint32_t)q * 2u * SM::Q_TILE, ks = ring + (uint32_t)(k_stage(j) % PA_RING) * SM::SLOT;
#pragma unroll
                for (int b = 0; b < KB; ++b) {
                    const uint64_t a = umma_desc(qs + (uint32_t)b * 16384u), al = umma_desc(qs + SM::Q_TILE + (uint32_t)b * 16384u), kd = umma_desc(ks + (uint32_t)b * 16384u);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        umma_f16(tmem + 128u * q, a + 2u * k, kd + 2u * k, idesc_s, (b | k) != 0);
                        if (p.split) umma_f16(tmem + 128u * q, al + 2u * k, kd + 2u * k, idesc_s, 1u);
                    }
                }
                umma_commit(s_full + 8u * q);
            };
            auto full = [&](int st) {
                if (!wait(full0 + 8u * (st % PA_RING), (st / PA_RING) & 1)) return false;
                tc_fence_after();
                return true;
            };
            int done[2] = {0, 0};
            if (j0 < j1 && full(0)) {
                for (int q = 0; q < 2; ++q)
                    if (jb[q] <= j0 && j0 < je[q]) scores(q, j0);
                umma_commit(empty0);
            }
            for (int j = j0; j < j1 && !failed; ++j) {
                const int vst = k_stage(j) + 1, kst = vst + 1;
                if (!full(vst)) break;
                if (j + 1 < j1 && !full(kst)) break;
                for (int q = 0; q < 2 && !failed; ++q) {
                    if (jb[q] <= j && j < je[q]) {  // O_q += P_q V_j
                        if (!wait(p_full + 8u * q, done[q] & 1)) break;
                        done[q] += 1;
                        tc_fence_after();
                        const uint32_t vs = ring + (uint32_t)(vst % PA_RING) * SM::SLOT;
#pragma unroll
                        for (int k = 0; k < PA_KEYS / 16; ++k) {
                            const uint64_t vd = umma_desc_mn(vs + (uint32_t)k * 2048u, 16384u);
                            umma_f16_ta(tmem + TM_O + 128u * q, tmem + 128u * q + 8u * k, vd, idesc_o, (j > jb[q]) || k != 0);
                            if (p.split) umma_f16_ta(tmem + TM_O + 128u * q, tmem + 128u * q + 64u + 8u * k, vd, idesc_o, 1u);
                        }
                        umma_commit(o_done + 8u * q);
                    }
                    // (the MMAs run in the order they are issued: these scores overwrite the probabilities read just before)
                    if (j + 1 < j1 && jb[q] <= j + 1 && j + 1 < je[q]) scores(q, j + 1);
                }
                umma_commit(empty0 + 8u * (vst % PA_RING));
                if (j + 1 < j1) umma_commit(empty0 + 8u * (kst % PA_RING));
            }
        }
    } else {  // ---- softmax, a query row per thread
        asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
        const int q = warp >> 2, quad = warp & 3;
        const int row = row0 + 128 * q + 32 * quad + lane, pos = p.pos0 + row;
        const uint32_t lanes = (uint32_t)(32 * quad) << 16;
        const uint32_t ts = tmem + lanes + 128u * q, to = tmem + lanes + TM_O + 128u * q;
        const int nkeys = p.pos0 + p.rows;
        const float slope = BIAS ? p.slopes[h] * 1.4426950408889634f : 0.0f;
        float ref = -1e30f, sum = 0.0f;  // reference of the exponents (log2), sum of the probabilities relative to it
        int n = 0;
        for (int j = jb[q]; j < je[q] && !failed; ++j, ++n) {
            if (!wait_warp(s_full + 8u * q, n & 1)) break;
            tc_fence_after();
            float s[128];
            tmem_ld128(ts, s);
            const int key0 = j * PA_KEYS;
            const int first_pos = p.pos0 + row0 + 128 * q;
            // whole tile visible to every row of this query tile?
            const bool inner = key0 + PA_KEYS - 1 <= first_pos && (p.window <= 0 || key0 > first_pos + 127 - p.window);
            float mx = -INFINITY;
            if (BIAS) {
                const float d0 = (float)(pos - key0);
#pragma unroll
                for (int i = 0; i < 128; ++i) s[i] = fmaf(-slope, d0 - (float)i, s[i] * p.scale_log2);
            }
            if (!inner) {
                const int hi = pos - key0, lo = p.window > 0 ? hi - p.window : -1;  // visible: lo < i <= hi
#pragma unroll
                for (int i = 0; i < 128; ++i) s[i] = i <= hi && i > lo ? s[i] : -INFINITY;
            }
#pragma unroll
            for (int i = 0; i < 128; ++i) mx = fmaxf(mx, s[i]);
            const float c = BIAS ? 1.0f : p.scale_log2;
            mx *= c;
            // raise the reference where a row's maximum has outgrown it
            if (__any_sync(0xffffffffu, mx > ref + 8.0f)) {
                const float nref = mx > ref + 8.0f ? mx : ref;
                const float f = exp2_fast(ref - nref);
                ref = nref;
                sum *= f;
                if (n > 0) {
                    if (!wait_warp(o_done + 8u * q, (n - 1) & 1)) break;
                    tc_fence_after();
#pragma unroll 1
                    for (int b = 0; b < VD / 32; ++b) {
                        float o[32];
                        tmem_ld32(to + 32u * b, o);
                        uint32_t r[32];
#pragma unroll
                        for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(o[i] * f);
                        tmem_st32(to + 32u * b, r);
                    }
                }
            }
            float part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int b = 0; b < 2; ++b) {  // 64 keys: 32 columns hi, 32 columns lo
                uint32_t hi[32], lo[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    const float u = exp2_fast(fmaf(s[64 * b + 2 * i], c, -ref)), v = exp2_fast(fmaf(s[64 * b + 2 * i + 1], c, -ref));
                    part[i & 3] += u + v;
                    hi[i] = pa_split<KT>(u, v, lo[i]);
                }
                tmem_st32(ts + 32u * b, hi);
                if (p.split) tmem_st32(ts + 64u + 32u * b, lo);
            }
            sum += (part[0] + part[1]) + (part[2] + part[3]);
            tmem_st_wait();
            if (key0 + PA_KEYS > nkeys) {
                // rows of V behind the last key: their probabilities are zero, and whatever the cache holds there must not
                // become NaN in the product
                const int st = 2 * (j - j0) + 1;
                if (!wait_warp(full0 + 8u * (st % PA_RING), (st / PA_RING) & 1)) break;
                const uint32_t vs = ring + (uint32_t)(st % PA_RING) * SM::SLOT;
                const int dead = key0 + PA_KEYS - nkeys;  // rows 128 - dead .. 127
                for (int i = threadIdx.x & 127; i < dead * VB * 8; i += 128) {
                    const int b = i / (dead * 8), r = (i / 8) % dead;
                    asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(vs + (uint32_t)b * 16384u + (uint32_t)(PA_KEYS - dead + r) * 128u + (uint32_t)(i & 7) * 16u), "r"(0u) : "memory");
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full + 8u * q);
        }
        if (n > 0 && !failed && wait_warp(o_done + 8u * q, (n - 1) & 1)) {
            tc_fence_after();
            const float f = row < p.rows ? epi.factor(z, row, ref, sum) : 0.0f;
#pragma unroll 1
            for (int b = 0; b < VD / 32; ++b) {
                float v[32];
                tmem_ld32(to + 32u * b, v);
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] *= f;
                if (row < p.rows) epi(z, row, 32 * b, v);
            }
        }
    }
    if (__any_sync(0xffffffffu, failed)) {  // give copies that may still be in flight time to land before the CTA leaves
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 9) tmem_dealloc(tmem, 512);
}

}  // namespace cd
