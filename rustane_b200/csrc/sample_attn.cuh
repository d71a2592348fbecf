// Attention of one step of several samples that share a prompt (SampleAttn): every sample sits at the same position, the
// prompt's full pages are common, later pages a sample's own.
//
// Scores against the shared positions are a product with M = (sample, q head) pairs that look at one kv head: mma.m16n8k16,
// eight pairs a block, their q split into three 16-bit parts in rows 0-7 and 8-15, so one instruction gives two parts of eight
// positions' scores and no shuffle adds them up.  Probabilities and their products with V stay fp32 FMAs.
//
// grid = (kv heads, slices, blocks of pairs).  The first slices cut the shared positions; the slices behind them cut the samples' own
// positions, each the same positions of all samples of the block.  A CTA has four warps; a warp takes sixteen positions (of one
// sample, where they are its own) at a time; K and V go from global memory to registers in the layout their use needs.  Shared
// positions are requested ahead of griddepcontrol.wait: they are older than the step.  The CTA that arrives last for its block
// (a counter, nobody waits) merges the slices in slice order and leaves the output as the hi + lo operand of the GEMM that follows.
//
// What bounds it: the chain of latencies behind q (its load, scores, softmax, the merge of warps, the last arriver's merge);
// the bytes (16.8 MB a layer of the 5B model at 1024 positions) are there before q is.  One CUDA-core CTA per q head, slice and two
// samples, with five shuffles per position, head and sample, took 33 us of the layer; a conversion kernel followed.
#pragma once
#include <type_traits>

#include "common.cuh"
#include "sample_split.h"

namespace cd {

struct SampleAttn {
    const float* q;          // [samples][heads][hd]
    const int* page_table;   // [samples][pages_per_seq]
    const DevState* st;      // the samples' common position
    float *part_acc, *part_ml;  // [samples][heads][max_slices][hd], [...][2] (max, sum)
    unsigned int* counters;  // [blocks][kv heads], zero between launches
    int kv_heads, page_tokens, pages_per_seq, max_slices, shared_tokens;
    SaBlocks blocks;
    SaSplit split;
    float scale;
};

// T16: the following GEMM's operand; out[sample][heads * hd] its hi part, out_lo (or nullptr) the remainder
template <typename KT, typename T16, int HD>
__global__ void __launch_bounds__(SA_THREADS, SA_PER_SM)
sample_attn_kernel(const __grid_constant__ SampleAttn p, const KT* __restrict__ kv_pool, T16* __restrict__ out, T16* __restrict__ out_lo) {
    using X = Mma16<KT>;
    constexpr bool SCALED = std::is_same<KT, __half>::value;
    constexpr float NEG = -3.402823466e+38f;
    constexpr int CH = HD / 8, SIDES = 32 / CH, NV = 16 / SIDES, NK = CH / 4;  // 16-byte chunks of a row; V rows side by side, and in turn; K chunks a lane
    constexpr int LDQ = HD + 4;                                                 // (rows of q on different banks)
    __shared__ __align__(16) float qs[SA_ROWS * LDQ];
    __shared__ __align__(16) float probs_all[4][16 * SA_ROWS];
    __shared__ __align__(16) float accs[4][SA_ROWS * HD];
    __shared__ float ms[4][SA_ROWS], ls[4][SA_ROWS], down[SA_ROWS];
    __shared__ int is_last;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int kvh = blockIdx.x, slice = blockIdx.y, gqa = p.blocks.gqa, heads = p.kv_heads * gqa;
    const int hb = blockIdx.z % p.blocks.head_blocks(), z0 = blockIdx.z / p.blocks.head_blocks() * p.blocks.per_block();
    const int nz = min(p.blocks.per_block(), p.blocks.samples - z0), h0 = hb * SA_ROWS, nh = min(p.blocks.heads(), gqa - h0);
    const int rows = nz * nh;  // row r: sample z0 + r / nh, q head kvh gqa + h0 + r % nh
    const bool own = slice >= p.split.shared;
    auto row_at = [&](int r) { return (size_t)(z0 + r / nh) * heads + kvh * gqa + h0 + r % nh; };

    // the position is older than the kernel ahead; a slice of shared positions requests its first ones before that one ends
    const int end = own ? __ldcg(&p.st->pos) + 1 : p.shared_tokens;
    const size_t head_stride = (size_t)p.page_tokens * HD, page_stride = (size_t)2 * p.kv_heads * head_stride, v_off = (size_t)p.kv_heads * head_stride;
    // turn i of this warp: positions w0 .. w0 + 15 (below `end`), as sample z0 + z has them
    int w0 = 0, z = 0;
    auto turn = [&](int i) {
        if (!own) {
            w0 = (slice * p.split.rounds + i) * SA_TILE + warp * SA_WARP_TILE;
            return i < p.split.rounds && w0 < end;
        }
        const int task = warp + 4 * i;
        z = task % nz;
        w0 = p.shared_tokens + ((slice - p.split.shared) * p.split.spans + task / nz) * SA_WARP_TILE;
        return task < nz * p.split.spans && w0 < end;
    };
    uint4 kw[2][NK], vw[NV];
    const int vch = lane % CH, vside = lane / CH;
    auto row_of = [&](int pos) {
        const int page = p.page_table[(size_t)(z0 + z) * p.pages_per_seq + pos / p.page_tokens];
        return kv_pool + (size_t)page * page_stride + (size_t)kvh * head_stride + (size_t)(pos % p.page_tokens) * HD;
    };
    auto fetch_k = [&]() {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int pos = w0 + 8 * j + g;
            const KT* row = pos < end ? row_of(pos) : nullptr;
#pragma unroll
            for (int i = 0; i < NK; ++i) kw[j][i] = row != nullptr ? ldg_stream_coherent(row + (4 * i + t) * 8) : make_uint4(0, 0, 0, 0);
        }
    };
    auto fetch_v = [&]() {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int pos = w0 + vside + SIDES * i;
            vw[i] = pos < end ? ldg_stream_coherent(row_of(pos) + v_off + vch * 8) : make_uint4(0, 0, 0, 0);
        }
    };
    bool more = turn(0);
    if (!own && more) { fetch_k(); fetch_v(); }
    pdl_wait();
    pdl_launch_dependents();
    if (own && more) { fetch_k(); fetch_v(); }

    // q of the block's rows, sixteen threads a row, times the row's power of two (largest magnitude to [2^14, 2^15)) for fp16
    {
        const int r = tid >> 4, c = tid & 15;
        constexpr int N4 = HD / 64;
        float4 v[N4];
        float mx = 0.0f;
#pragma unroll
        for (int i = 0; i < N4; ++i) {
            v[i] = r < rows ? __ldcg(reinterpret_cast<const float4*>(p.q + row_at(r) * HD) + c + 16 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
            mx = fmaxf(fmaxf(fmaxf(mx, fabsf(v[i].x)), fmaxf(fabsf(v[i].y), fabsf(v[i].z))), fabsf(v[i].w));
        }
        float up = 1.0f, dn = 1.0f;
        if (SCALED) {
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const int e = (int)(__float_as_uint(mx) >> 23), f = e == 255 ? 127 : min(253, max(1, 268 - e));
            up = __uint_as_float((uint32_t)f << 23);
            dn = __uint_as_float((uint32_t)(254 - f) << 23);
        }
#pragma unroll
        for (int i = 0; i < N4; ++i)
            *reinterpret_cast<float4*>(qs + r * LDQ + 4 * (c + 16 * i)) = make_float4(v[i].x * up, v[i].y * up, v[i].z * up, v[i].w * up);
        if (c == 0) down[r] = dn * p.scale;
    }
    __syncthreads();

    float acc[SA_ROWS][8], m = NEG, lsum = 0.0f;  // m, lsum: of row g (lsum of this lane's positions)
#pragma unroll
    for (int r = 0; r < SA_ROWS; ++r)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[r][i] = 0.0f;
    float* probs = probs_all[warp];
    const float dn = down[g];
    for (int i = 0; more;) {  // (uniform in the warp)
        const bool seen = g < rows && (!own || g / nh == z);  // a sample's own positions are its rows' only
        const int at = w0, zt = z;
        {
            // A step's product starts at zero and is added in fp32: an MMA truncates where it adds to its accumulator, and the chain of
            // them through a head's 128 elements left 2.1 times the error of fp32 FMAs in the output (7.1e-7 and 3.4e-7 behind 1024
            // positions).  So, with q's 24 bits and one rounding less ahead of the exponential, it is 0.83 to 1.11 times
            // theirs (heads of 64 and 128, 12 to 1044 positions, even and heavy-tailed q; 16 seeds each); the 5B model's eight
            // samples take 47.7 ms a call instead of 47.3.
            float c[2][4] = {}, even[2][4];
#pragma unroll
            for (int s = 0; s < HD / 16; ++s) {  // step s: elements 4 b .. 4 b + 3, b = s % 2, of chunk 4 (s / 2) + t
                float4 v = *reinterpret_cast<const float4*>(qs + g * LDQ + (4 * (s >> 1) + t) * 8 + 4 * (s & 1));
                // hi parts in rows 0-7, the next in rows 8-15; the third joins the second's sum.  Together they hold all 24 bits (fp16: of
                // a value within 2^-15 of the row's largest)
                uint32_t a[3], b[3];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    a[k] = X::part(v.x, v.y);
                    b[k] = X::part(v.z, v.w);
                }
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const uint32_t k0 = (s & 1) ? kw[j][s >> 1].z : kw[j][s >> 1].x, k1 = (s & 1) ? kw[j][s >> 1].w : kw[j][s >> 1].y;
                    float part[4] = {};
                    X::mma(part, {0u, a[2], 0u, b[2]}, k0, k1);
                    X::mma(part, {a[0], a[1], b[0], b[1]}, k0, k1);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (s & 1) c[j][i] += even[j][i] + part[i];
                        else even[j][i] = part[i];
                    }
                }
            }
            float sc[2][2], top = NEG;  // row g, positions w0 + 8 j + 2 t + {0, 1}, ahead of the factor `dn`
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const bool live = seen && at + 8 * j + 2 * t + i < end;
                    sc[j][i] = live ? c[j][i] + c[j][i + 2] : NEG;
                    top = fmaxf(top, sc[j][i]);
                }
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
            const float mnew = top > NEG ? fmaxf(m, top * dn) : m, corr = expf(m - mnew);
            more = turn(++i);
            if (more) fetch_k();  // (the products with the last ones are done)
            __syncwarp();
            lsum *= corr;
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const bool live = seen && at + 8 * j + 2 * t + i < end;
                    const float e = live ? expf(fmaf(sc[j][i], dn, -mnew)) : 0.0f;
                    lsum += e;
                    probs[(8 * j + 2 * t + i) * SA_ROWS + g] = e;
                }
            m = mnew;
            __syncwarp();
            // the rows these positions belong to: all of the block's, or one sample's.  A probability of zero does not keep another
            // sample's rows clean: an fp16 cache stores what overflows as infinity, and 0 * inf is NaN
            const uint32_t mine = own ? ((1u << nh) - 1u) << (zt * nh) : (1u << SA_ROWS) - 1u;
            if (i > 1) {
#pragma unroll
                for (int r = 0; r < SA_ROWS; ++r) {
                    const float cr = __shfl_sync(0xffffffffu, corr, 4 * r);
#pragma unroll
                    for (int i = 0; i < 8; ++i) acc[r][i] *= cr;
                }
            }
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                const float* pr = probs + (vside + SIDES * k) * SA_ROWS;
                const float4 lo = *reinterpret_cast<const float4*>(pr), hi = *reinterpret_cast<const float4*>(pr + 4);
                const float e[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
                float x[8];
                Elem<KT>::unpack(vw[k], x);
#pragma unroll
                for (int r = 0; r < SA_ROWS; ++r) {
                    if (mine >> r & 1u) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) acc[r][i] = fmaf(e[r], x[i], acc[r][i]);
                    }
                }
            }
            if (more) fetch_v();
        }
    }
    // ---- the warps' sums, relative to the CTA's maximum
    lsum += __shfl_xor_sync(0xffffffffu, lsum, 1);
    lsum += __shfl_xor_sync(0xffffffffu, lsum, 2);
    if (t == 0) { ms[warp][g] = m; ls[warp][g] = lsum; }
#pragma unroll
    for (int r = 0; r < SA_ROWS; ++r) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
#pragma unroll
            for (int o = 16; o >= CH; o >>= 1) acc[r][i] += __shfl_xor_sync(0xffffffffu, acc[r][i], o);
        }
        if (vside == 0) {
            *reinterpret_cast<float4*>(&accs[warp][r * HD + vch * 8]) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
            *reinterpret_cast<float4*>(&accs[warp][r * HD + vch * 8 + 4]) = make_float4(acc[r][4], acc[r][5], acc[r][6], acc[r][7]);
        }
    }
    __syncthreads();
    const int r = tid >> 4, c = tid & 15;  // sixteen threads a row, float4 c, c + 16, ...
    if (r < rows) {
        const size_t at = row_at(r) * p.max_slices + slice;
        float M = fmaxf(fmaxf(ms[0][r], ms[1][r]), fmaxf(ms[2][r], ms[3][r])), L = 0.0f, w[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            w[k] = ls[k][r] > 0.0f ? expf(ms[k][r] - M) : 0.0f;
            if (w[k] > 0.0f) L += ls[k][r] * w[k];
        }
#pragma unroll
        for (int i = 0; i < HD / 64; ++i) {
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float4 a = *reinterpret_cast<const float4*>(&accs[k][r * HD + 4 * (c + 16 * i)]);
                if (w[k] > 0.0f) { o.x = fmaf(a.x, w[k], o.x); o.y = fmaf(a.y, w[k], o.y); o.z = fmaf(a.z, w[k], o.z); o.w = fmaf(a.w, w[k], o.w); }
            }
            *reinterpret_cast<float4*>(p.part_acc + at * HD + 4 * (c + 16 * i)) = o;
        }
        if (c == 0) *reinterpret_cast<float2*>(p.part_ml + at * 2) = make_float2(M, L);
    }
    // ---- the last CTA of this block merges the slices
    unsigned int* counter = p.counters + (size_t)blockIdx.z * p.kv_heads + kvh;
    __threadfence();
    __syncthreads();
    if (tid == 0) is_last = atomicAdd(counter, 1u) == gridDim.y - 1u;
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    if (tid == 0) *counter = 0u;  // for the next layer or step
    if (r >= rows) return;
    const size_t row = row_at(r) * p.max_slices;
    const int n = p.split.shared + p.split.own;
    float M = NEG, L = 0.0f;
    float4 o[HD / 64];
#pragma unroll
    for (int i = 0; i < HD / 64; ++i) o[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    constexpr int B = 6;  // slices in flight
    for (int s0 = 0; s0 < n; s0 += B) {
        float2 ml[B];
        float4 a[B][HD / 64];
#pragma unroll
        for (int k = 0; k < B; ++k) {
            const size_t at = row + min(s0 + k, n - 1);
            ml[k] = __ldcg(reinterpret_cast<const float2*>(p.part_ml) + at);
#pragma unroll
            for (int i = 0; i < HD / 64; ++i) a[k][i] = __ldcg(reinterpret_cast<const float4*>(p.part_acc + at * HD) + c + 16 * i);
        }
#pragma unroll
        for (int k = 0; k < B; ++k) {
            if (s0 + k < n && ml[k].y > 0.0f) {
                const float Mn = fmaxf(M, ml[k].x), corr = expf(M - Mn), w = expf(ml[k].x - Mn);
                L = L * corr + ml[k].y * w;
#pragma unroll
                for (int i = 0; i < HD / 64; ++i) {
                    o[i].x = o[i].x * corr + a[k][i].x * w; o[i].y = o[i].y * corr + a[k][i].y * w;
                    o[i].z = o[i].z * corr + a[k][i].z * w; o[i].w = o[i].w * corr + a[k][i].w * w;
                }
                M = Mn;
            }
        }
    }
    const float inv = L > 0.0f ? 1.0f / L : 0.0f;
    const size_t at = row_at(r) * HD;
#pragma unroll
    for (int i = 0; i < HD / 64; ++i) {
        const float v[4] = {o[i].x * inv, o[i].y * inv, o[i].z * inv, o[i].w * inv};
        uint2 hi, lo;
        T16* h = reinterpret_cast<T16*>(&hi);
        T16* l = reinterpret_cast<T16*>(&lo);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            h[k] = Elem<T16>::from_f32(v[k]);
            l[k] = Elem<T16>::from_f32(v[k] - Elem<T16>::to_f32(h[k]));
        }
        *reinterpret_cast<uint2*>(out + at + 4 * (c + 16 * i)) = hi;
        if (out_lo != nullptr) *reinterpret_cast<uint2*>(out_lo + at + 4 * (c + 16 * i)) = lo;
    }
}

}  // namespace cd
