// Host side of the tensor-core GEMMs of prefill.cuh, shared by the families' prompt passes: tensor maps and launches.
#pragma once
#include "pf_attn.cuh"
#include "prefill.cuh"

#include <algorithm>
#include <type_traits>

#include "model.h"

namespace cd {
namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_tiled_fn() {  // nullptr: this driver does not have it
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess || qres != cudaDriverEntryPointSuccess) return nullptr;
    return (EncodeTiledFn)fn;
}

inline size_t round_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

bool encode_2d(EncodeTiledFn encode, CUtensorMap* map, CUtensorMapDataType dt, const void* base, uint64_t inner, uint64_t rows,
               uint64_t row_bytes, uint32_t box_rows) {
    const cuuint64_t dims[2] = {inner, rows};
    const cuuint64_t strides[1] = {row_bytes};
    const cuuint32_t box[2] = {(cuuint32_t)PF_BK, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return encode(map, dt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// instruction descriptor of tcgen05.mma kind::f16: fp32 accumulate, both operands K-major
inline uint32_t make_idesc(int bn, bool bf16, int bm = PF_BM) {
    const uint32_t fmt = bf16 ? 1u : 0u;
    return (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(bm >> 4) << 24);
}

struct PfPlan { int cg, bn; };

// How a product is cut: the tile (one CTA or a pair, 32-256 columns) with the least modelled time, in clocks.  Measured per
// step of 64 along K (hi + lo / plain): 624 / 446 at 32 columns, where the chain of dependent MMAs is what counts, 752 / 494 at
// 128, 1104 / 558 at 256; a step's bytes come at about 48 a clock; starting a pair costs 1 us more than starting a CTA.
// Over 27 shapes (16-4096 rows, 96-22016 columns, K 72-11008; every tile timed, one and two parts of A) the choice takes 1.016 of the
// best one's time in the mean and 1.15 at most, 1.22 among launches below 15 us.
inline PfPlan pf_plan(int M, int N, int K, bool split, int sms, bool grouped) {
    const int nkb = (K + PF_BK - 1) / PF_BK, halves = split ? 2 : 1;
    PfPlan best{1, PF_MAX_BN};
    double best_t = 1e30;
    for (int cg = 1; cg <= (grouped || M <= PF_BM ? 1 : 2); ++cg)
        for (int bn = PF_MAX_BN; bn >= 32; bn -= 32) {
            const long tiles = (long)((M + cg * PF_BM - 1) / (cg * PF_BM)) * ((N + bn - 1) / bn);
            const int units = sms / cg;
            const double rounds = (double)((tiles + units - 1) / units);
            const double mma = split ? std::max(624.0, 400.0 + 2.75 * bn) : 430.0 + 0.5 * bn;
            const double load = (halves * (double)PF_A_BYTES * std::min(M, PF_BM) / PF_BM + bn / cg * PF_BK * 2.0) / 48.0;
            const double t = rounds * nkb * std::max(mma, load) + 12.0 * bn + (cg == 2 ? 2000.0 : 0.0);
            if (t < best_t) { best_t = t; best = PfPlan{cg, bn}; }
        }
    return best;
}

template <int CG, bool SPLIT, class Epi>
cudaError_t pf_launch_t(cd_model* m, const CUtensorMap (&a)[2], const CUtensorMap& b, const PfGemm& p, bool bf16, const Epi& epi) {
    auto kern = pf_gemm_kernel<CG, SPLIT, Epi>;
    static bool attr_set = false;  // per instantiation
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PF_SMEM);
        if (e != cudaSuccess) return e;
        attr_set = true;
    }
    const int tiles = ((p.M + CG * PF_BM - 1) / (CG * PF_BM)) * ((p.N + p.bn - 1) / p.bn);
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(CG * std::min(tiles, m->sm_count / CG));
    lc.blockDim = dim3(PF_THREADS);
    lc.dynamicSmemBytes = PF_SMEM;
    lc.stream = m->stream;
    cudaLaunchAttribute at[2];
    if (CG == 2) {
        at[lc.numAttrs].id = cudaLaunchAttributeClusterDimension;
        at[lc.numAttrs].val.clusterDim.x = CG; at[lc.numAttrs].val.clusterDim.y = 1; at[lc.numAttrs].val.clusterDim.z = 1;
        lc.numAttrs++;
    }
    if (m->pdl) {  // barriers and tensor memory are set up before the previous kernel ends
        at[lc.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[lc.numAttrs].val.programmaticStreamSerializationAllowed = 1;
        lc.numAttrs++;
    }
    lc.attrs = at;
    m->launches++;
    return cudaLaunchKernelEx(&lc, kern, a[0], SPLIT ? a[1] : a[0], b, p, make_idesc(p.bn, bf16, CG * PF_BM), epi);
}

// C[p.M][p.N] = A[p.M][p.K] (hi, and lo unless that is nullptr) * B[b_rows][p.K]^T through `epi`.  Rows of A behind p.M are
// neither read nor stored.
template <class Epi>
cudaError_t pf_launch(cd_model* m, EncodeTiledFn encode, const void* hi, const void* lo, const void* B, size_t b_rows, PfGemm p, bool bf16, const Epi& epi) {
    if (p.M <= 0 || p.N <= 0) return cudaSuccess;
    const CUtensorMapDataType dt = bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    const PfPlan plan = pf_plan(p.M, p.N, p.K, lo != nullptr, m->sm_count, p.tile_group != nullptr);
    p.bn = plan.bn;
    CUtensorMap a[2], b;
    const uint64_t row = (uint64_t)p.K * 2;
    if (!encode_2d(encode, &a[0], dt, hi, p.K, p.M, row, PF_BM) || (lo != nullptr && !encode_2d(encode, &a[1], dt, lo, p.K, p.M, row, PF_BM)) ||
        !encode_2d(encode, &b, dt, B, p.K, b_rows, row, plan.bn / plan.cg))
        return cudaErrorInvalidValue;
    if (plan.cg == 2) return lo ? pf_launch_t<2, true>(m, a, b, p, bf16, epi) : pf_launch_t<2, false>(m, a, b, p, bf16, epi);
    return lo ? pf_launch_t<1, true>(m, a, b, p, bf16, epi) : pf_launch_t<1, false>(m, a, b, p, bf16, epi);
}

// cached rows {d, token in page, head, page} in boxes of 64 columns and 128 tokens of one head
inline bool encode_rows_4d(EncodeTiledFn encode, CUtensorMap* map, CUtensorMapDataType dt, const void* base, uint64_t d, int page_tokens, int heads, uint64_t pages,
                           uint64_t row_bytes, uint64_t head_bytes, uint64_t page_bytes) {
    const cuuint64_t dims[4] = {d, (cuuint64_t)page_tokens, (cuuint64_t)heads, pages};
    const cuuint64_t strides[3] = {row_bytes, head_bytes, page_bytes};
    const cuuint32_t box[4] = {64, (cuuint32_t)std::min(page_tokens, PA_KEYS), 1, (cuuint32_t)std::max(1, PA_KEYS / page_tokens)};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    return encode(map, dt, 4, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// q: the queries' hi and lo maps; nz = heads * maps
template <typename KT, int KD, int VD, bool BIAS, class Epi>
cudaError_t pa_launch(cd_model* m, const CUtensorMap (&q)[2], bool split, const CUtensorMap& k, const CUtensorMap& v, const PfAttn& p, int nz, const Epi& epi) {
    auto kern = pf_attn_kernel<KT, KD, VD, BIAS, Epi>;
    constexpr size_t smem = PaSmem<KD, VD>::BYTES;
    static bool attr_set = false;  // per instantiation
    if (!attr_set) {
        cudaFuncAttributes fa;
        cudaError_t e = cudaFuncGetAttributes(&fa, kern);
        if (e == cudaSuccess && fa.numRegs * PA_THREADS < PA_REGS) e = cudaErrorInvalidConfiguration;  // the warpgroups' split would wait for registers that the block does not have
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        attr_set = true;
    }
    const bool bf16 = std::is_same<KT, __nv_bfloat16>::value;
    kern<<<dim3((p.rows + PA_ROWS - 1) / PA_ROWS, nz), PA_THREADS, smem, m->stream>>>(q[0], split ? q[1] : q[0], k, v, p, make_idesc(PA_KEYS, bf16),
                                                                                 make_idesc(VD, bf16) | (1u << 16) /* V is MN-major */, epi);
    m->launches++;
    return cudaGetLastError();
}

}  // namespace
}  // namespace cd
