// How the attention of a sampled step (sample_attn.cuh) is cut into CTAs.  Host code only but for SaBlocks' arithmetic.
#pragma once
#include <algorithm>

#if defined(__CUDACC__)
#define SA_BOTH __host__ __device__
#else
#define SA_BOTH
#endif

namespace cd {

constexpr int SA_ROWS = 8, SA_TILE = 64, SA_WARP_TILE = 16, SA_THREADS = 128, SA_PER_SM = 3;

// How `heads / kv_heads` q heads of `samples` samples make blocks of at most SA_ROWS pairs: several samples with all their heads
// of the group, or some heads of one sample.
struct SaBlocks {
    int gqa, samples;
    SA_BOTH int heads() const { return gqa < SA_ROWS ? gqa : SA_ROWS; }            // q heads of a sample in a block
    SA_BOTH int head_blocks() const { return (gqa + SA_ROWS - 1) / SA_ROWS; }
    SA_BOTH int per_block() const { return SA_ROWS / heads(); }                    // samples in a block (1 where the heads fill it)
    SA_BOTH int count() const { return head_blocks() * ((samples + per_block() - 1) / per_block()); }
};

// Slices of a step at this length: every CTA takes at most `rounds` turns of sixteen positions a warp (a slice of own positions:
// `spans` times sixteen positions of each sample), as few as the partials' buffers and one wave of CTAs allow.  (A second wave costs
// as much as the first: its positions are requested only when it starts.)  A captured step belongs to one cut: a new one comes every
// 16 tokens or more.  With own positions counted in 64s there are a quarter of them, which saves 0.7 to 1.5 ms of a loop's first 16
// steps, but their slices are more: 200 steps of eight samples of the 5B model behind 1024 positions 597 ms instead of 588, of
// sixteen samples of a 2048-wide one (heads of 64, 100 positions) 182 instead of 176.
struct SaSplit {
    int rounds, spans, shared, own;
    int id() const { return (rounds * 64 + shared) * 64 + own; }
};
inline SaSplit sa_split(int shared_tokens, int attn_len, const SaBlocks& blocks, int kv_heads, int max_slices, int sms) {
    auto up = [](int a, int b) { return (a + b - 1) / b; };
    const int ts = up(shared_tokens, SA_TILE), to = up(attn_len - shared_tokens, SA_WARP_TILE);
    const int most = std::min(max_slices, std::max(sms * SA_PER_SM / (kv_heads * blocks.count()), ts > 0 ? 2 : 1));
    for (int r = 1;; ++r) {
        const SaSplit s{r, std::max(1, 4 * r / std::min(blocks.per_block(), blocks.samples)), up(ts, r), 0};
        const int own = up(to, s.spans);
        if (s.shared + own <= most || r >= ts + to * SA_ROWS) return SaSplit{r, s.spans, s.shared, own};
    }
}

}  // namespace cd
