// One token through the persistent kernel.  WT: storage of the embedding and the LM head; LT: row format of the linears; KT:
// storage of the KV cache.  cudaErrorNotSupported: its buffers do not fit in shared memory (nothing was launched).
#pragma once
#include <algorithm>

#include "mega.cuh"
#include "model.h"

namespace cd {
// Rows of a ring stage by the chunks a thread takes of a row; a stage's bytes (row_*: bytes of a row of max(dim, q_dim), hidden
// and of the head); cached positions of an attention tile: the largest power of two that stays inside a page and fits a stage.
enum MegaRows { MEGA_PLAIN = 0, MEGA_FP8 = 1, MEGA_INT4 = 2 };
constexpr int mega_stage_rows(int chunks, MegaRows f) { return f == MEGA_INT4 ? (chunks == 1 ? 8 : chunks < 4 ? 4 : 2) : chunks == 1 ? 4 : chunks == 2 || f == MEGA_FP8 ? 2 : 1; }
constexpr int mega_head_rows(int nd, MegaRows f) { return f != MEGA_PLAIN ? (nd == 1 ? 2 : 1) : mega_stage_rows(nd, f); }  // (a quantised chunk is twice as many elements)
inline size_t mega_stage_bytes(int nd, int nh, MegaRows f, size_t row_d, size_t row_h, size_t row_o) {
    return (std::max({mega_stage_rows(nd, f) * row_d, mega_stage_rows(nh, f) * row_h, mega_head_rows(nd, f) * row_o}) + 127) / 128 * 128;
}
inline int mega_tile_tokens(int page_tokens, size_t row_bytes, size_t stage_bytes) {
    int tile = 64;
    while (tile > 1 && (tile > page_tokens || page_tokens % tile || tile * row_bytes > stage_bytes)) tile >>= 1;
    return tile;
}

template <typename WT, typename LT, typename KT>
cudaError_t launch_mega(cd_model* m, int input_embed, int want_logits);
}  // namespace cd
