// One token through the persistent kernel.  WT: storage of the embedding and the LM head; LT: row format of the linears; KT:
// storage of the KV cache.  cudaErrorNotSupported: its buffers do not fit in shared memory (nothing was launched).
#pragma once
#include "mega.cuh"
#include "model.h"

namespace cd {
template <typename WT, typename LT, typename KT>
cudaError_t launch_mega(cd_model* m, int input_embed, int want_logits);
}  // namespace cd
