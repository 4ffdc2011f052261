// Long passes of the hybrid model: prompt portions of many positions at once (hybrid_prefill.cu).
#pragma once
#include "exec.cuh"
#include "packed_gemm.cuh"

namespace ctox {

// Buffers of long passes, allocated at warm-up.
struct LongPass {
    uint32_t cap = 0;  // positions
    LongIn in{};
    float *y = nullptr;  // outputs of a projection (partial sums)
    size_t y_floats = 0;
    float *h = nullptr, *final_hidden = nullptr;         // [cap][hidden]
    float *qkv = nullptr, *core = nullptr;               // [cap][channels], [cap][value width]
    float *g = nullptr, *beta = nullptr;                 // [cap][value heads]
    float *aq = nullptr, *attn = nullptr;                // [cap][query width], [cap][query heads][head_dim + 2]
    uint32_t *tokens = nullptr;
};

// Fewest remaining tokens worth a long pass. Its products unpack every weight for a tile of positions whatever it holds: 17
// tokens take 2.41 ms against 2.90 in three short passes (8 layers of width 5120), 0.49 against 0.98 (4 layers of
// width 1024); 16 take 2.40 against 2.15 in two short passes of the wide model.
constexpr uint32_t kLongMin = 17;

// Allocates the buffers; leaves e->long_pass null (short passes only) where they do not fit or do not apply.
ctox_status long_warmup(ctox_exec *e);
// Consumes m tokens (kLongMin .. cap) at the session's position: target layers, committed state, the MTP cache of
// all but the last (m - 1) % 8 + 1 pairs, which like those of a short pass are left to the next call.
ctox_status long_target_pass(ctox_exec *e, const uint32_t *tokens, uint32_t m);

// One CTA row of the attention kernels per group of `per_group` positions (layers.cu); no split of the context.
uint32_t attention_group_positions(const AttnGeom &g, int kv_bf16);
void launch_attention_groups(cudaStream_t st, const AttnGeom &g, const float *q, const void *k_cache, const void *v_cache,
                             int kv_bf16, const uint32_t *page_table, uint32_t page_tokens, uint64_t cache_slot, uint32_t m,
                             float *workspace);

}  // namespace ctox
