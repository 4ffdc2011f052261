// Long passes of the hybrid model: prompt portions of many positions at once (hybrid_prefill.cu).
#pragma once
#include "exec.cuh"
#include "packed_gemm.cuh"

namespace ctox {

// Buffers of long passes, allocated at warm-up and given back when another allocation of the context fails.
struct LongPass {
    uint32_t cap = 0;  // positions
    bool busy = false;  // a call that takes long passes is on its way
    cudaEvent_t layer_done[2] = {nullptr, nullptr};
    std::vector<std::pair<void *, size_t>> owned;
    LongIn in{};
    float *y = nullptr;  // outputs of a projection (partial sums)
    size_t y_floats = 0;
    float *h = nullptr, *final_hidden = nullptr;         // [cap][hidden]
    float *qkv = nullptr, *core = nullptr;               // [cap][channels], [cap][value width]
    float *g = nullptr, *beta = nullptr;                 // [cap][value heads]
    float *coefs = nullptr;                              // [groups of four][value heads][factors of the scan]
    float *aq = nullptr, *attn = nullptr;                // [cap][query width], [cap][query heads][head_dim + 2] (all splits)
    uint32_t *tokens = nullptr;
};

// Fewest remaining tokens worth a long pass. Its products unpack every weight for a tile of positions whatever it holds: at
// position 0, 17 tokens take 2.20 ms against 2.35 in three short passes (8 layers of width 5120), 0.37 against 0.67 (4
// layers of width 1024); 16 took 2.40 against 2.15 in two short passes of the wide model. On a long session attention
// decides. The tensor-core kernel needs one group of positions for 32 queries: 17 tokens on 32000, 24 heads of 256, 2.54
// against 5.19 ms. On CUDA cores a group's time follows its queries and the last group is as long as the others: 20
// tokens on 8192, 1.80 against 1.72 ms (32-bit cache, 4 layers), 1.29 against 1.30 on 2048; 25 on 32000, 4.60 against
// 4.55; 33, 5.60 against 5.87.
constexpr uint32_t kLongMin = 17, kLongMinDeepCores = 26;
constexpr uint64_t kDeepCores = 2048;  // position from which the second one holds
uint32_t long_min(const ctox_exec *e);

// Allocates the buffers; leaves e->long_pass null (short passes only) where they do not fit or do not apply.
ctox_status long_warmup(ctox_exec *e);
void long_release(ctox_exec *e);
// Consumes m tokens (long_min .. cap) at the session's position: target layers, committed state, the MTP cache of
// all but the last (m - 1) % 8 + 1 pairs, which like those of a short pass are left to the next call. With `cancel` the
// host stays two layers ahead of the device and reads the word before each one: a layer of the flagship takes 2.3 ms for
// 1024 tokens, a short pass of all 64 layers 10 ms. A pass that was cancelled leaves no usable session.
ctox_status long_target_pass(ctox_exec *e, const uint32_t *tokens, uint32_t m, const volatile int32_t *cancel);

// One CTA row of the attention kernels per group of `per_group` positions (layers.cu), over `splits` parts of the context;
// workspace: m * splits rows [query heads][head_dim + 2], those of a group side by side.
bool attention_on_tensor_cores(const AttnGeom &g, int kv_bf16);
uint32_t attention_group_positions(const AttnGeom &g, int kv_bf16, uint32_t m);
void launch_attention_groups(cudaStream_t st, const AttnGeom &g, const float *q, const void *k_cache, const void *v_cache,
                             int kv_bf16, const uint32_t *page_table, uint32_t page_tokens, uint64_t cache_slot, uint32_t m,
                             uint32_t splits, float *workspace);

}  // namespace ctox
