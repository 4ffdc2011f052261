// Device code shared by the kernels with dense bf16 weights (dense.cu, dense_stream.cu).
#pragma once
#include "dense.cuh"

namespace ctox {

// Columns c .. c + 3 of p, zero from `end` on.
__device__ __forceinline__ float4 load4(const float *p, uint32_t c, uint32_t end, bool vec) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c + 4 <= end && vec) return *reinterpret_cast<const float4 *>(p + c);
    if (c < end) v.x = p[c];
    if (c + 1 < end) v.y = p[c + 1];
    if (c + 2 < end) v.z = p[c + 2];
    if (c + 3 < end) v.w = p[c + 3];
    return v;
}
__device__ __forceinline__ void store4(float *p, uint32_t c, uint32_t end, const float4 &v) {
    if (c + 4 <= end && ((uintptr_t)p & 15) == 0) {
        *reinterpret_cast<float4 *>(p + c) = v;
        return;
    }
    if (c < end) p[c] = v.x;
    if (c + 1 < end) p[c + 1] = v.y;
    if (c + 2 < end) p[c + 2] = v.z;
    if (c + 3 < end) p[c + 3] = v.w;
}
__device__ __forceinline__ void latent_append_row(const LatentAppend &a, uint32_t m, uint32_t tid, uint32_t nthreads, float *red) {
    const float *row = a.fan + (size_t)m * a.fan_stride + a.fan_off;
    float sq = 0.f;
    for (uint32_t c = tid; c < a.kv_rank; c += nthreads) sq += row[c] * row[c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    __syncthreads();
    if ((tid & 31) == 0) red[tid >> 5] = sq;
    __syncthreads();
    float total = 0.f;
    for (uint32_t w = 0; w < nthreads / 32; ++w) total += red[w];
    const float inv = 1.0f / sqrtf(total / (float)a.kv_rank + a.eps);
    const uint32_t pos = a.pos0 + m;
    const size_t base = paged_slot(a.page_table, a.page_tokens, pos) * (a.kv_pad + a.rot_pad);
    auto store = [&](uint32_t c, float v) {
        if (a.bf16)
            ((__nv_bfloat16 *)a.cache)[base + c] = __float2bfloat16_rn(v);
        else
            ((float *)a.cache)[base + c] = v;
    };
    for (uint32_t c = tid; c < a.kv_pad; c += nthreads) store(c, c < a.kv_rank ? row[c] * inv * a.norm_w[c] : 0.f);
    for (uint32_t i = tid; i < a.rot_pad / 2; i += nthreads) {
        float u = 0.f, v = 0.f;
        if (2 * i < a.rot_dim) {
            u = row[a.kv_rank + 2 * i];
            v = row[a.kv_rank + 2 * i + 1];
            rope_pair(u, v, (float)pos * a.freq[i]);
        }
        store(a.kv_pad + 2 * i, u);
        store(a.kv_pad + 2 * i + 1, v);
    }
}

// What the output of row `row` of a group (first row row0, `rows` rows) takes beside its sum: biases of the row and of row ^ 1, and
// the turn. Constants of a launch: a kernel may form them ahead of its dependency wait.
// KIND: an OutKind, or -1 for what the launch says.
struct RowConstants {
    float bias, pair_bias, sin, cos;
    bool turned;
};
template <int KIND = -1>
__device__ __forceinline__ RowConstants row_constants(const VecOut &out, uint32_t m, uint32_t row, uint32_t rows, uint32_t row0 = 0) {
    RowConstants k{0.f, 0.f, 0.f, 1.f, false};
    if (row >= rows) return k;
    if (out.bias) {
        k.bias = out.bias[(size_t)row0 + row];
        if ((row ^ 1u) < rows) k.pair_bias = out.bias[(size_t)row0 + (row ^ 1u)];
    }
    if (KIND < 0 ? out.kind == OUT_ROPE : KIND == OUT_ROPE) {
        const uint32_t w = row % out.head_width;
        k.turned = w >= out.rope0 && w < out.rope0 + out.rope_dims;
        if (k.turned) sincosf((float)(out.pos0 + m) * out.freq[(w - out.rope0) >> 1], &k.sin, &k.cos);
    }
    return k;
}
// One output of a matrix-vector product: row `row` of a group whose first row is row0, with the sum v; `pair` is the sum of
// row ^ 1 (read where that row exists).
template <int KIND = -1>
__device__ __forceinline__ void emit_row(const VecOut &out, uint32_t m, uint32_t row0, uint32_t row, float v, float pair,
                                         const RowConstants &k) {
    const int kind = KIND < 0 ? out.kind : KIND;
    v += k.bias;
    pair += k.pair_bias;
    if (kind == OUT_CLAMPED_GLU) {
        if (!(row & 1)) out.y[(size_t)m * out.y_stride + (row >> 1)] = clamped_glu(v, pair, out.cap, out.slope);
        return;
    }
    if (kind == OUT_RELU2) {
        v = v > 0.f ? v * v : 0.f;
    } else if (kind == OUT_SOFTCAP) {
        v = out.cap * tanhf(v / out.cap);
    } else if (kind == OUT_ROPE && k.turned) {
        float a = (row & 1) ? pair : v, b = (row & 1) ? v : pair;
        turn_pair(a, b, k.sin, k.cos);
        v = (row & 1) ? b : a;
    }
    out.y[(size_t)m * out.y_stride + (size_t)row0 + row] = v;
}

}  // namespace ctox
