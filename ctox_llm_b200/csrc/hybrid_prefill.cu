// Long passes of the hybrid model. A prompt portion of up to LongPass::cap positions goes through a layer at once:
// the packed products on tcgen05 (packed_gemm.cu), between them the kernels below, one CTA per position for what
// works on rows, a token scan for the recurrence. Arithmetic and order of operations are those of the short passes
// (decoder.rs:636-938, 1009-1046); sums of many terms are taken in another order.
//
// Short passes read every weight once per eight positions and are bound by unpacking it; measured on 8 layers of the
// flagship's width, 999 tokens: 163 ms in 125 short passes.
#include "hybrid_prefill.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "f32x2.cuh"
#include "prep.cuh"

namespace ctox {

__device__ __forceinline__ float lp_out(const LongOut &o, uint32_t row, uint32_t pos) {
    const float *p = o.y + (size_t)pos * o.rows + row;
    float v = p[0];
    for (uint32_t s = 1; s < o.splits; ++s) v += p[s * o.split_stride];  // index order
    return v;
}
// Four rows row .. row + 3 (a multiple of four, o.rows too).
__device__ __forceinline__ float4 lp_out4(const LongOut &o, uint32_t row, uint32_t pos) {
    const float *p = o.y + (size_t)pos * o.rows + row;
    float4 v = *reinterpret_cast<const float4 *>(p);
    for (uint32_t s = 1; s < o.splits; ++s) {
        const float4 w = *reinterpret_cast<const float4 *>(p + s * o.split_stride);
        v.x += w.x;
        v.y += w.y;
        v.z += w.z;
        v.w += w.w;
    }
    return v;
}
template <int OP>  // 0 sum, 1 maximum
__device__ __forceinline__ float lp_block(float v, float *red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float t = __shfl_xor_sync(0xffffffffu, v, o);
        v = OP ? fmaxf(v, t) : v + t;
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = red[0];
    for (uint32_t w = 1; w < blockDim.x / 32; ++w) v = OP ? fmaxf(v, red[w]) : v + red[w];
    return v;
}

// Row of the attention kernels' workspace that holds a query's part of one split: per group of positions
// [kv head][split][position][head of the kv head].
__device__ __forceinline__ size_t attn_row(uint32_t pos, uint32_t head, uint32_t split, uint32_t m, uint32_t per_group,
                                           uint32_t splits, uint32_t q_heads, uint32_t kv_heads) {
    const uint32_t G = q_heads / kv_heads, group = pos / per_group, n = min(per_group, m - group * per_group);
    return (size_t)group * per_group * splits * q_heads +
           ((size_t)(head / G) * splits + split) * G * n + pos % per_group * G + head % G;
}

// ------------------------------------------------------------------ rows: one CTA per position
// Forms the next product's input row and writes it as hi and lo parts. Bound by memory: a projection's fp32 outputs are read
// once, four bytes per input column are written.
enum : int { ROWS_NORM, ROWS_SWIGLU, ROWS_ATTENTION, ROWS_DELTA, ROWS_MTP };
// More threads have more of a long row's loads in flight, fewer leave room for more rows per SM. 999 positions at a width of 5120, 512
// and 256 threads: SWIGLU 53 and 59 us, NORM 36 and 30, DELTA 27 and 21, ATTENTION 31 and 23.
__host__ __device__ constexpr int rows_threads(int mode) { return mode == ROWS_SWIGLU ? 512 : 256; }

struct RowsArgs {
    LongOut o;              // NORM: addend (o.y null: none); SWIGLU: [gate | up]; ATTENTION, DELTA: where the gates are
    const float *a, *b;     // NORM: a = input row when `h` starts there (else h); MTP: embedding and hidden rows
    const float *w, *w2;    // norm weights
    float *h, *xn_out;      // NORM: residual row (written), normalised row (optional)
    float eps;
    uint32_t width;         // columns of h / inter / query width / value width / hidden
    uint32_t off;           // DELTA: first gate row of o
    uint32_t q_heads, kv_heads, head_dim, per_group, splits, m;  // ATTENTION
    LongIn in;
    const float *s_in;      // of the next product (null: 1)
    uint32_t blocks_padded;
    int dt, has_next;
};

template <int MODE>
__global__ void __launch_bounds__(rows_threads(MODE)) k_long_rows(const RowsArgs p) {
    constexpr uint32_t kRowsThreads = rows_threads(MODE);
    pdl_launch();
    pdl_wait();
    extern __shared__ __align__(16) float vals[];  // two float4 of each unit, then the largest value of each block
    __shared__ float red[kRowsThreads / 32];
    const uint32_t pos = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    const uint32_t columns = MODE == ROWS_MTP ? 2 * p.width : p.width, units = p.has_next ? p.blocks_padded * 8 : p.width / 8;
    // A unit is what one 16-byte chunk of a part holds (inv_perm): columns c .. c + 3 and, 4 (4-bit codes) or 8 further, four more. Its
    // thread keeps it throughout: in two places of its own in shared memory, one after the other over the lanes. Eight lanes
    // hold a block; all lanes of a warp have a unit or none has (blocks_padded is a multiple of four).
    const uint32_t step = p.dt ? 4 : 8;
    auto column = [&](uint32_t unit) { return (unit >> 1) * 16 + (unit & 1) * (12 - step); };
    float4 *first = reinterpret_cast<float4 *>(vals), *second = first + units;
    float *block_max = vals + units * 8;
    auto at4 = [](const float *q) { return *reinterpret_cast<const float4 *>(q); };
    float amax = 0.f;
    auto put = [&](uint32_t unit, uint32_t c, float4 a, float4 b) {
        if (p.s_in && c < columns) {
            const float4 x = at4(p.s_in + c), y = at4(p.s_in + c + step);
            a = make_float4(a.x * x.x, a.y * x.y, a.z * x.z, a.w * x.w);
            b = make_float4(b.x * y.x, b.y * y.y, b.z * y.z, b.w * y.w);
        }
        first[unit] = a;
        second[unit] = b;
        float mx = fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(a.w))),
                         fmaxf(fmaxf(fabsf(b.x), fabsf(b.y)), fmaxf(fabsf(b.z), fabsf(b.w))));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
        if ((lane & 7) == 0) block_max[unit >> 3] = mx;
        amax = fmaxf(amax, mx);
    };
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    auto sq4 = [](float4 v) { return (v.x * v.x + v.y * v.y) + (v.z * v.z + v.w * v.w); };
    if constexpr (MODE == ROWS_NORM) {
        float *h = p.h + (size_t)pos * p.width;
        const float *base = p.a ? p.a + (size_t)pos * p.width : nullptr;
        float sq = 0.f;
        for (uint32_t unit = tid; unit < units; unit += kRowsThreads) {
            const uint32_t c = column(unit);
            float4 v[2] = {zero, zero};
            if (c < p.width)
#pragma unroll
                for (uint32_t i = 0; i < 2; ++i) {
                    if (base) v[i] = at4(base + c + i * step);
                    if (p.o.y) {
                        const float4 y = lp_out4(p.o, c + i * step, pos);
                        v[i] = make_float4(v[i].x + y.x, v[i].y + y.y, v[i].z + y.z, v[i].w + y.w);
                    }
                    *reinterpret_cast<float4 *>(h + c + i * step) = v[i];
                }
            first[unit] = v[0];
            second[unit] = v[1];
            sq += sq4(v[0]) + sq4(v[1]);
        }
        const float inv = 1.0f / sqrtf(lp_block<0>(sq, red) / (float)p.width + p.eps);
        for (uint32_t unit = tid; unit < units; unit += kRowsThreads) {  // each thread its own units again
            const uint32_t c = column(unit);
            float4 v[2] = {first[unit], second[unit]};
            if (c < p.width)
#pragma unroll
                for (uint32_t i = 0; i < 2; ++i) {
                    const float4 w = at4(p.w + c + i * step);
                    v[i] = make_float4(v[i].x * inv * (1.0f + w.x), v[i].y * inv * (1.0f + w.y), v[i].z * inv * (1.0f + w.z),
                                       v[i].w * inv * (1.0f + w.w));
                    if (p.xn_out) *reinterpret_cast<float4 *>(p.xn_out + (size_t)pos * p.width + c + i * step) = v[i];
                }
            if (p.has_next) put(unit, c, v[0], v[1]);
        }
        if (!p.has_next) return;
    } else if constexpr (MODE == ROWS_MTP) {
        const float *e = p.a + (size_t)pos * p.width, *h = p.b + (size_t)pos * p.width;
        float se = 0.f, sh = 0.f;
        for (uint32_t c = tid * 4; c < p.width; c += kRowsThreads * 4) {
            se += sq4(at4(e + c));
            sh += sq4(at4(h + c));
        }
        const float ie = 1.0f / sqrtf(lp_block<0>(se, red) / (float)p.width + p.eps);
        const float ih = 1.0f / sqrtf(lp_block<0>(sh, red) / (float)p.width + p.eps);
        for (uint32_t unit = tid; unit < units; unit += kRowsThreads) {
            const uint32_t c = column(unit);
            const bool hidden = c >= p.width;
            const uint32_t cc = hidden ? c - p.width : c;
            const float inv = hidden ? ih : ie;
            float4 v[2] = {zero, zero};
            if (c < columns)
#pragma unroll
                for (uint32_t i = 0; i < 2; ++i) {
                    const float4 x = at4((hidden ? h : e) + cc + i * step), w = at4((hidden ? p.w2 : p.w) + cc + i * step);
                    v[i] = make_float4(x.x * inv * (1.0f + w.x), x.y * inv * (1.0f + w.y), x.z * inv * (1.0f + w.z),
                                       x.w * inv * (1.0f + w.w));
                }
            put(unit, c, v[0], v[1]);
        }
    } else if constexpr (MODE == ROWS_SWIGLU) {
        for (uint32_t unit = tid; unit < units; unit += kRowsThreads) {
            const uint32_t c = column(unit);
            float4 v[2] = {zero, zero};
            if (c < p.width) {
                const float4 g[2] = {lp_out4(p.o, c, pos), lp_out4(p.o, c + step, pos)};
                const float4 u[2] = {lp_out4(p.o, p.width + c, pos), lp_out4(p.o, p.width + c + step, pos)};
#pragma unroll
                for (uint32_t i = 0; i < 2; ++i)
                    v[i] = make_float4(silu_f(g[i].x) * u[i].x, silu_f(g[i].y) * u[i].y, silu_f(g[i].z) * u[i].z, silu_f(g[i].w) * u[i].w);
            }
            put(unit, c, v[0], v[1]);
        }
    } else if constexpr (MODE == ROWS_ATTENTION) {
        // attention left (unnormalised output, maximum, sum) of each query; of several splits the first holds the merged one
        const uint32_t hd = p.head_dim;
        for (uint32_t unit = tid; unit < units; unit += kRowsThreads) {
            const uint32_t c = column(unit);
            float4 v[2] = {zero, zero};
            if (c < p.width) {
                const uint32_t hq = c / hd, d = c % hd;
                const float *r = p.a + attn_row(pos, hq, 0, p.m, p.per_group, p.splits, p.q_heads, p.kv_heads) * (hd + 2);
                const float inv = 1.0f / r[hd + 1];
#pragma unroll
                for (uint32_t i = 0; i < 2; ++i) {  // rows of hd + 2 floats are aligned for two of them
                    const float2 x = *reinterpret_cast<const float2 *>(r + d + i * step), y = *reinterpret_cast<const float2 *>(r + d + i * step + 2);
                    const float4 g = lp_out4(p.o, hq * 2 * hd + hd + d + i * step, pos);
                    v[i] = make_float4(x.x * inv * (1.0f / (1.0f + expf(-g.x))), x.y * inv * (1.0f / (1.0f + expf(-g.y))),
                                       y.x * inv * (1.0f / (1.0f + expf(-g.z))), y.y * inv * (1.0f / (1.0f + expf(-g.w))));
                }
            }
            put(unit, c, v[0], v[1]);
        }
    } else {
        // rms_norm_gated per value head (reference.rs:66-93): sixteen lanes per head
        for (uint32_t unit = tid; unit < units; unit += kRowsThreads) {
            const uint32_t c = column(unit);
            float4 v[2] = {zero, zero}, g[2] = {zero, zero};
            if (c < p.width)
#pragma unroll
                for (uint32_t i = 0; i < 2; ++i) {
                    v[i] = at4(p.a + (size_t)pos * p.width + c + i * step);
                    g[i] = lp_out4(p.o, p.off + c + i * step, pos);
                }
            float sq = sq4(v[0]) + sq4(v[1]);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
            const float inv = 1.0f / sqrtf(sq / 128.0f + p.eps);
            if (c < p.width)
#pragma unroll
                for (uint32_t i = 0; i < 2; ++i) {
                    const float4 w = at4(p.w + c % 128 + i * step);
                    v[i] = make_float4(v[i].x * inv * w.x * silu_f(g[i].x), v[i].y * inv * w.y * silu_f(g[i].y),
                                       v[i].z * inv * w.z * silu_f(g[i].z), v[i].w * inv * w.w * silu_f(g[i].w));
                }
            put(unit, c, v[0], v[1]);
        }
    }
    amax = lp_block<1>(amax, red);  // its barriers also publish the blocks' largest values
    // One unit of value per position: the largest value lies in [2^14, 2^15). hi + lo then keep 22 bits of every value above
    // 2^-28 of the largest, and an absolute 2^-50 of it below. A streaming product has a unit for each block and keeps 22
    // bits above 2^-13 (4-bit codes) or 2^-9 of the block's largest value, 2^-35 or 2^-31 of it below: the row's unit leaves
    // no block fewer unless its largest value is below 2^-15 of the row's. Then every block gets its own unit.
    auto exponent = [](float x) { return (int)((__float_as_uint(x) >> 23) & 0xff) - 127; };
    int spread = 0;
    for (uint32_t i = tid; i < p.blocks_padded; i += kRowsThreads)
        if (block_max[i] > 0.f && exponent(block_max[i]) < exponent(amax) - 15) spread = 1;
    spread = __syncthreads_or(spread);
    auto unit_exponent = [&](float largest) {
        const int e = exponent(largest);
        return max(!(largest > 0.f) || e > 127 ? 14 : e, -100);  // zero or non-finite: factor 1
    };
    if (tid == 0) {
        p.in.unit[pos] = __uint_as_float((uint32_t)(unit_exponent(amax) - 14 + 127) << 23);
        p.in.spread[pos] = spread ? 0xff : 0;
    }
    for (uint32_t unit = tid; unit < units; unit += kRowsThreads) {
        const uint32_t block = unit >> 3;
        const int e = unit_exponent(spread ? block_max[block] : amax);
        const float f = __uint_as_float((uint32_t)(14 - e + 127) << 23);
        if ((unit & 7) == 0) p.in.block_unit[(size_t)block * p.in.pos_pad + pos] = __uint_as_float((uint32_t)(e - 14 + 127) << 23);
        const float4 a = first[unit], b = second[unit];
        const float x[4] = {a.x * f, a.y * f, a.z * f, a.w * f}, y[4] = {b.x * f, b.y * f, b.z * f, b.w * f};
        __align__(16) __half2 hi[4], lo[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            hi[s] = __floats2half2_rn(x[s], y[s]);
            lo[s] = __floats2half2_rn((x[s] - __low2float(hi[s])) * (float)(1 << kLoShift), (y[s] - __high2float(hi[s])) * (float)(1 << kLoShift));
        }
        uint8_t *d = p.in.x + ((size_t)block * 2 * p.in.pos_pad + pos) * 128 + ((unit & 7) ^ (pos & 7)) * 16;
        *reinterpret_cast<uint4 *>(d) = *reinterpret_cast<uint4 *>(hi);
        *reinterpret_cast<uint4 *>(d + (size_t)p.in.pos_pad * 128) = *reinterpret_cast<uint4 *>(lo);
    }
}

// ------------------------------------------------------------------ linear attention
// Causal conv + SiLU (reference.rs:159-187) for sixteen positions of 128 channels, which are one head of q, k or v;
// q and k leave normalised (k^ and q^ / sqrt(128) of delta.cu).
constexpr int kConvTokens = 16;
struct LongConv {
    LongOut o;
    const float *conv_state, *conv_w;
    float *qkv;
    uint32_t key_width, channels, kernel, m;
};
__global__ void __launch_bounds__(128) k_long_conv(const LongConv p) {
    pdl_launch();
    pdl_wait();
    __shared__ float red[kConvTokens][4];
    const uint32_t ch = blockIdx.x * 128 + threadIdx.x, m0 = blockIdx.y * kConvTokens, warp = threadIdx.x >> 5;
    const uint32_t K = p.kernel;
    float st[8], cw[8], y[kConvTokens];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        st[j] = cw[j] = 0.f;
        if ((uint32_t)j < K) {
            cw[j] = p.conv_w[(size_t)ch * K + j];
            // st[j]: input of position m0 - K + j
            const int at = (int)m0 - (int)K + j;
            st[j] = at >= 0 ? p.o.y[(size_t)at * p.o.rows + ch] : p.conv_state[(size_t)ch * K + (uint32_t)((int)K + at)];
        }
    }
#pragma unroll
    for (int i = 0; i < kConvTokens; ++i) y[i] = m0 + i < p.m ? p.o.y[(size_t)(m0 + i) * p.o.rows + ch] : 0.f;
    for (uint32_t sp = 1; sp < p.o.splits; ++sp) {  // all loads of a partial sum together
        const float *o = p.o.y + sp * p.o.split_stride + ch;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int at = (int)m0 - (int)K + j;
            if ((uint32_t)j < K && at >= 0) st[j] += o[(size_t)at * p.o.rows];
        }
#pragma unroll
        for (int i = 0; i < kConvTokens; ++i)
            if (m0 + i < p.m) y[i] += o[(size_t)(m0 + i) * p.o.rows];
    }
#pragma unroll
    for (int i = 0; i < kConvTokens; ++i) {
        const float x = y[i];
#pragma unroll
        for (int j = 0; j < 7; ++j)
            if ((uint32_t)j + 1 < K) st[j] = st[j + 1];
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if ((uint32_t)j + 1 == K) st[j] = x;
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if ((uint32_t)j < K) sum += st[j] * cw[j];
        y[i] = silu_f(sum);
    }
    if (ch < 2 * p.key_width) {  // all 128 channels of the CTA alike
#pragma unroll
        for (int i = 0; i < kConvTokens; ++i) {
            float s = y[i] * y[i];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if ((threadIdx.x & 31) == 0) red[i][warp] = s;
        }
        __syncthreads();
        const float scale = ch < p.key_width ? 1.0f / sqrtf(128.0f) : 1.0f;
#pragma unroll
        for (int i = 0; i < kConvTokens; ++i)
            y[i] = y[i] * (1.0f / sqrtf(red[i][0] + red[i][1] + red[i][2] + red[i][3] + 1e-6f)) * scale;
    }
#pragma unroll
    for (int i = 0; i < kConvTokens; ++i)
        if (m0 + i < p.m) p.qkv[(size_t)(m0 + i) * p.channels + ch] = y[i];
}

// Decay and beta of every (position, head) (decoder.rs:29-35,881,897-902), and the conv state after the pass (m is
// at least the kernel's width). In a kernel of its own: the conv kernel's CTAs read the state before the pass.
struct LongGates {
    LongOut o;
    const float *a_log, *dt_bias;
    float *decay, *beta, *conv_state;
    uint32_t heads, off, channels, kernel, m;
};
__global__ void __launch_bounds__(256) k_long_gates(const LongGates p) {
    pdl_launch();
    pdl_wait();
    const uint32_t i = blockIdx.x * 256 + threadIdx.x, n = p.m * p.heads;
    if (i < n) {
        const uint32_t pos = i / p.heads, h = i % p.heads;
        const float x = lp_out(p.o, p.off + h, pos) + p.dt_bias[h];
        const float sp = x > 20.0f ? x : log1pf(expf(x));
        p.decay[i] = expf(-expf(p.a_log[h]) * sp);
        p.beta[i] = 1.0f / (1.0f + expf(-lp_out(p.o, p.off + p.heads + h, pos)));
    } else if (i - n < p.channels * p.kernel) {
        const uint32_t ch = (i - n) / p.kernel, j = (i - n) % p.kernel;
        p.conv_state[(i - n)] = lp_out(p.o, ch, p.m - p.kernel + j);
    }
}

// The gated-delta recurrence (delta.cu) over all positions, four tokens at a time. With the state S before the group, the decays'
// products D_j = d_0 .. d_j, D_ij = d_(i+1) .. d_j and e_j = (v_j - memory read by k_j) * beta_j,
//     e_j      = beta_j (v_j - D_j S k_j - sum_(i<j) D_ij (k_i . k_j) e_i)
//     output_j = D_j S q_j + sum_(i<=j) D_ij (k_i . q_j) e_i
//     S'       = D_3 S + sum_i D_i3 k_i e_i
// so that the group's eight products with the state are independent and the chain (products, sums across lanes, update) is walked once
// in four tokens. With u_j = v_j - D_j S k_j, e is a triangular matrix times u; k_long_coefs forms that matrix, which is the same for all
// columns of a head, and leaves it with D_i3 (F, for the update) and with the outputs' factors (G) multiplied in.
constexpr uint32_t kGroup = 4, kCoefs = 36;  // of a group: D[4], F[j][i], G[j][i] (zero for i > j)
struct LongCoefs {
    const float *qkv, *decay, *beta;
    float *coefs;  // [group][head][kCoefs]
    uint32_t key_width, channels, heads, qk_heads, m;
};
// A warp per (group, key head), then a lane per factor of each of its value heads. Tokens past the last one have decay 1 and factors 0.
__global__ void __launch_bounds__(128) k_long_coefs(const LongCoefs p) {
    pdl_launch();
    pdl_wait();
    __shared__ float dots[4][kGroup][2 * kGroup];  // per warp: k_i . (k_0 .. k_3, q_0 .. q_3)
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, item = blockIdx.x * 4 + warp;
    const uint32_t group = item / p.qk_heads, kh = item % p.qk_heads, t0 = group * kGroup;
    if (t0 >= p.m) return;
    float4 x[2 * kGroup];
#pragma unroll
    for (uint32_t j = 0; j < 2 * kGroup; ++j) {
        const uint32_t t = t0 + j % kGroup;
        x[j] = t < p.m ? *reinterpret_cast<const float4 *>(p.qkv + (size_t)t * p.channels + (j < kGroup ? p.key_width : 0) + kh * 128 + lane * 4)
                       : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (uint32_t i = 0; i < kGroup; ++i)
#pragma unroll
        for (uint32_t j = i + 1; j < kGroup + kGroup; ++j) {
            if (j >= kGroup && j - kGroup < i) continue;
            float v = (x[i].x * x[j].x + x[i].y * x[j].y) + (x[i].z * x[j].z + x[i].w * x[j].w);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) dots[warp][i][j] = v;
        }
    __syncwarp();
    const uint32_t repeat = p.heads / p.qk_heads;
    for (uint32_t r = 0; r < repeat; ++r) {
        const uint32_t head = kh * repeat + r;
        float d[kGroup], beta[kGroup];
#pragma unroll
        for (uint32_t j = 0; j < kGroup; ++j) {
            const bool in = t0 + j < p.m;
            d[j] = in ? p.decay[(size_t)(t0 + j) * p.heads + head] : 1.0f;
            beta[j] = in ? p.beta[(size_t)(t0 + j) * p.heads + head] : 0.f;
        }
        auto between = [&](uint32_t i, uint32_t j) {  // the decays of tokens i + 1 .. j
            float v = 1.0f;
#pragma unroll
            for (uint32_t l = 0; l < kGroup; ++l)
                if (l > i && l <= j) v *= d[l];
            return v;
        };
        float kk[kGroup][kGroup], T[kGroup][kGroup];  // e = T u; every lane forms all of it
#pragma unroll
        for (uint32_t j = 0; j < kGroup; ++j)
#pragma unroll
            for (uint32_t i = 0; i < kGroup; ++i) {
                if (i < j) kk[i][j] = between(i, j) * dots[warp][i][j];
                T[j][i] = i == j ? 1.0f : 0.f;
            }
#pragma unroll
        for (uint32_t j = 0; j < kGroup; ++j)
#pragma unroll
            for (uint32_t i = 0; i <= j; ++i) {
#pragma unroll
                for (uint32_t l = i; l < j; ++l) T[j][i] -= kk[l][j] * T[l][i];
                T[j][i] *= beta[j];
            }
        float mine = 0.f, last = 0.f;  // factors `lane` and, of the first lanes, 32 + lane
#pragma unroll
        for (uint32_t j = 0; j < kGroup; ++j) {
            if (lane == j) mine = d[0] * between(0, j);
#pragma unroll
            for (uint32_t i = 0; i <= j; ++i) {
                if (lane == kGroup + j * kGroup + i) mine = between(j, kGroup - 1) * T[j][i];
                float g = 0.f;
#pragma unroll
                for (uint32_t l = i; l <= j; ++l) g += between(l, j) * dots[warp][l][kGroup + j] * T[l][i];
                const uint32_t at = kGroup + kGroup * kGroup + j * kGroup + i;
                if (lane == at) mine = g;
                if (lane + 32 == at) last = g;
            }
        }
        float *out = p.coefs + ((size_t)group * p.heads + head) * kCoefs;
        out[lane] = mine;
        if (lane + 32 < kCoefs) out[lane + 32] = last;
    }
}

// The scan itself. Bound by what goes through shared memory (a 16-byte read of all lanes is four cycles of its pipe, whether lanes share
// addresses or not) and by the packed products with the state. A warp owns four value columns with their 128 keys: 16 lanes per
// pair of columns, 2 x 8 state values each in registers, so that a key or query read serves two columns. 16 columns and 4 warps per
// CTA, 8 CTAs per head: the fullest SM decides (48 heads: 48 columns on it, 64 with 32 columns per CTA). The tokens' inputs are
// staged sixteen at a time, a block ahead. 999 tokens of 48 heads: 238 us and 10 for the factors; token by token with 8 lanes per column
// 332, groups of four on that layout 309 (the shared-memory pipe 86 % busy), with two columns per 8 lanes 325 (too few warps).
constexpr int kScanTokens = 16, kScanCols = 16, kScanThreads = kScanCols * 8, kScanCtas = 128 / kScanCols;  // CTAs per head
struct LongScan {
    const float *qkv, *coefs;
    float *state, *out;
    uint32_t key_width, channels, heads, qk_heads, m;
};
__global__ void __launch_bounds__(kScanThreads) k_long_delta(const LongScan p) {
    pdl_launch();
    pdl_wait();
    constexpr uint32_t kGroups = kScanTokens / kGroup;
    __shared__ __align__(16) float qs[2][kScanTokens][128], ks[2][kScanTokens][128], vs[2][kScanTokens][kScanCols];
    __shared__ __align__(16) float cs[2][kGroups][kCoefs];
    __shared__ __align__(8) float os[kScanTokens][kScanCols];
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, sub = lane & 15, c = warp * 4 + (lane >> 4) * 2;
    const uint32_t head = blockIdx.x / kScanCtas, col0 = blockIdx.x % kScanCtas * kScanCols, kh = head / (p.heads / p.qk_heads);
    // this lane's keys are sub * 4 + 64 i .. + 3, i < 2, of columns c and c + 1; two keys per register pair
    f32x2 s[2][4];
    float *state = p.state + (size_t)head * 128 * 128 + col0 + c;
    auto state_at = [&](int i) { return reinterpret_cast<float2 *>(state + (size_t)((i >> 1) * 64 + sub * 4 + (i & 1) * 2) * 128); };
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 a = state_at(i)[0], b = state_at(i)[64];
        s[0][i] = pack2(a.x, b.x);
        s[1][i] = pack2(a.y, b.y);
    }
    auto load = [&](f32x2(&d)[4], const float *row) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const ulonglong2 u = *reinterpret_cast<const ulonglong2 *>(row + i * 64 + sub * 4);
            d[2 * i] = u.x;
            d[2 * i + 1] = u.y;
        }
    };
    auto dot = [](const f32x2(&a)[4], const f32x2(&b)[4]) {
        float u, v;
        unpack2(fma2(a[3], b[3], fma2(a[2], b[2], fma2(a[1], b[1], mul2(a[0], b[0])))), u, v);
        return u + v;
    };
    // After the sums over a pair's lanes, lane sub holds token sub & 3, column c + (sub >> 3), the product with its query (sub & 4) or key.
    const bool b8 = sub & 8, b4 = sub & 4, b2 = sub & 2, b1 = sub & 1;
    const uint32_t tok = sub & 3, of_column = (lane & 24);  // first lane of this one's column
    auto copy16 = [](void *dst, const void *src) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                     : "memory");
    };
    auto fetch = [&](uint32_t t0, uint32_t b) {
        const uint32_t n = min((uint32_t)kScanTokens, p.m - t0), groups = (n + kGroup - 1) / kGroup;
        for (uint32_t i = tid; i < groups * kGroup * 32; i += kScanThreads) {
            const uint32_t t = i >> 5, at = (i & 31) * 4;
            const float *row = p.qkv + (size_t)(t0 + t) * p.channels + kh * 128 + at;
            if (t < n) {
                copy16(&qs[b][t][at], row);
                copy16(&ks[b][t][at], row + p.key_width);
            } else {  // the last group's missing tokens: their factors are 0
                *reinterpret_cast<float4 *>(&qs[b][t][at]) = make_float4(0.f, 0.f, 0.f, 0.f);
                *reinterpret_cast<float4 *>(&ks[b][t][at]) = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        for (uint32_t i = tid; i < groups * kGroup * (kScanCols / 4); i += kScanThreads) {
            const uint32_t t = i / (kScanCols / 4), at = i % (kScanCols / 4) * 4;
            if (t < n)
                copy16(&vs[b][t][at], p.qkv + (size_t)(t0 + t) * p.channels + 2 * p.key_width + head * 128 + col0 + at);
            else
                *reinterpret_cast<float4 *>(&vs[b][t][at]) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        for (uint32_t i = tid; i < groups * (kCoefs / 4); i += kScanThreads)
            copy16(&cs[b][i / (kCoefs / 4)][i % (kCoefs / 4) * 4],
                   p.coefs + ((size_t)(t0 / kGroup + i / (kCoefs / 4)) * p.heads + head) * kCoefs + i % (kCoefs / 4) * 4);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0, 0);
    for (uint32_t t0 = 0, b = 0; t0 < p.m; t0 += kScanTokens, b ^= 1) {
        const uint32_t n = min((uint32_t)kScanTokens, p.m - t0);
        if (t0 + kScanTokens < p.m) {
            fetch(t0 + kScanTokens, b ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        for (uint32_t g = 0; g < (n + kGroup - 1) / kGroup; ++g) {
            const uint32_t t = g * kGroup;
            const float *co = cs[b][g];
            const float D = co[tok], D3 = co[kGroup - 1], v = vs[b][t + tok][c + b8];
            const float4 F = *reinterpret_cast<const float4 *>(co + kGroup + (b4 ? kGroup * kGroup : 0) + tok * kGroup);
            f32x2 k[kGroup][4];
            float x[2][2 * kGroup];
#pragma unroll
            for (uint32_t j = 0; j < kGroup; ++j) {
                load(k[j], ks[b][t + j]);
                x[0][j] = dot(s[0], k[j]);
                x[1][j] = dot(s[1], k[j]);
            }
#pragma unroll
            for (uint32_t j = 0; j < kGroup; ++j) {
                f32x2 q[4];
                load(q, qs[b][t + j]);
                x[0][kGroup + j] = dot(s[0], q);
                x[1][kGroup + j] = dot(s[1], q);
            }
            float r[8], y[4], z[2];
#pragma unroll
            for (int i = 0; i < 8; ++i) r[i] = (b8 ? x[1][i] : x[0][i]) + __shfl_xor_sync(0xffffffffu, b8 ? x[0][i] : x[1][i], 8);
#pragma unroll
            for (int i = 0; i < 4; ++i) y[i] = (b4 ? r[4 + i] : r[i]) + __shfl_xor_sync(0xffffffffu, b4 ? r[i] : r[4 + i], 4);
#pragma unroll
            for (int i = 0; i < 2; ++i) z[i] = (b2 ? y[2 + i] : y[i]) + __shfl_xor_sync(0xffffffffu, b2 ? y[i] : y[2 + i], 2);
            const float w = (b1 ? z[1] : z[0]) + __shfl_xor_sync(0xffffffffu, b1 ? z[0] : z[1], 1);
            const f32x2 d2 = pack2(D3, D3);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                s[0][i] = mul2(s[0][i], d2);
                s[1][i] = mul2(s[1][i], d2);
            }
            const float u = v - D * w;  // of a key's lane
            float us[kGroup];
#pragma unroll
            for (uint32_t i = 0; i < kGroup; ++i) us[i] = __shfl_sync(0xffffffffu, u, of_column + i);
            float e = F.x * us[0];  // no term of a later token, whatever its value
            if (b1 || b2) e += F.y * us[1];
            if (b2) e += F.z * us[2];
            if (b2 && b1) e += F.w * us[3];
            if (b4) os[t + tok][c + b8] = D * w + e;
#pragma unroll
            for (uint32_t j = 0; j < kGroup; ++j) {
                const float f0 = __shfl_sync(0xffffffffu, e, (lane & 16) + j), f1 = __shfl_sync(0xffffffffu, e, (lane & 16) + 8 + j);
                const f32x2 e0 = pack2(f0, f0), e1 = pack2(f1, f1);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    s[0][i] = fma2(k[j][i], e0, s[0][i]);
                    s[1][i] = fma2(k[j][i], e1, s[1][i]);
                }
            }
        }
        __syncthreads();  // outputs complete, and buffer b free for the fetch of the next round
        for (uint32_t i = tid; i < n * kScanCols; i += kScanThreads)
            p.out[((size_t)(t0 + i / kScanCols) * p.heads + head) * 128 + col0 + i % kScanCols] = os[i / kScanCols][i % kScanCols];
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float2 a, b;
        unpack2(s[0][i], a.x, b.x);
        unpack2(s[1][i], a.y, b.y);
        state_at(i)[0] = a;
        state_at(i)[64] = b;
    }
}

// ------------------------------------------------------------------ full attention, before the cache
// k_attn_pre (layers.cu) for a whole pass: one CTA per position, its angles once, a warp per head.
struct LongAttnPre {
    LongOut o;
    AttnGeom g;
    const float *q_norm, *k_norm;
    uint64_t rope_position, cache_slot;
    float *q;
    void *k_cache, *v_cache;
    const uint32_t *page_table;
    uint32_t page_tokens;
    int kv_only;
};
__device__ __forceinline__ void lp_store(float *p, float v) { *p = v; }
__device__ __forceinline__ void lp_store(__nv_bfloat16 *p, float v) { *p = __float2bfloat16_rn(v); }
template <typename T>
__global__ void __launch_bounds__(256) k_long_attn_pre(const LongAttnPre p) {
    pdl_launch();
    pdl_wait();
    __shared__ float cs[128], sn[128], buf[8][256];
    const AttnGeom &g = p.g;
    const uint32_t m = blockIdx.x, hd = g.head_dim, half = g.rotary_dim / 2, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t at = p.cache_slot + m;
    const size_t slot = (size_t)p.page_table[at / p.page_tokens] * p.page_tokens + at % p.page_tokens;
    if (threadIdx.x < half) {
        const float inv_freq = powf(g.theta, -((float)(2 * threadIdx.x)) / (float)g.rotary_dim);
        const float ang = (float)(p.rope_position + m) * inv_freq;
        cs[threadIdx.x] = cosf(ang);
        sn[threadIdx.x] = sinf(ang);
    }
    __syncthreads();
    const uint32_t k_row0 = g.q_heads * 2 * hd, v_row0 = k_row0 + g.kv_heads * hd;
    for (uint32_t hi = (p.kv_only ? g.q_heads : 0) + warp; hi < g.q_heads + 2 * g.kv_heads; hi += 8) {
        if (hi >= g.q_heads + g.kv_heads) {
            const uint32_t kh = hi - g.q_heads - g.kv_heads;
            T *v = (T *)p.v_cache + (slot * g.kv_heads + kh) * hd;
            for (uint32_t d = lane; d < hd; d += 32) lp_store(v + d, lp_out(p.o, v_row0 + kh * hd + d, m));
            continue;
        }
        const bool is_q = hi < g.q_heads;
        const uint32_t head = is_q ? hi : hi - g.q_heads, row0 = is_q ? head * 2 * hd : k_row0 + head * hd;
        float x[8], sq = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            x[j] = (uint32_t)j * 32 < hd ? lp_out(p.o, row0 + j * 32 + lane, m) : 0.f;  // hd is a multiple of 64
            sq += x[j] * x[j];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        const float inv = 1.0f / sqrtf(sq / (float)hd + g.eps);
        const float *w = is_q ? p.q_norm : p.k_norm;
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if ((uint32_t)j * 32 < hd) {
                x[j] = x[j] * inv * (1.0f + w[j * 32 + lane]);
                buf[warp][j * 32 + lane] = x[j];
            }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if ((uint32_t)j * 32 < hd) {
                const uint32_t d = j * 32 + lane;
                float v = x[j];
                if (d < half)
                    v = x[j] * cs[d] - buf[warp][d + half] * sn[d];
                else if (d < 2 * half)
                    v = x[j] * cs[d - half] + buf[warp][d - half] * sn[d - half];
                if (is_q)
                    p.q[((size_t)m * g.q_heads + head) * hd + d] = v;
                else
                    lp_store((T *)p.k_cache + (slot * g.kv_heads + head) * hd + d, v);
            }
        __syncwarp();
    }
}

// The splits of a query's context merged into the first one's row (sum 1: normalised). One CTA per (position, head), a
// thread per dimension; a warp forms the splits' weights.
struct LongMerge {
    float *ws;
    uint32_t q_heads, kv_heads, per_group, splits, m;
};
__global__ void __launch_bounds__(256) k_long_attn_merge(const LongMerge p) {
    pdl_launch();
    pdl_wait();
    __shared__ float wgt[kAttnMaxSplits];
    const uint32_t hd = blockDim.x, pos = blockIdx.x / p.q_heads, head = blockIdx.x % p.q_heads, d = threadIdx.x;
    float *r = p.ws + attn_row(pos, head, 0, p.m, p.per_group, p.splits, p.q_heads, p.kv_heads) * (hd + 2);
    const size_t stride = (attn_row(pos, head, 1, p.m, p.per_group, p.splits, p.q_heads, p.kv_heads) -
                           attn_row(pos, head, 0, p.m, p.per_group, p.splits, p.q_heads, p.kv_heads)) * (hd + 2);
    if (d < 32) {
        float mx = -INFINITY, den = 0.f;
        for (uint32_t s = d; s < p.splits; s += 32) mx = fmaxf(mx, r[s * stride + hd]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        for (uint32_t s = d; s < p.splits; s += 32) {
            const float ms = r[s * stride + hd], w = ms > -INFINITY ? expf(ms - mx) : 0.f;
            wgt[s] = w;
            den += r[s * stride + hd + 1] * w;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
        for (uint32_t s = d; s < p.splits; s += 32) wgt[s] /= den;
    }
    __syncthreads();
    float acc = 0.f;
#pragma unroll 8
    for (uint32_t s = 0; s < p.splits; ++s) acc += r[s * stride + d] * wgt[s];
    r[d] = acc;
    if (d == 0) r[hd + 1] = 1.0f;
}

// ------------------------------------------------------------------ host side
namespace {

// Splits of the context in a long pass of m positions. A group's CTAs are one per KV head, too few of them where the pass is
// short: 17 positions at four KV heads are 16 CTAs. The parts are as many as finish soonest, counted in rounds over the SMs
// of tiles of 64 tokens with two tiles' time for a CTA's start and end, and no more than the workspace holds.
uint32_t attention_splits(const ctox_exec *e, uint32_t per_group, uint64_t pos0, uint32_t m) {
    const uint64_t tiles = (pos0 + m + 63) / 64, sms = (uint64_t)e->ctx->sm_count;
    const uint64_t ctas = (uint64_t)e->cfg.num_key_value_heads * ((m + per_group - 1) / per_group);
    uint64_t most = std::min<uint64_t>(e->attn_splits_max, e->long_pass->cap / m), best = 1, best_cost = ~0ull;
    most = std::min(most, tiles);
    for (uint64_t s = 1; s <= most; ++s) {
        const uint64_t cost = (ctas * s + sms - 1) / sms * ((tiles + s - 1) / s + 2);
        if (cost < best_cost) {
            best_cost = cost;
            best = s;
        }
    }
    return (uint32_t)best;
}

constexpr uint32_t kLongCap = 1024;  // positions per pass: the buffers take 0.39 GB at the flagship's widths

AttnGeom geom(const ctox_exec *e) {
    const ctox_model_config &c = e->cfg;
    return AttnGeom{c.num_attention_heads, c.num_key_value_heads, c.head_dim, c.rotary_dim, c.rope_theta, c.rms_norm_epsilon,
                    e->ctx->dev_error};
}

template <int MODE>
ctox_status rows(ctox_exec *e, RowsArgs &a, uint32_t m, ctox_matvec *next) {
    ctox_ctx *ctx = e->ctx;
    a.in = e->long_pass->in;
    a.has_next = next != nullptr;
    if (next) {
        a.s_in = next->s_in;
        a.blocks_padded = next->blocks_padded;
        a.dt = next->parts[0].dt;
    }
    const size_t smem = (next ? (size_t)next->blocks_padded * 65 : a.width) * 4;
    CTOX_CUDA(ctx, launch_pdl(k_long_rows<MODE>, dim3(m), dim3(rows_threads(MODE)), smem, ctx->stream, a));
    return CTOX_OK;
}

// h = base (null: 0) + add, then the norm: into xn_out and / or as the input of `next`.
ctox_status rows_norm(ctox_exec *e, uint32_t m, const float *base, const LongOut *add, const float *w, float *xn_out,
                      ctox_matvec *next) {
    RowsArgs a{};
    if (add) a.o = *add;
    a.a = base;
    a.h = e->long_pass->h;
    a.w = w;
    a.xn_out = xn_out;
    a.eps = e->cfg.rms_norm_epsilon;
    a.width = e->cfg.hidden_size;
    return rows<ROWS_NORM>(e, a, m, next);
}

ctox_status product(ctox_exec *e, ctox_matvec *mv, uint32_t m, LongOut *out, uint64_t row0 = 0) {
    LongPass &L = *e->long_pass;
    return launch_packed_gemm(mv, L.in, m, row0, mv->rows, L.y, L.y_floats, out);
}

ctox_status attn_pre(ctox_exec *e, uint32_t l, const LongOut &o, uint32_t m, uint64_t rope_pos0, uint64_t slot0,
                     const uint32_t *page_table, bool kv_only) {
    ctox_ctx *ctx = e->ctx;
    const ctox_model_config &c = e->cfg;
    const LongAttnPre a{o, geom(e), e->w[l].q_norm, e->w[l].k_norm, rope_pos0, slot0, e->long_pass->aq, e->s[l].k_cache,
                        e->s[l].v_cache, page_table, c.kv_page_tokens, kv_only};
    if (c.kv_dtype == CTOX_BF16)
        CTOX_CUDA(ctx, launch_pdl(k_long_attn_pre<__nv_bfloat16>, dim3(m), dim3(256), 0, ctx->stream, a));
    else
        CTOX_CUDA(ctx, launch_pdl(k_long_attn_pre<float>, dim3(m), dim3(256), 0, ctx->stream, a));
    return CTOX_OK;
}

// The mixer of layer l; its input projection's output is `o`. Leaves the input of the output projection.
ctox_status mixer(ctox_exec *e, uint32_t l, const LongOut &o, uint32_t m, uint64_t pos0) {
    ctox_ctx *ctx = e->ctx;
    const ctox_model_config &c = e->cfg;
    LongPass &L = *e->long_pass;
    LayerW &lw = e->w[l];
    LayerS &ls = e->s[l];
    RowsArgs a{};
    a.o = o;
    a.eps = c.rms_norm_epsilon;
    a.m = m;
    if (lw.full) {
        const AttnGeom g = geom(e);
        const int bf16 = c.kv_dtype == CTOX_BF16;
        EX(attn_pre(e, l, o, m, pos0, pos0, e->page_table, false));
        a.per_group = attention_group_positions(g, bf16, m);
        a.splits = attention_splits(e, a.per_group, pos0, m);
        timing_begin(ctx);
        launch_attention_groups(ctx->stream, g, L.aq, ls.k_cache, ls.v_cache, bf16, e->page_table, c.kv_page_tokens, pos0, m,
                                a.splits, L.attn);
        if (a.splits > 1)
            launch_pdl(k_long_attn_merge, dim3(m * g.q_heads), dim3(g.head_dim), 0, ctx->stream,
                       LongMerge{L.attn, g.q_heads, g.kv_heads, a.per_group, a.splits, m});
        timing_end(ctx, KC_ATTENTION, 2.0 * (double)(pos0 + m) * e->kv_width * (bf16 ? 2 : 4),
                   4.0 * ((double)pos0 + 0.5 * m) * e->q_width * m);
        CTOX_CUDA(ctx, cudaGetLastError());
        a.a = L.attn;
        a.width = e->q_width;
        a.q_heads = g.q_heads;
        a.kv_heads = g.kv_heads;
        a.head_dim = g.head_dim;
        return rows<ROWS_ATTENTION>(e, a, m, lw.out);
    }
    const uint32_t heads = c.linear_num_value_heads, kernel = c.linear_conv_kernel_dim;
    CTOX_CUDA(ctx, launch_pdl(k_long_conv, dim3(e->channels / 128, (m + kConvTokens - 1) / kConvTokens), dim3(128), 0, ctx->stream,
                              LongConv{o, ls.conv_state, lw.conv_w, L.qkv, e->key_width, e->channels, kernel, m}));
    CTOX_CUDA(ctx, launch_pdl(k_long_gates, dim3((m * heads + e->channels * kernel + 255) / 256), dim3(256), 0, ctx->stream,
                              LongGates{o, lw.a_log, lw.dt_bias, L.g, L.beta, ls.conv_state, heads, e->channels + e->value_width,
                                        e->channels, kernel, m}));
    timing_begin(ctx);
    CTOX_CUDA(ctx, launch_pdl(k_long_coefs, dim3(((m + kGroup - 1) / kGroup * c.linear_num_key_heads + 3) / 4), dim3(128), 0, ctx->stream,
                              LongCoefs{L.qkv, L.g, L.beta, L.coefs, e->key_width, e->channels, heads, c.linear_num_key_heads, m}));
    CTOX_CUDA(ctx, launch_pdl(k_long_delta, dim3(heads * kScanCtas), dim3(kScanThreads), 0, ctx->stream,
                              LongScan{L.qkv, L.coefs, ls.delta[ls.cur], L.core, e->key_width, e->channels, heads,
                                       c.linear_num_key_heads, m}));
    timing_end(ctx, KC_LINEAR_ATTENTION, 2.0 * 4.0 * 128 * 128 * heads, 8.0 * 128 * 128 * heads * m);
    a.a = L.core;
    a.w = lw.lin_norm;
    a.width = e->value_width;
    a.off = e->channels;
    return rows<ROWS_DELTA>(e, a, m, lw.out);
}

}  // namespace

uint32_t long_min(const ctox_exec *e) {
    const bool cores = !attention_on_tensor_cores(geom(e), e->cfg.kv_dtype == CTOX_BF16);
    return cores && e->position > kDeepCores ? kLongMinDeepCores : kLongMin;
}

ctox_status long_warmup(ctox_exec *e) {
    ctox_ctx *ctx = e->ctx;
    const ctox_model_config &c = e->cfg;
    if (e->long_pass || e->tp_world > 1 || c.max_context_tokens < 64) return CTOX_OK;
    std::vector<ctox_matvec *> mats;
    for (LayerW &lw : e->w)
        for (ctox_matvec *mv : {lw.in_fan, lw.out, lw.gate_up, lw.down}) mats.push_back(mv);
    if (e->mtp_fc) mats.push_back(e->mtp_fc);
    uint32_t blocks = 0;
    uint64_t rows = 0;
    for (ctox_matvec *mv : mats) {
        if (mv->parts.size() != 1 || (size_t)mv->blocks_padded * 260 + 2048 > (size_t)ctx->max_smem_optin) return CTOX_OK;
        blocks = mv->blocks_padded > blocks ? mv->blocks_padded : blocks;
        rows = mv->rows > rows ? mv->rows : rows;
    }
    bool usable = false;
    EX(packed_gemm_init(ctx, &usable));
    if (!usable) return CTOX_OK;
    for (auto kernel : {k_long_rows<ROWS_NORM>, k_long_rows<ROWS_SWIGLU>, k_long_rows<ROWS_ATTENTION>, k_long_rows<ROWS_DELTA>,
                        k_long_rows<ROWS_MTP>})
        CTOX_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ctx->max_smem_optin - 1024));
    const uint32_t cap = c.max_context_tokens < kLongCap ? (c.max_context_tokens + 7) / 8 * 8 : kLongCap;
    const uint32_t pos_pad = cap + kLongPosTile;  // a last tile may start anywhere below cap
    LongPass *L = new LongPass();
    e->long_pass = L;
    auto get = [&](auto **p, size_t n) {
        const ctox_status rc = dev_alloc(ctx, (void **)p, n * sizeof(**p), true);
        if (!rc) {
            L->owned.emplace_back((void *)*p, n * sizeof(**p));
            e->session_bytes += n * sizeof(**p);
        }
        return rc;
    };
    L->cap = cap;
    L->in.pos_pad = pos_pad;
    L->y_floats = (size_t)cap * rows;
    const uint64_t H = c.hidden_size;
    ctox_status rc = get(&L->in.x, long_in_bytes(blocks, pos_pad));
    if (!rc) rc = get(&L->in.unit, pos_pad);
    if (!rc) rc = get(&L->in.block_unit, (size_t)blocks * pos_pad + kUnitTail);
    if (!rc) rc = get(&L->in.spread, pos_pad + kUnitTail);
    if (!rc) rc = get(&L->y, L->y_floats);
    if (!rc) rc = get(&L->h, cap * H);
    if (!rc) rc = get(&L->final_hidden, cap * H);
    if (!rc) rc = get(&L->qkv, (size_t)cap * e->channels);
    if (!rc) rc = get(&L->core, (size_t)cap * e->value_width);
    if (!rc) rc = get(&L->g, (size_t)cap * c.linear_num_value_heads);
    if (!rc) rc = get(&L->beta, (size_t)cap * c.linear_num_value_heads);
    if (!rc) rc = get(&L->coefs, (size_t)(cap + kGroup - 1) / kGroup * c.linear_num_value_heads * kCoefs);
    if (!rc) rc = get(&L->aq, (size_t)cap * e->q_width);
    if (!rc) rc = get(&L->attn, (size_t)cap * c.num_attention_heads * (c.head_dim + 2));
    if (!rc) rc = get(&L->tokens, cap);
    for (cudaEvent_t &ev : L->layer_done)
        if (!rc && cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) rc = CTOX_INVALID_STATE;
    if (rc)  // no room: the model runs with short passes alone, as it would without them
        long_release(e);
    else
        ctx->spares.push_back(Spare{e, [](void *owner) {
            ctox_exec *e = (ctox_exec *)owner;
            if (e->long_pass->busy || cudaStreamSynchronize(e->ctx->stream) != cudaSuccess) return false;
            long_release(e);
            return true;
        }});
    return CTOX_OK;
}

void long_release(ctox_exec *e) {
    if (!e->long_pass) return;
    for (auto &o : e->long_pass->owned) {
        dev_free(e->ctx, o.first, o.second);
        e->session_bytes -= o.second;
    }
    for (cudaEvent_t ev : e->long_pass->layer_done)
        if (ev) cudaEventDestroy(ev);
    delete e->long_pass;
    e->long_pass = nullptr;
}

ctox_status long_target_pass(ctox_exec *e, const uint32_t *tokens, uint32_t m, const volatile int32_t *cancel) {
    ctox_ctx *ctx = e->ctx;
    const ctox_model_config &c = e->cfg;
    LongPass &L = *e->long_pass;
    const uint64_t pos0 = e->position;
    const size_t row = (size_t)c.hidden_size * 4;
    LongOut o;
    CTOX_CUDA(ctx, cudaMemcpyAsync(L.tokens, tokens, (size_t)m * 4, cudaMemcpyHostToDevice, ctx->stream));
    EX(matvec_embed_rows(e->embed, L.tokens, m, L.h));
    EX(rows_norm(e, m, L.h, nullptr, e->w[0].in_ln, nullptr, e->w[0].in_fan));
    for (uint32_t l = 0; l < e->n_layers; ++l) {
        LayerW &lw = e->w[l];
        const bool last = l + 1 == e->n_layers;
        if (cancel) {
            if (l >= 2) CTOX_CUDA(ctx, cudaEventSynchronize(L.layer_done[l & 1]));
            if (*cancel) return fail(ctx, CTOX_CANCELLED, "prefill cancelled in layer %u of a pass of %u tokens", l, m);
        }
        EX(product(e, lw.in_fan, m, &o));
        EX(mixer(e, l, o, m, pos0));
        EX(product(e, lw.out, m, &o));
        EX(rows_norm(e, m, L.h, &o, lw.post_ln, nullptr, lw.gate_up));
        EX(product(e, lw.gate_up, m, &o));
        RowsArgs a{};
        a.o = o;
        a.width = c.intermediate_size;
        EX(rows<ROWS_SWIGLU>(e, a, m, lw.down));
        EX(product(e, lw.down, m, &o));
        EX(rows_norm(e, m, L.h, &o, last ? e->final_norm : e->w[l + 1].in_ln, last ? L.final_hidden : nullptr,
                     last ? nullptr : e->w[l + 1].in_fan));
        if (cancel) CTOX_CUDA(ctx, cudaEventRecord(L.layer_done[l & 1], ctx->stream));
    }
    // What the pass leaves is committed. The last pairs stay for the next call, as many as a short pass would leave.
    const uint32_t keep = (m - 1) % kMaxPass + 1, pairs = m - keep;
    if (c.mtp_num_hidden_layers && pairs) {
        // The MTP layer over pairs (token p + 1, final hidden p): nothing reads more of it than its cache rows.
        const uint32_t X = e->n_layers;
        LayerW &lw = e->w[X];
        EX(matvec_embed_rows(e->embed, L.tokens + 1, pairs, L.h));
        RowsArgs a{};
        a.a = L.h;
        a.b = L.final_hidden;
        a.w = e->mtp_norm_e;
        a.w2 = e->mtp_norm_h;
        a.eps = c.rms_norm_epsilon;
        a.width = c.hidden_size;
        EX(rows<ROWS_MTP>(e, a, pairs, e->mtp_fc));
        EX(product(e, e->mtp_fc, pairs, &o));
        EX(rows_norm(e, pairs, nullptr, &o, lw.in_ln, nullptr, lw.in_fan));
        EX(product(e, lw.in_fan, pairs, &o, 2ull * e->q_width));
        EX(attn_pre(e, X, o, pairs, pos0 + 1, pos0, e->mtp_page_table, true));
    }
    CTOX_CUDA(ctx, cudaMemcpyAsync(e->hist_hidden, L.final_hidden + (size_t)pairs * c.hidden_size, keep * row,
                                   cudaMemcpyDeviceToDevice, ctx->stream));
    for (uint32_t j = 0; j + 1 < keep; ++j) e->hist_tokens[j] = tokens[pairs + 1 + j];
    e->hist_n = keep;
    e->have_hidden = true;
    e->position += m;
    return CTOX_OK;
}

}  // namespace ctox
