// Attention of the hybrid model over the paged bf16 cache on the fifth-generation tensor cores: head dimension 256, up to 32 query rows
// (heads of a key/value head x positions) per CTA, one part of the context per CTA.
//
// What bounds it: HBM (64 KB of keys and values per 64 tokens and head). mma.sync kept 16 x 256 sums in the registers of every warp and
// left its chain of products, softmax and products exposed: 55 us for 134 MB at four positions, 48 at one. Here the sums stand in
// tensor memory and the roles overlap: 40 and 36 us, 3.4 and 3.7 TB/s (each without overlap with the kernels around it).
//   two warps each   copy 64-token tiles of keys and of values (16-byte cp.async, rows of 64 dimensions, 128-byte swizzle) into rings of
//                    three, the values' of two beside 32 queries; tiles of earlier passes' tokens ahead of the dependency wait
//   one warp         issues tcgen05.mma: scores^T [64 tokens x queries] = K Q^T, the queries' bf16 hi and lo parts side by side,
//                    and output^T [256 x queries] += V^T P^T, V as it lies in the cache (rows along the tokens), P hi then lo
//   eight warps      softmax: a token per lane (the scores' 64 lanes of tensor memory belong to warps 0 and 1 of every four), a quarter
//                    of the queries per warp. The reference of a query moves only when a score exceeds it by 2^8 (as in
//                    stack_prefill.cu), so that the maxima are formed in a few tiles alone (with a maximum per query and tile,
//                    and half of the queries per warp, 56 us)
//   warps 0-3        also rescale the output when a reference moves, and store it
// Scores and weights enter the products as two bf16 parts (16 bits), the cache is exact: as in k_attention_mma.
#include "layers.cuh"
#include "umma.cuh"

#include <cuda_bf16.h>

namespace ctox {

constexpr uint32_t kAtThreads = 480, kAtTile = 64, kAtHd = 256;
constexpr uint32_t kAtMma = 14, kAtSoftWarps = 10;  // softmax: warps 0, 1 of every four; with 2 and 3 those of the output
constexpr uint32_t kAtKv = kAtTile * kAtHd * 2;                                  // bytes of a tile of keys or values
// A launch has room for 16, 24 or 32 queries: with 24 (four positions of six heads) and one buffer of weights three tiles of values
// fit. Products of 128 rows take multiples of 16 columns, so 24 queries have weights' rows and output columns for 32.
constexpr uint32_t kAtK = 3;
__host__ __device__ constexpr uint32_t at_v_stages(int nq) { return nq == 32 ? 2 : 3; }
__host__ __device__ constexpr uint32_t at_columns(int nq) { return nq == 16 ? 16 : 32; }
__host__ __device__ constexpr uint32_t at_p_buffers(int nq) { return nq == 24 ? 1 : 2; }
__host__ __device__ constexpr uint32_t at_smem(int nq) {
    return (uint32_t)nq * 2 * kAtHd * 2 + at_p_buffers(nq) * at_columns(nq) * 256 + (kAtK + at_v_stages(nq)) * kAtKv + 1024;
}

__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ bool any_of_soft(bool p) {  // a barrier of the kAtSoftWarps
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, 1, 320, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)p)
        : "memory");
    return r != 0;
}
__device__ __forceinline__ void soft_sync() { asm volatile("bar.sync 1, 320;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void at_load(uint32_t tmem, float *v) {  // 32 lanes x N columns
    if constexpr (N == 4) {
        uint32_t *r = reinterpret_cast<uint32_t *>(v);
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(tmem));
    } else if constexpr (N == 8) {
        uint32_t *r = reinterpret_cast<uint32_t *>(v);
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "r"(tmem));
    } else if constexpr (N == 16) {
        umma::tmem_ld16(tmem, v);
    } else {
        umma::tmem_ld32(tmem, v);
    }
}
template <int N>
__device__ __forceinline__ void at_store(uint32_t tmem, const float *v) {
    if constexpr (N == 16)
        umma::tmem_st16(tmem, v);
    else
        umma::tmem_st32(tmem, reinterpret_cast<const uint32_t *>(v));
}

struct AttnTensor {
    AttnGeom g;
    const float *q;
    const __nv_bfloat16 *k_cache, *v_cache;
    const uint32_t *page_table;
    uint32_t page_tokens;
    uint64_t cache_slot;
    uint32_t npos, splits;
    float *ws;
    int32_t *error_word;
};

template <int NQ>
__global__ void __launch_bounds__(kAtThreads, 1) k_attention_tensor(const __grid_constant__ AttnTensor a) {
    using namespace umma;
    constexpr uint32_t KS = kAtK, VS = at_v_stages(NQ), H = NQ / 4;  // H: queries of a softmax warp
    constexpr uint32_t NC = at_columns(NQ), PB = at_p_buffers(NQ);
    constexpr uint32_t kQBytes = NQ * 2 * kAtHd * 2, kPPart = NC * 128, kPBuf = 2 * kPPart;
    constexpr uint32_t kCols = NC == 32 ? 256 : 128, kS = 2 * NC, kO = 2 * kS;  // tensor memory: two buffers of scores, the output
    constexpr uint32_t HL = H <= 4 ? 4 : 8;                                       // columns of a load of scores
    extern __shared__ uint8_t raw[];
    __shared__ __align__(8) uint64_t bars[2 * KS + 2 * VS + 8];
    __shared__ float max_s[2][NC], alpha_s[NC], ref_s[NC], sum_s[2][NC];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int dead;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t base = (smem_addr(raw) + 1023) & ~1023u;
    const uint32_t q_s = base, p_s = q_s + kQBytes, k_s = p_s + PB * kPBuf, v_s = k_s + KS * kAtKv;
    const uint32_t k_full = smem_addr(bars), k_empty = k_full + 8 * KS, v_full = k_empty + 8 * KS, v_empty = v_full + 8 * VS,
                   s_full = v_empty + 8 * VS, p_full = s_full + 16, o_done = p_full + 16, q_full = o_done + 16, drained = q_full + 8;
    if (tid == 0) {
        dead = 0;
        for (uint32_t i = 0; i < KS; ++i) {
            bar_init(k_full + 8 * i, 2);
            bar_init(k_empty + 8 * i, 1);
        }
        for (uint32_t i = 0; i < VS; ++i) {
            bar_init(v_full + 8 * i, 2);
            bar_init(v_empty + 8 * i, 1);
        }
        for (uint32_t i = 0; i < 2; ++i) {
            bar_init(s_full + 8 * i, 1);
            bar_init(p_full + 8 * i, 8);
            bar_init(o_done + 8 * i, 1);
        }
        bar_init(q_full, kAtSoftWarps);
        bar_init(drained, 1);
        bar_init_fence();
    }
    if (warp == kAtMma) tmem_alloc(smem_addr(&tmem_slot), kCols);
    fence_before();
    __syncthreads();
    fence_after();
    pdl_launch();  // after the allocation (umma.cuh)
    const uint32_t tmem = tmem_slot;

    const AttnGeom &g = a.g;
    const uint32_t G = g.q_heads / g.kv_heads, nq = G * a.npos, kh = blockIdx.x / a.splits, sp = blockIdx.x % a.splits;
    const uint64_t slot0 = a.cache_slot, total = slot0 + a.npos, tiles = (total + kAtTile - 1) / kAtTile;
    const uint64_t tile_beg = tiles * sp / a.splits;
    const uint32_t n = (uint32_t)(tiles * (sp + 1) / a.splits - tile_beg);
    bool ok = true;

    if (warp == 6 || warp == 7 || warp == 10 || warp == 11) {
        // ---- tiles: warps 6 and 7 the keys', 10 and 11 the values'; thread (warp, lane) copies the 16-byte chunk `lane` of every
        // second row
        const uint32_t lw = warp & 1;
        const bool keys = warp < 8;
        const __nv_bfloat16 *cache = keys ? a.k_cache : a.v_cache;
        const uint32_t ring = keys ? k_s : v_s, full = keys ? k_full : v_full, empty = keys ? k_empty : v_empty, stages = keys ? KS : VS;
        const int shift = (a.page_tokens & (a.page_tokens - 1)) == 0 ? 31 - __clz(a.page_tokens) : -1;
        constexpr uint32_t kRows = kAtTile / 2;
        uint32_t slots[kRows];
        auto fetch_slots = [&](uint64_t tile) {
            if (shift >= 1 && a.page_tokens <= kAtTile) {  // a tile is 1..32 whole pages: a lookup per lane
                const uint32_t page0 = (uint32_t)(tile * kAtTile) >> shift, pages = kAtTile >> shift, last = (uint32_t)(total - 1) >> shift;
                const uint32_t mine = lane < pages && page0 + lane <= last ? a.page_table[page0 + lane] : 0;
#pragma unroll
                for (uint32_t j = 0; j < kRows; ++j) {
                    const uint32_t r = lw + 2 * j, pg = __shfl_sync(0xffffffffu, mine, r >> shift);
                    slots[j] = tile * kAtTile + r < total ? (pg << shift) + (r & (a.page_tokens - 1)) : 0xffffffffu;
                }
            } else {
#pragma unroll
                for (uint32_t j = 0; j < kRows; ++j) {
                    const uint64_t t = tile * kAtTile + lw + 2 * j;
                    slots[j] = t < total ? a.page_table[(uint32_t)t / a.page_tokens] * a.page_tokens + (uint32_t)t % a.page_tokens : 0xffffffffu;
                }
            }
        };
        const uint32_t to = (lane >> 3) * (kAtTile * 128);
        uint32_t reported = 0, st_reported = 0;  // tiles that have landed
        auto report = [&](uint32_t upto) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            for (; reported < upto; ++reported) {
                if (lane == 0) bar_arrive(full + 8 * st_reported);
                if (++st_reported == stages) st_reported = 0;
            }
        };
        bool waited = false;
        uint32_t st = 0, parity = 1;  // of the phase before the ring's first: passes at once
        if (n) fetch_slots(tile_beg);
        for (uint32_t t = 0; t < n; ++t) {
            // Tokens of earlier passes may be read ahead of the dependency wait: the kernel that appends this pass's lets no later one
            // start before all of the pass before has finished (k_attn_pre).
            if (!waited && (tile_beg + t + 1) * kAtTile > slot0) {
                pdl_wait();
                waited = true;
            }
            if (!__all_sync(0xffffffffu, bar_try(empty + 8 * st, parity))) {
                asm volatile("cp.async.wait_group 0;" ::: "memory");  // nothing else to do: report what is on its way as it lands
                report(t);
                if (!(ok = __all_sync(0xffffffffu, bar_wait(empty + 8 * st, parity, &dead)))) break;
            }
            const uint32_t buffer = ring + st * kAtKv + to;
#pragma unroll
            for (uint32_t j = 0; j < kRows; ++j) {
                const uint32_t r = lw + 2 * j, dst = buffer + r * 128 + (((lane & 7) ^ (r & 7)) * 16);
                if (slots[j] != 0xffffffffu)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst),
                                 "l"(cache + ((size_t)slots[j] * g.kv_heads + kh) * kAtHd + lane * 8)
                                 : "memory");
                else
                    asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};" ::"r"(dst), "r"(0u) : "memory");
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            if (t + 1 < n) fetch_slots(tile_beg + t + 1);
            if (stages == 3)
                asm volatile("cp.async.wait_group 2;" ::: "memory");
            else
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            if (t + 1 >= stages) report(t + 2 - stages);
            if (++st == stages) {
                st = 0;
                parity ^= 1;
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (ok) report(n);
        if (!waited) pdl_wait();
    } else if (warp == kAtMma) {
        pdl_wait();
        const bool issuer = elect_one();
        const uint32_t idesc_s = idesc_bf16(128, 2 * NQ), idesc_o = idesc_bf16_mn(128, NC, true, false);
        const uint64_t dq = smem_desc(q_s, 128), dk = smem_desc(k_s, 128), dp = smem_desc(p_s, 128);
        const uint64_t dv = smem_desc_mn(v_s, 128, kAtTile * 128);
        uint32_t ks = 0, k_par = 0, vs = 0, v_par = 0;
        // Scores of tile t. The product has 128 rows: those past the tile's 64 tokens read what lies behind it, and nothing reads them.
        auto scores = [&](uint32_t t) {
            if (!__all_sync(0xffffffffu, bar_wait(k_full + 8 * ks, k_par, &dead))) return false;
            fence_after();
            if (issuer) {
#pragma unroll
                for (uint32_t i = 0; i < 16; ++i)
                    mma_f16(tmem + (t & 1) * kS, dk + ((ks * kAtKv + (i >> 2) * (kAtTile * 128) + (i & 3) * 32) >> 4),
                            dq + (((i >> 2) * (2 * NQ * 128) + (i & 3) * 32) >> 4), idesc_s, i > 0);
                commit(k_empty + 8 * ks);
                commit(s_full + 8 * (t & 1));
            }
            __syncwarp();
            if (++ks == KS) {
                ks = 0;
                k_par ^= 1;
            }
            return true;
        };
        if (n) ok = __all_sync(0xffffffffu, bar_wait(q_full, 0, &dead)) && scores(0);
        for (uint32_t t = 0; t < n && ok; ++t) {
            if (t + 1 < n && !(ok = scores(t + 1))) break;
            ok = __all_sync(0xffffffffu, bar_wait(p_full + 8 * (t & 1), (t >> 1) & 1, &dead));
            ok = ok && __all_sync(0xffffffffu, bar_wait(v_full + 8 * vs, v_par, &dead));
            if (!ok) break;
            fence_after();
            if (issuer) {
#pragma unroll
                for (uint32_t h = 0; h < 2; ++h)
#pragma unroll
                    for (uint32_t i = 0; i < 8; ++i)  // 16 tokens of the hi, then of the lo part
                        mma_f16(tmem + kO + h * NC, dv + ((vs * kAtKv + h * 2 * (kAtTile * 128) + (i >> 1) * 2048) >> 4),
                                dp + ((t % PB * kPBuf + (i & 1) * kPPart + (i >> 1) * 32) >> 4), idesc_o, t > 0 || i > 0);
                commit(v_empty + 8 * vs);
                commit(o_done + 8 * (t & 1));
            }
            __syncwarp();
            if (++vs == VS) {
                vs = 0;
                v_par ^= 1;
            }
        }
        if (!ok && issuer) {
            commit(drained);
            bar_drain(drained, 0);
        }
    } else {
        pdl_wait();
        {  // the queries, in units of log 2, as bf16 hi and lo rows
            const float scale = 1.4426950408889634f / sqrtf((float)kAtHd);
            constexpr uint32_t kThreads = kAtSoftWarps * 32, kVec = (NQ * (kAtHd / 4) + kThreads - 1) / kThreads;
            const uint32_t me = tid - (warp < 6 ? 0 : warp < 10 ? 64 : 128);
            float4 v[kVec];
#pragma unroll
            for (uint32_t j = 0; j < kVec; ++j) {
                const uint32_t i = me + j * kThreads, row = i / (kAtHd / 4), d = i % (kAtHd / 4) * 4;
                v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (row < nq) v[j] = *reinterpret_cast<const float4 *>(a.q + ((size_t)(row / G) * g.q_heads + kh * G + row % G) * kAtHd + d);
            }
#pragma unroll
            for (uint32_t j = 0; j < kVec; ++j) {
                const uint32_t i = me + j * kThreads, row = i / (kAtHd / 4), d = i % (kAtHd / 4) * 4;
                if (row >= NQ) continue;
                const float x[4] = {v[j].x * scale, v[j].y * scale, v[j].z * scale, v[j].w * scale};
                __nv_bfloat162 hi[2], lo[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    hi[k] = __floats2bfloat162_rn(x[2 * k], x[2 * k + 1]);
                    lo[k] = __floats2bfloat162_rn(x[2 * k] - __bfloat162float(hi[k].x), x[2 * k + 1] - __bfloat162float(hi[k].y));
                }
#pragma unroll
                for (uint32_t part = 0; part < 2; ++part) {
                    const uint32_t r = part * NQ + row;
                    const uint32_t at = q_s + (d >> 6) * (2 * NQ * 128) + r * 128 + (((d >> 3 & 7) ^ (r & 7)) * 16) + (d & 7) * 2;
                    const uint32_t *w = reinterpret_cast<const uint32_t *>(part ? lo : hi);
                    asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(at), "r"(w[0]), "r"(w[1]) : "memory");
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) bar_arrive(q_full);
        }
        const bool soft = (warp & 2) == 0;
        const uint32_t row0 = (warp >> 2) * H, part = warp & 1;  // queries row0 .., tokens part * 32 ..
        const uint32_t lanes = ((warp & 3) * 32) << 16, tok = part * 32 + lane;
        float ref[H], limit[H], sum[H];  // limit: the score beyond which the reference moves (-inf: there is none yet)
        uint32_t p_at[H];
#pragma unroll
        for (uint32_t i = 0; i < H; ++i) {
            ref[i] = sum[i] = 0.f;
            limit[i] = -INFINITY;
            p_at[i] = p_s + (row0 + i) * 128 + (((tok >> 3) ^ ((row0 + i) & 7)) * 16) + (tok & 7) * 2;
        }
        for (uint32_t t = 0; t < n; ++t) {
            float s[HL];
            bool move = false;
            if (soft) {
                ok = __all_sync(0xffffffffu, ok && bar_wait(s_full + 8 * (t & 1), (t >> 1) & 1, &dead));
                fence_after();
                float lo[HL];
                const uint32_t src = tmem + lanes + (t & 1) * kS + row0;
                at_load<HL>(src, s);
                at_load<HL>(src + NQ, lo);
                tmem_ld_wait();
                const uint64_t token = (tile_beg + t) * kAtTile + tok;
                const bool whole = (tile_beg + t + 1) * kAtTile <= slot0 + 1;  // every query sees all of the tile
#pragma unroll
                for (uint32_t i = 0; i < H; ++i) s[i] = fmaxf(s[i] + lo[i], -INFINITY);  // NaN: no weight, as in k_attention_mma
                if (!whole)
#pragma unroll
                    for (uint32_t i = 0; i < H; ++i)
                        if (token > slot0 + (row0 + i < nq ? (row0 + i) / G : 0)) s[i] = -INFINITY;
#pragma unroll
                for (uint32_t i = 0; i < H; ++i) move |= s[i] > limit[i];
            }
            if (any_of_soft(move)) {
                if (soft)
#pragma unroll
                    for (uint32_t i = 0; i < H; ++i) {
                        const float mx = warp_max(s[i]);
                        if (lane == 0) max_s[part][row0 + i] = mx;
                    }
                soft_sync();
                if (soft) {
#pragma unroll
                    for (uint32_t i = 0; i < H; ++i) {
                        const float mx = fmaxf(max_s[0][row0 + i], max_s[1][row0 + i]);
                        const bool fresh = limit[i] == -INFINITY;
                        float f = 1.0f;
                        if (mx > -INFINITY && (fresh || mx > ref[i])) {
                            if (!fresh) f = exp2f(ref[i] - mx);  // else nothing has been added yet
                            ref[i] = mx;
                            limit[i] = mx + 8.0f;
                        }
                        sum[i] *= f;
                        if (part == 0 && lane == 0) alpha_s[row0 + i] = f;
                    }
                }
                soft_sync();
                if (t > 0 && warp < 4) {
                    ok = __all_sync(0xffffffffu, ok && bar_wait(o_done + 8 * ((t - 1) & 1), ((t - 1) >> 1) & 1, &dead));
                    fence_after();
                    if (ok)
#pragma unroll
                        for (uint32_t h = 0; h < 2; ++h) {
                            float o[NC];
                            at_load<NC>(tmem + lanes + kO + h * NC, o);
                            tmem_ld_wait();
#pragma unroll
                            for (uint32_t i = 0; i < NQ; ++i) o[i] *= alpha_s[i];
                            at_store<NC>(tmem + lanes + kO + h * NC, o);
                        }
                    tmem_st_wait();
                    fence_before();
                }
                soft_sync();
            }
            if (soft) {
                // the weights' buffer: the product that read it last (of two tiles ago, or one) has finished
                if (t >= PB) ok = __all_sync(0xffffffffu, ok && bar_wait(o_done + 8 * ((t - PB) & 1), ((t - PB) >> 1) & 1, &dead));
                const uint32_t buffer = t % PB * kPBuf;
#pragma unroll
                for (uint32_t i = 0; i < H; ++i) {
                    const float p = ex2(s[i] - ref[i]);
                    sum[i] += p;
                    const __nv_bfloat16 hi = __float2bfloat16_rn(p), lo = __float2bfloat16_rn(p - __bfloat162float(hi));
                    const uint32_t at = p_at[i] + buffer;
                    asm volatile("st.shared.b16 [%0], %1;" ::"r"(at), "h"(__bfloat16_as_ushort(hi)) : "memory");
                    asm volatile("st.shared.b16 [%0], %1;" ::"r"(at + kPPart), "h"(__bfloat16_as_ushort(lo)) : "memory");
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                fence_before();
                __syncwarp();
                if (lane == 0 && ok) bar_arrive(p_full + 8 * (t & 1));
            }
        }
        // ---- output of this part of the context: [query][256 sums, maximum, sum of weights]
        if (soft) {
#pragma unroll
            for (uint32_t i = 0; i < H; ++i) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], o);
                if (lane == 0) {
                    sum_s[part][row0 + i] = sum[i];
                    if (part == 0) ref_s[row0 + i] = limit[i] == -INFINITY ? -INFINITY : ref[i];
                }
            }
        }
        if (n) ok = __all_sync(0xffffffffu, ok && bar_wait(o_done + 8 * ((n - 1) & 1), ((n - 1) >> 1) & 1, &dead));
        fence_after();
        soft_sync();
        float *out = a.ws + (size_t)(kh * a.splits + sp) * nq * (kAtHd + 2);
        if (warp < 4) {
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
                float o[NC];
                at_load<NC>(tmem + lanes + kO + h * NC, o);
                tmem_ld_wait();
#pragma unroll
                for (uint32_t i = 0; i < NQ; ++i)
                    if (i < nq) out[(size_t)i * (kAtHd + 2) + h * 128 + warp * 32 + lane] = n ? o[i] : 0.f;
            }
        } else if (warp == 4 && lane < nq) {
            out[(size_t)lane * (kAtHd + 2) + kAtHd] = ref_s[lane] * 0.6931471805599453f;
            out[(size_t)lane * (kAtHd + 2) + kAtHd + 1] = sum_s[0][lane] + sum_s[1][lane];
        }
        if (!ok && lane == 0) atomicExch(a.error_word, DEV_ERR_WAIT_TIMEOUT);
    }
    fence_before();
    __syncthreads();
    fence_after();
    if (warp == kAtMma) tmem_free(tmem, kCols);
}

void launch_attention_tensor(cudaStream_t st, const AttnGeom &g, const float *q, const void *k_cache, const void *v_cache,
                             const uint32_t *page_table, uint32_t page_tokens, uint64_t cache_slot, uint32_t m, uint32_t splits,
                             float *workspace) {
    const AttnTensor a{g, q, (const __nv_bfloat16 *)k_cache, (const __nv_bfloat16 *)v_cache, page_table, page_tokens, cache_slot, m, splits,
                       workspace, g.error_word};
    static thread_local unsigned long long ready = 0;  // devices on which the kernels may use their shared memory
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 64 && !(ready >> dev & 1ull) &&
        cudaFuncSetAttribute(k_attention_tensor<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)at_smem(16)) == cudaSuccess &&
        cudaFuncSetAttribute(k_attention_tensor<24>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)at_smem(24)) == cudaSuccess &&
        cudaFuncSetAttribute(k_attention_tensor<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)at_smem(32)) == cudaSuccess)
        ready |= 1ull << dev;
    const dim3 grid(g.kv_heads * splits);
    const uint32_t nq = g.q_heads / g.kv_heads * m;
    if (nq <= 16)
        launch_pdl(k_attention_tensor<16>, grid, dim3(kAtThreads), at_smem(16), st, a);
    else if (nq <= 24)
        launch_pdl(k_attention_tensor<24>, grid, dim3(kAtThreads), at_smem(24), st, a);
    else
        launch_pdl(k_attention_tensor<32>, grid, dim3(kAtThreads), at_smem(32), st, a);
}

}  // namespace ctox
