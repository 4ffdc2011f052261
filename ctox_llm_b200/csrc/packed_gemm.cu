// Product of a packed Q2 / Q4 matrix with the activations of a long pass on the fifth-generation tensor cores.
//
// What bounds it: tensor work. Every weight meets the hi and the lo part of an activation (two fp16 products, as
// in the streaming matvec), 4 m FLOPs per weight where a plain bf16 product has 2 m. Streaming the same
// weights once per eight positions, as short passes do, costs 125 passes over the matrix for 1000 positions and is
// bound by unpacking the codes each time; here a code is unpacked once per 64, 128 or 256 positions.
//
// One CTA of 16 warps per SM works through units (128 rows x N positions x a range of columns):
//   warp 0     one thread copies the activation tiles (bulk copies into a ring, hi and lo separately)
//   warp 1     one thread issues tcgen05.mma: per 64-column block lo then hi into one accumulator
//   warps 4-7  unpack codes to fp16 (code - offset, exact) and write them as the swizzled A operand
//   warps 8-15 take the 64-column sum out of tensor memory and add scale[row][block] * sum to fp32 registers
// The block scales therefore act in fp32 on sums of 64 products, exactly as in the streaming matvec: folding them
// into fp16 weights would need a second weight part (scale and code have 15 significant bits).
#include "packed_gemm.cuh"

#include <cuda_fp16.h>

#include "layout.cuh"
#include "umma.cuh"

namespace ctox {

constexpr int kPgThreads = 512;

template <uint32_t N>
struct PgCfg {
    static constexpr uint32_t kB = N == 256 ? 5 : N == 128 ? 8 : 12;  // activation tiles in the ring
    static constexpr uint32_t kA = N == 256 ? 3 : 4;                  // weight tiles
    static constexpr uint32_t kD = N == 256 ? 2 : 4;                  // accumulators in tensor memory
    static constexpr uint32_t kBBytes = N * 128, kABytes = 128 * 128;
    static constexpr uint32_t kSmem = kB * kBBytes + kA * kABytes + 1024;
};

struct PgParams {
    const uint8_t *w, *x;
    const float *unit, *s_out;
    float *y;
    size_t split_stride;
    uint32_t rows, rt0, units, m, pos_pad, pos_tiles, pairs, kst, kst_s, splits;
    int32_t *error_word;
};

__device__ __forceinline__ uint32_t pg_sub(uint32_t v, uint32_t offset) {
    const __half2 r = __hsub2(*reinterpret_cast<const __half2 *>(&v), *reinterpret_cast<const __half2 *>(&offset));
    return *reinterpret_cast<const uint32_t *>(&r);
}
__device__ __forceinline__ void pg_store(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// Codes to fp16: the code bits become mantissa bits of a power of two large enough that a step is 1, and the
// same power plus the offset is subtracted: code - 7.5 (Q4) or code - 1.5 (Q2), exact.
// Eight Q4 codes -> one 16-byte chunk, columns (0,4)(1,5)(2,6)(3,7).
__device__ __forceinline__ void pg_q4(uint32_t addr, uint32_t w) {
    constexpr uint32_t kM = 0x00f000f0u, kE = 0x54005400u, kO = 0x54785478u;  // 64, 71.5
    pg_store(addr, pg_sub(((w << 4) & kM) | kE, kO), pg_sub((w & kM) | kE, kO), pg_sub(((w >> 4) & kM) | kE, kO),
             pg_sub(((w >> 8) & kM) | kE, kO));
}
// Sixteen Q2 codes -> two chunks, columns (0,8)(1,9)...(7,15).
__device__ __forceinline__ void pg_q2(uint32_t addr0, uint32_t addr1, uint32_t w) {
    constexpr uint32_t kM2 = 0x000c000cu, kM4 = 0x00300030u, kM6 = 0x00c000c0u, kM8 = 0x03000300u;
    constexpr uint32_t kE2 = 0x5c005c00u, kE4 = 0x54005400u, kE6 = 0x4c004c00u, kE8 = 0x44004400u;  // 256, 64, 16, 4
    constexpr uint32_t kO2 = 0x5c065c06u, kO4 = 0x54185418u, kO6 = 0x4c604c60u, kO8 = 0x45804580u;  // the same + 1.5
    const uint32_t t = w >> 8;
    pg_store(addr0, pg_sub(((w << 2) & kM2) | kE2, kO2), pg_sub((w & kM2) | kE2, kO2), pg_sub((w & kM4) | kE4, kO4),
             pg_sub((w & kM6) | kE6, kO6));
    pg_store(addr1, pg_sub((w & kM8) | kE8, kO8), pg_sub((t & kM2) | kE2, kO2), pg_sub((t & kM4) | kE4, kO4),
             pg_sub((t & kM6) | kE6, kO6));
}

// A unit of work: rows rt * 128 .., positions n0 .., super-tiles ks0 .. ks1 (256 columns each), partial sum sp.
struct PgUnit {
    uint32_t rt, n0, sp, ks0, ks1;
};
template <uint32_t N>
__device__ __forceinline__ PgUnit pg_unit(const PgParams &p, uint32_t u) {
    // positions fastest: the CTAs that read the same weights run side by side
    const uint32_t v = u / p.pos_tiles, sp = v % p.splits;
    return PgUnit{p.rt0 + v / p.splits, (u % p.pos_tiles) * N, sp, (uint32_t)((uint64_t)p.kst * sp / p.splits),
                  (uint32_t)((uint64_t)p.kst * (sp + 1) / p.splits)};
}
// Super-tile `tile` (0, 1) of row pair `pair` at column super-tile ks.
template <int DT>
__device__ __forceinline__ const uint8_t *pg_tile(const PgParams &p, uint32_t pair, uint32_t ks, uint32_t tile) {
    const uint32_t slice = ks / p.kst_s, in = ks - slice * p.kst_s;
    return p.w + ((((size_t)slice * p.pairs + pair) * p.kst_s + in) * 2 + tile) * Fmt<DT>::kSuperTileBytes;
}

template <int DT, uint32_t N>
__global__ void __launch_bounds__(kPgThreads, 1) k_packed_gemm(const PgParams p) {
    using namespace umma;
    using C = PgCfg<N>;
    extern __shared__ uint8_t raw[];
    __shared__ __align__(8) uint64_t bars[2 * (C::kB + C::kA + C::kD) + 1];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int dead;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t b_base = (smem_addr(raw) + 1023) & ~1023u, a_base = b_base + C::kB * C::kBBytes;
    const uint32_t b_full = smem_addr(bars), b_empty = b_full + C::kB * 8, a_full = b_empty + C::kB * 8,
                   a_empty = a_full + C::kA * 8, d_full = a_empty + C::kA * 8, d_empty = d_full + C::kD * 8,
                   drained = d_empty + C::kD * 8;
    constexpr uint32_t kCols = C::kD * N;
    if (tid == 0) {
        dead = 0;
        for (uint32_t i = 0; i < C::kB; ++i) {
            bar_init(b_full + i * 8, 1);
            bar_init(b_empty + i * 8, 1);
        }
        for (uint32_t i = 0; i < C::kA; ++i) {
            bar_init(a_full + i * 8, 4);
            bar_init(a_empty + i * 8, 1);
        }
        for (uint32_t i = 0; i < C::kD; ++i) {
            bar_init(d_full + i * 8, 1);
            bar_init(d_empty + i * 8, 8);
        }
        bar_init(drained, 1);
        bar_init_fence();
    }
    if (warp == 1) tmem_alloc(smem_addr(&tmem_slot), kCols);
    fence_before();
    __syncthreads();
    fence_after();
    pdl_launch();  // after the allocation (umma.cuh)
    const uint32_t tmem = tmem_slot;
    if (warp < 4) {
        // N = 256 keeps 128 sums per accumulating thread: those warps take registers from these. The launch has
        // 512 x 128 registers; 128 x (56 + 96) + 256 x 176 = 64512 of its 65536 are asked for.
        if constexpr (N == 256) asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        if (warp == 0 && lane == 0) {
            pdl_wait();
            asm volatile("fence.proxy.async;" ::: "memory");  // the kernel before wrote x with ordinary stores
            uint32_t issued = 0;
            bool ok = true;
            for (uint32_t u = blockIdx.x; u < p.units && ok; u += gridDim.x) {
                const PgUnit t = pg_unit<N>(p, u);
                const uint8_t *src = p.x + ((size_t)t.ks0 * 8 * p.pos_pad + t.n0) * 128;
                const size_t part = (size_t)p.pos_pad * 128;
                for (uint32_t i = 0; i < (t.ks1 - t.ks0) * 8; ++i, ++issued) {
                    const uint32_t s = issued % C::kB, round = issued / C::kB;
                    if (round > 0 && !(ok = bar_wait(b_empty + s * 8, (round - 1) & 1, &dead))) break;
                    bar_expect(b_full + s * 8, C::kBBytes);
                    asm volatile(
                        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                            b_base + s * C::kBBytes),
                        "l"(src + (size_t)(i ^ 1) * part), "r"(C::kBBytes), "r"(b_full + s * 8)  // lo, hi, lo, hi ...
                        : "memory");
                }
            }
            if (!ok) {  // leave no copy in flight behind
                for (uint32_t s = 0; s < C::kB && s < issued; ++s) {
                    const uint32_t i = issued - 1 - s;
                    bar_drain(b_full + (i % C::kB) * 8, (i / C::kB) & 1);
                }
            }
        } else if (warp == 1 && lane == 0) {
            uint32_t used_b = 0, used_a = 0;
            bool ok = true;
            constexpr uint32_t idesc = (1u << 4) | ((N >> 3) << 17) | ((128u >> 4) << 24);  // fp16 x fp16 -> fp32
            for (uint32_t u = blockIdx.x; u < p.units && ok; u += gridDim.x) {
                const PgUnit t = pg_unit<N>(p, u);
                for (uint32_t k = 0; k < (t.ks1 - t.ks0) * 4; ++k, ++used_a) {
                    const uint32_t a = used_a % C::kA, d = used_a % C::kD;
                    if (used_a >= C::kD && !(ok = bar_wait(d_empty + d * 8, (used_a / C::kD - 1) & 1, &dead))) break;
                    if (!(ok = bar_wait(a_full + a * 8, (used_a / C::kA) & 1, &dead))) break;
                    for (uint32_t part = 0; part < 2; ++part, ++used_b) {
                        const uint32_t b = used_b % C::kB;
                        if (!(ok = bar_wait(b_full + b * 8, (used_b / C::kB) & 1, &dead))) break;
                        fence_after();
                        const uint64_t da = smem_desc(a_base + a * C::kABytes, 128), db = smem_desc(b_base + b * C::kBBytes, 128);
#pragma unroll
                        for (uint32_t i = 0; i < 4; ++i) mma_f16(tmem + d * N, da + i * 2, db + i * 2, idesc, part > 0 || i > 0);
                        commit(b_empty + b * 8);
                    }
                    if (!ok) break;
                    commit(a_empty + a * 8);
                    commit(d_full + d * 8);
                }
            }
            if (!ok) {
                commit(drained);
                bar_drain(drained, 0);
            }
        }
    } else if (warp < 8) {
        if constexpr (N == 256) asm volatile("setmaxnreg.dec.sync.aligned.u32 96;");
        // Weights do not depend on earlier kernels: no dependency wait. Warp w takes row pair w of the tile; the
        // codes of the super-tile after this one are on their way while this one is unpacked.
        const uint32_t w4 = warp - 4, g = lane >> 2, t4 = lane & 3;
        constexpr uint32_t kVec = DT == 1 ? 4 : 2;
        uint4 q[2][kVec];
        uint32_t used = 0;
        bool ok = true;
        auto load = [&](const uint8_t *base, bool live, uint32_t tile, uint32_t j) {
            q[tile][j] = live ? __ldg(reinterpret_cast<const uint4 *>(base + tile * Fmt<DT>::kSuperTileBytes + kScaleBytes +
                                                                     j * 512 + lane * 16))
                              : make_uint4(0, 0, 0, 0);
        };
        for (uint32_t u = blockIdx.x; u < p.units && ok; u += gridDim.x) {
            const PgUnit t = pg_unit<N>(p, u);
            const uint32_t pair = t.rt * 4 + w4;
            const bool live = pair < p.pairs;
            if (used == 0) {
                const uint8_t *first = pg_tile<DT>(p, live ? pair : 0, t.ks0, 0);
#pragma unroll
                for (uint32_t j = 0; j < kVec; ++j) {
                    load(first, live, 0, j);
                    load(first, live, 1, j);
                }
            }
            for (uint32_t ks = t.ks0; ks < t.ks1 && ok; ++ks) {
                // the super-tile after this one: of this unit, or the first of the next
                bool next_live = live;
                const uint8_t *next;
                if (ks + 1 < t.ks1) {
                    next = pg_tile<DT>(p, live ? pair : 0, ks + 1, 0);
                } else if (u + gridDim.x < p.units) {
                    const PgUnit n = pg_unit<N>(p, u + gridDim.x);
                    next_live = n.rt * 4 + w4 < p.pairs;
                    next = pg_tile<DT>(p, next_live ? n.rt * 4 + w4 : 0, n.ks0, 0);
                } else {
                    next_live = false;
                    next = p.w;
                }
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j, ++used) {
                    const uint32_t a = used % C::kA;
                    if (used >= C::kA && !__all_sync(0xffffffffu, bar_wait(a_empty + a * 8, (used / C::kA - 1) & 1, &dead))) {
                        ok = false;
                        break;
                    }
                    const uint32_t row = a_base + a * C::kABytes + (w4 * 32 + g) * 128;
                    const uint32_t c0 = ((2 * t4) ^ g) * 16, c1 = ((2 * t4 + 1) ^ g) * 16;
#pragma unroll
                    for (uint32_t tile = 0; tile < 2; ++tile) {
                        const uint32_t r0 = row + tile * 16 * 128, r1 = r0 + 8 * 128;
                        if constexpr (DT == 1) {
                            const uint4 v = q[tile][j];
                            pg_q4(r0 + c0, v.x);
                            pg_q4(r0 + c1, v.y);
                            pg_q4(r1 + c0, v.z);
                            pg_q4(r1 + c1, v.w);
                            load(next, next_live, tile, j);
                        } else {
                            const uint4 v = q[tile][j >> 1];
                            pg_q2(r0 + c0, r0 + c1, (j & 1) ? v.z : v.x);
                            pg_q2(r1 + c0, r1 + c1, (j & 1) ? v.w : v.y);
                            if (j & 1) load(next, next_live, tile, j >> 1);
                        }
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) bar_arrive(a_full + a * 8);
                }
            }
        }
    } else {
        if constexpr (N == 256) asm volatile("setmaxnreg.inc.sync.aligned.u32 176;");
        pdl_wait();
        const uint32_t quarter = warp & 3, half = (warp - 8) >> 2;  // tensor-memory lanes and columns of this warp
        const uint32_t src = tmem + half * (N / 2) + ((quarter * 32) << 16);
        uint32_t used = 0;
        bool ok = true;
        for (uint32_t u = blockIdx.x; u < p.units && ok; u += gridDim.x) {
            const PgUnit t = pg_unit<N>(p, u);
            const uint32_t pair = t.rt * 4 + quarter, row = t.rt * 128 + quarter * 32 + lane;
            const bool live = pair < p.pairs;
            // scales of this row: four fp16 per super-tile
            const uint32_t sc_off = (lane & 7) * 16 + ((lane >> 3) & 1) * 8;
            auto scales = [&](uint32_t ks) {
                return live && ks < t.ks1
                           ? __ldg(reinterpret_cast<const uint2 *>(pg_tile<DT>(p, pair, ks, lane >> 4) + sc_off))
                           : make_uint2(0, 0);
            };
            float acc[N / 2];
#pragma unroll
            for (uint32_t i = 0; i < N / 2; ++i) acc[i] = 0.f;
            uint2 sc = scales(t.ks0);
            for (uint32_t ks = t.ks0; ks < t.ks1 && ok; ++ks) {
                const uint2 sc_next = scales(ks + 1);
#pragma unroll 1
                for (uint32_t j = 0; j < 4; ++j, ++used) {
                    const uint32_t d = used % C::kD;
                    if (!__all_sync(0xffffffffu, bar_wait(d_full + d * 8, (used / C::kD) & 1, &dead))) {
                        ok = false;
                        break;
                    }
                    fence_after();
                    const uint32_t word = j & 2 ? sc.y : sc.x;
                    const float s = __half2float(__ushort_as_half((uint16_t)(j & 1 ? word >> 16 : word & 0xffff)));
#pragma unroll
                    for (uint32_t c = 0; c < N / 2; c += 32) {
                        float v[32];
                        tmem_ld32(src + d * N + c, v);
                        tmem_ld_wait();
#pragma unroll
                        for (uint32_t i = 0; i < 32; ++i) acc[c + i] = fmaf(s, v[i], acc[c + i]);
                    }
                    fence_before();
                    __syncwarp();
                    if (lane == 0) bar_arrive(d_empty + d * 8);
                }
                sc = sc_next;
            }
            if (ok && row < p.rows) {
                const float so = (p.s_out ? p.s_out[row] : 1.0f) * code_unit(DT);
                const uint32_t n0 = t.n0 + half * (N / 2);
                float *y = p.y + t.sp * p.split_stride + (size_t)n0 * p.rows + row;
#pragma unroll
                for (uint32_t i = 0; i < N / 2; ++i)
                    if (n0 + i < p.m) y[(size_t)i * p.rows] = acc[i] * p.unit[n0 + i] * so;
            }
        }
    }
    __syncwarp();
    __syncthreads();
    if (warp == 1) {
        fence_after();
        tmem_free(tmem, kCols);
    }
    if (tid == 0 && dead) *p.error_word = DEV_ERR_WAIT_TIMEOUT;
}

namespace {

template <int DT, uint32_t N>
ctox_status pg_launch(ctox_ctx *ctx, const PgParams &p) {
    if constexpr (N == 256) {  // the register split in the kernel counts on 128 per thread at launch
        cudaFuncAttributes attr;
        CTOX_CUDA(ctx, cudaFuncGetAttributes(&attr, k_packed_gemm<DT, N>));
        if (attr.numRegs != 128) return fail(ctx, CTOX_INVALID_STATE, "packed product: built with %d registers", attr.numRegs);
    }
    CTOX_CUDA(ctx, cudaFuncSetAttribute(k_packed_gemm<DT, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PgCfg<N>::kSmem));
    const uint32_t grid = p.units < (uint32_t)ctx->sm_count ? p.units : (uint32_t)ctx->sm_count;
    CTOX_CUDA(ctx, launch_pdl(k_packed_gemm<DT, N>, dim3(grid), dim3(kPgThreads), PgCfg<N>::kSmem, ctx->stream, p));
    return CTOX_OK;
}

}  // namespace

ctox_status launch_packed_gemm(ctox_matvec *mv, const LongIn &in, uint32_t m, uint64_t row0, uint64_t row_end, float *y,
                               size_t capacity, LongOut *out) {
    ctox_ctx *ctx = mv->ctx;
    const MatvecPart &part = mv->parts[0];
    if (mv->parts.size() != 1 || m == 0 || m > in.pos_pad || in.pos_pad % kLongPosTile || row_end > mv->rows ||
        (size_t)m * mv->rows > capacity)
        return fail(ctx, CTOX_SHAPE, "packed product: %u positions of a %llu-row matrix", m, (unsigned long long)mv->rows);
    PgParams p{};
    p.w = part.prep;
    p.x = in.x;
    p.unit = in.unit;
    p.s_out = mv->s_out;
    p.y = y;
    p.rows = (uint32_t)mv->rows;
    p.split_stride = (size_t)m * mv->rows;
    p.rt0 = (uint32_t)(row0 / 128);
    p.m = m;
    p.pos_pad = in.pos_pad;
    p.pairs = part.pairs;
    p.kst_s = part.kst_s;
    p.kst = part.kst_s * part.slices;
    p.error_word = ctx->dev_error;
    const uint32_t row_tiles = (uint32_t)((row_end + 127) / 128) - p.rt0;
    // Tile width and column split by the time of the longest chain of units on an SM: a 64-column block takes
    // `step` (measured, in units of a block of 256 positions), a unit `start` more for filling its pipeline and
    // writing its sums. A split is only as good as the extra partial sums its consumer reads.
    uint32_t best_n = 0;
    double best = 1e30;
    for (uint32_t n : {64u, 128u, 256u}) {
        const double step = n == 256 ? 1.0 : n == 128 ? 0.6 : 0.4, start = n == 256 ? 6.0 : n == 128 ? 5.0 : 4.0;
        const uint32_t tiles = (m + n - 1) / n;
        for (uint32_t s = 1; s <= p.kst && s <= 16 && s * p.split_stride <= capacity; ++s) {
            const uint32_t units = row_tiles * tiles * s, rounds = (units + ctx->sm_count - 1) / ctx->sm_count;
            const double cost = rounds * (((p.kst + s - 1) / s) * 4 * step + start) + (s - 1) * 2.0;
            if (cost < best) {
                best = cost;
                best_n = n;
                p.splits = s;
            }
        }
    }
    p.pos_tiles = (m + best_n - 1) / best_n;
    p.units = row_tiles * p.pos_tiles * p.splits;
    timing_begin(ctx);
    if (part.dt)
        EX(best_n == 256 ? (pg_launch<1, 256>(ctx, p)) : best_n == 128 ? (pg_launch<1, 128>(ctx, p)) : (pg_launch<1, 64>(ctx, p)));
    else
        EX(best_n == 256 ? (pg_launch<0, 256>(ctx, p)) : best_n == 128 ? (pg_launch<0, 128>(ctx, p)) : (pg_launch<0, 64>(ctx, p)));
    timing_end(ctx, KC_GEMM, (double)part.prep_bytes + 4.0 * m * ((double)mv->columns + mv->rows),
               2.0 * (double)(row_end - row0) * (double)mv->columns * m);
    *out = LongOut{y, p.rows, p.splits, p.split_stride};
    return CTOX_OK;
}

}  // namespace ctox
