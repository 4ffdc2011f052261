// Product of a packed Q2 / Q4 matrix with the activations of a long pass on the fifth-generation tensor cores.
//
// What bounds it: tensor work. Every weight meets the hi and the lo part of an activation (two fp16 products, as
// in the streaming matvec), 4 m FLOPs per weight where a plain bf16 product has 2 m. Streaming the same
// weights once per eight positions, as short passes do, costs 125 passes over the matrix for 1000 positions and is
// bound by unpacking the codes each time; here a code is unpacked once per up to 256 positions.
//
// A CTA of 16 warps per SM works through units (128 rows x n positions x a range of columns):
//   warp 0     one thread copies the activation tiles (bulk copies, hi and lo parts)
//   warp 1     issues tcgen05.mma: per 64-column block lo then hi into one accumulator
//   warp 2     (second CTA of a pair) reports its stages to the first
//   warps 4-7  unpack codes to fp16 (code - offset, exact) and write them as the swizzled A operand
//   warps 8-15 take the 64-column sum out of tensor memory and add scale[row][block] * sum to fp32 registers; where a
//              position of the tile is marked (packed_gemm.cuh), scale[row][block] * unit[block][position] * sum, which
//              takes a third longer (999 positions of a 9088 x 5056 and a 5056 x 4544 product, all marked: 497 against 376 us)
// The block scales therefore act in fp32 on sums of 64 products, exactly as in the streaming matvec: folding them
// into fp16 weights would need a second weight part (scale and code have 15 significant bits).
//
// Tiles of more than 128 positions are computed by pairs of CTAs (cta_group::2, 256 rows): each copies half of the
// positions, which halves what every SM draws from L2 (64 KB per block of 256 positions, 9.7 TB/s over the chip, bound
// the single-CTA form at 1.01 us a block; a pair takes 0.90). Then the accumulators bound it: with two of 256 columns,
// products wait for sums to be taken out (two thirds of the tensor time is used). 34816 x 5120 (Q2), 999
// positions: 573 us, 621 TFLOP/s of a plain product, twice that counting both parts.
#include "packed_gemm.cuh"

#include <cuda_fp16.h>

#include <type_traits>

#include "layout.cuh"
#include "umma.cuh"

namespace ctox {

constexpr int kPgThreads = 512;

// W: widest position tile of the kernel; G: CTAs that share a tile. A launch takes n <= W positions per tile (a
// multiple of 16 G) and as many stages (weights of 128 rows, activations of n / G positions) as fit.
template <uint32_t W, uint32_t G>
struct PgCfg {
    static constexpr uint32_t kD = W == 256 ? 2 : 4;  // accumulators in tensor memory
    static constexpr uint32_t kABytes = 128 * 128;
};
constexpr uint32_t kPgStages = 6;

struct PgParams {
    const uint8_t *w, *x;
    const float *unit, *block_unit, *s_out;
    const uint8_t *spread;
    float *y;
    size_t split_stride;
    uint32_t rows, rt0, units, m, pos_pad, pos_tiles, n, stages, pairs, kst, kst_s, splits;
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

// acc[0..1] += s * v[0..1]
__device__ __forceinline__ void pg_fma2(float *acc, float s, const float *v) {
    asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 b, {%2, %2};\n\tmov.b64 c, {%3, %4};\n\t"
        "fma.rn.f32x2 a, b, c, a;\n\tmov.b64 {%0, %1}, a;\n\t}"
        : "+f"(acc[0]), "+f"(acc[1])
        : "f"(s), "f"(v[0]), "f"(v[1]));
}

// A unit of work: rows rt * 128 .., positions n0 .., super-tiles ks0 .. ks1 (256 columns each), partial sum sp.
struct PgUnit {
    uint32_t rt, n0, sp, ks0, ks1;
};
__device__ __forceinline__ PgUnit pg_unit(const PgParams &p, uint32_t u) {
    // positions fastest: the CTAs that read the same weights run side by side
    const uint32_t v = u / p.pos_tiles, sp = v % p.splits;
    return PgUnit{p.rt0 + v / p.splits, (u % p.pos_tiles) * p.n, sp, (uint32_t)((uint64_t)p.kst * sp / p.splits),
                  (uint32_t)((uint64_t)p.kst * (sp + 1) / p.splits)};
}
// Super-tile `tile` (0, 1) of row pair `pair` at column super-tile ks.
template <int DT>
__device__ __forceinline__ const uint8_t *pg_tile(const PgParams &p, uint32_t pair, uint32_t ks, uint32_t tile) {
    const uint32_t slice = ks / p.kst_s, in = ks - slice * p.kst_s;
    return p.w + ((((size_t)slice * p.pairs + pair) * p.kst_s + in) * 2 + tile) * Fmt<DT>::kSuperTileBytes;
}

template <int DT, uint32_t W, uint32_t G>
__global__ void __launch_bounds__(kPgThreads, 1) k_packed_gemm(const PgParams p) {
    using namespace umma;
    using C = PgCfg<W, G>;
    extern __shared__ uint8_t raw[];
    __shared__ __align__(8) uint64_t bars[2 * (kPgStages + C::kD) + 1];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int dead;
    __shared__ volatile uint32_t marked_tiles[8];
    __shared__ __align__(16) float unit_stage[8][W / 2];  // of an accumulating warp's columns
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t base = (smem_addr(raw) + 1023) & ~1023u, stages = p.stages;
    const uint32_t half_bytes = p.n / G * 128, stage_bytes = C::kABytes + 2 * half_bytes;  // A | lo | hi
    const uint32_t full = smem_addr(bars), empty = full + kPgStages * 8, d_full = empty + kPgStages * 8,
                   d_empty = d_full + C::kD * 8, drained = d_empty + C::kD * 8;
    constexpr uint32_t kCols = C::kD * W;
    const uint32_t rank = G == 2 ? cluster_rank() : 0, first_unit = blockIdx.x / G, unit_step = gridDim.x / G;
    if (tid == 0) {
        dead = 0;
        for (uint32_t i = 0; i < stages; ++i) {
            // this CTA's copies and unpacking warps; at the issuing CTA of a pair also the other's report of the same
            bar_init(full + i * 8, G == 2 && rank == 0 ? 6 : 5);
            bar_init(empty + i * 8, 1);
        }
        for (uint32_t i = 0; i < C::kD; ++i) {
            bar_init(d_full + i * 8, 1);
            bar_init(d_empty + i * 8, 8 * G);
        }
        bar_init(drained, 1);
        bar_init_fence();
    }
    if (warp == 1) {
        if constexpr (G == 2)
            tmem_alloc_pair(smem_addr(&tmem_slot), kCols);
        else
            tmem_alloc(smem_addr(&tmem_slot), kCols);
    }
    fence_before();
    __syncthreads();
    if constexpr (G == 2) cluster_sync();  // the other CTA's barriers are ready
    fence_after();
    pdl_launch();  // after the allocation (umma.cuh)
    const uint32_t tmem = tmem_slot;
    if (warp < 4) {
        // Wide tiles keep up to 128 sums per accumulating thread beside 64 values on their way: those warps take
        // registers from these. The launch has 512 x 128; 128 x (32 + 64) + 256 x 208 = 65536 are asked for.
        if constexpr (W > 64) asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
        if (warp == 0 && lane == 0) {
            pdl_wait();
            asm volatile("fence.proxy.async;" ::: "memory");  // the kernel before wrote x with ordinary stores
            uint32_t st = 0, parity = 1;  // parity of the phase before a ring's first: passes at once
            bool ok = true;
            const size_t part = (size_t)p.pos_pad * 128;
            for (uint32_t u = first_unit; u < p.units && ok; u += unit_step) {
                const PgUnit t = pg_unit(p, u);
                const uint8_t *src = p.x + (size_t)t.ks0 * 8 * part + (size_t)(t.n0 + rank * (p.n / G)) * 128;
                for (uint32_t i = (t.ks1 - t.ks0) * 4; i > 0; --i) {
                    const uint32_t bar = full + st * 8, dst = base + st * stage_bytes + C::kABytes;
                    if (!(ok = bar_wait(empty + st * 8, parity, &dead))) break;
                    bar_expect(bar, 2 * half_bytes);
#pragma unroll
                    for (uint32_t h = 0; h < 2; ++h)
                        asm volatile(
                            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                dst + h * half_bytes),
                            "l"(src + (h ? 0 : part)), "r"(half_bytes), "r"(bar)
                            : "memory");
                    src += 2 * part;
                    if (++st == stages) {
                        st = 0;
                        parity ^= 1;
                    }
                }
            }
            if (!ok) {  // leave no copy in flight behind: a phase lacks other arrivals, so wait for the data as such
                const long long t0 = clock64();
                while (clock64() - t0 < 2000000) {
                }
            }
        } else if (warp == 1) {
            // One thread feeds the tensor cores: 8 products and 4 commits per block. The whole warp runs the loop, so that
            // its values are uniform and descriptors need no moves between register files; ring positions are kept, not
            // divided out.
            const bool issuer = elect_one();
            uint32_t st = 0, parity = 0, d = 0, d_par = 1;
            bool ok = true;
            const uint32_t idesc = (1u << 4) | ((p.n >> 3) << 17) | ((128u * G >> 4) << 24);  // fp16 x fp16 -> fp32
            const uint64_t desc0 = smem_desc(base, 128);
            for (uint32_t u = rank == 0 ? first_unit : p.units; u < p.units && ok; u += unit_step) {
                const PgUnit t = pg_unit(p, u);
                for (uint32_t k = (t.ks1 - t.ks0) * 4; k > 0; --k) {
                    if (!(ok = __all_sync(0xffffffffu, bar_wait<G == 2 ? BAR_PAIR_TURN : BAR_CTA>(d_empty + d * 8, d_par, &dead)))) break;
                    if (!(ok = __all_sync(0xffffffffu, bar_wait<G == 2 ? BAR_PAIR : BAR_CTA>(full + st * 8, parity, &dead)))) break;
                    fence_after();
                    const uint64_t da = desc0 + st * (stage_bytes >> 4), db = da + (C::kABytes >> 4);
                    const uint32_t acc = tmem + d * W;
                    if (issuer) {
#pragma unroll
                        for (uint32_t i = 0; i < 8; ++i) {
                            const uint64_t a = da + (i & 3) * 2, b = db + (i & 3) * 2 + (i < 4 ? 0 : half_bytes >> 4);
                            if (i == 4)  // the lo parts are summed: back to the unit of the hi parts
                                mma_f16_shifted<G, kLoShift>(acc, a, b, idesc);
                            else if constexpr (G == 2)
                                mma_f16_pair(acc, a, b, idesc, i > 0);
                            else
                                mma_f16(acc, a, b, idesc, i > 0);
                        }
                        if constexpr (G == 2) {
                            commit_pair(empty + st * 8);
                            commit_pair(d_full + d * 8);
                        } else {
                            commit(empty + st * 8);
                            commit(d_full + d * 8);
                        }
                    }
                    if (++st == stages) {
                        st = 0;
                        parity ^= 1;
                    }
                    if (++d == C::kD) {
                        d = 0;
                        d_par ^= 1;
                    }
                }
            }
            if (!ok && issuer) {
                if constexpr (G == 2)
                    commit_pair(drained);
                else
                    commit(drained);
                bar_drain(drained, 0);
            }
        } else if (G == 2 && warp == 2 && lane == 0 && rank == 1) {
            // this CTA's copies and unpacked weights of a stage are complete: tell the issuing CTA
            uint32_t st = 0, parity = 0;
            bool ok = true;
            for (uint32_t u = first_unit; u < p.units && ok; u += unit_step) {
                const PgUnit t = pg_unit(p, u);
                for (uint32_t i = (t.ks1 - t.ks0) * 4; i > 0; --i) {
                    if (!(ok = bar_wait(full + st * 8, parity, &dead))) break;
                    bar_release_leader(leader_addr(full + st * 8));
                    if (++st == stages) {
                        st = 0;
                        parity ^= 1;
                    }
                }
            }
        }
    } else if (warp < 8) {
        if constexpr (W > 64) asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
        // Weights do not depend on earlier kernels: no dependency wait. Warp w takes row pair w of the tile; the
        // codes of the super-tile after this one are on their way while this one is unpacked.
        const uint32_t w4 = warp - 4, g = lane >> 2, t4 = lane & 3;
        constexpr uint32_t kVec = DT == 1 ? 4 : 2;
        uint4 q[2][kVec];
        uint32_t st = 0, parity = 1;
        bool ok = true;
        const uint32_t mine = base + (w4 * 32 + g) * 128;
        const uint32_t c0 = ((2 * t4) ^ g) * 16, c1 = ((2 * t4 + 1) ^ g) * 16;
        auto load = [&](const uint8_t *base, bool live, uint32_t tile, uint32_t j) {
            q[tile][j] = live ? __ldg(reinterpret_cast<const uint4 *>(base + tile * Fmt<DT>::kSuperTileBytes + kScaleBytes +
                                                                     j * 512 + lane * 16))
                              : make_uint4(0, 0, 0, 0);
        };
        for (uint32_t u = first_unit; u < p.units && ok; u += unit_step) {
            const PgUnit t = pg_unit(p, u);
            const uint32_t pair = (t.rt * G + rank) * 4 + w4;
            const bool live = pair < p.pairs;
            if (u == first_unit) {
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
                } else if (u + unit_step < p.units) {
                    const PgUnit n = pg_unit(p, u + unit_step);
                    const uint32_t next_pair = (n.rt * G + rank) * 4 + w4;
                    next_live = next_pair < p.pairs;
                    next = pg_tile<DT>(p, next_live ? next_pair : 0, n.ks0, 0);
                } else {
                    next_live = false;
                    next = p.w;
                }
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j) {
                    if (!__all_sync(0xffffffffu, bar_wait(empty + st * 8, parity, &dead))) {
                        ok = false;
                        break;
                    }
                    const uint32_t row = mine + st * stage_bytes;
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
                    if (lane == 0) bar_arrive(full + st * 8);
                    if (++st == stages) {
                        st = 0;
                        parity ^= 1;
                    }
                }
            }
        }
    } else {
        if constexpr (W > 64) asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
        pdl_wait();
        const uint32_t quarter = warp & 3, half = (warp - 8) >> 2;  // tensor-memory lanes and columns of this warp
        // the two warps of a quarter share its n columns, in chunks of 16
        const uint32_t first = half ? (p.n + 31) / 32 * 16 : 0, columns = half ? p.n - first : (p.n + 31) / 32 * 16;
        const uint32_t src = tmem + first + ((quarter * 32) << 16);
        uint32_t used = 0;
        const uint32_t report = G == 2 ? leader_addr(d_empty) : d_empty;
        bool ok = true;
        // Bit i: this warp's columns of tile i hold a position that is marked. In shared memory, because the loop below has no
        // register to spare.
        uint32_t tiles = 0;
        for (uint32_t i = 0; i < p.pos_tiles; ++i) {
            const uint32_t n0 = i * p.n + first, end = n0 >= p.m ? 0 : min(columns, p.m - n0);
            const uint32_t marks = lane * 4 < end ? *reinterpret_cast<const uint32_t *>(p.spread + n0 + lane * 4) : 0;
            const uint32_t live = end >= lane * 4 + 4 ? 0xffffffffu : (1u << (8 * (end & 3))) - 1;
            if (__any_sync(0xffffffffu, (marks & live) != 0)) tiles |= 1u << i;
        }
        if (lane == 0) marked_tiles[warp - 8] = tiles;
        __syncwarp();
        for (uint32_t u = first_unit; u < p.units && ok; u += unit_step) {
            const PgUnit t = pg_unit(p, u);
            const uint32_t pair = (t.rt * G + rank) * 4 + quarter, row = pair * 32 + lane;
            const bool live = pair < p.pairs;
            // scales of this row: four fp16 per super-tile
            const uint32_t sc_off = (lane & 7) * 16 + ((lane >> 3) & 1) * 8;
            auto scales = [&](uint32_t ks) {
                return live && ks < t.ks1
                           ? __ldg(reinterpret_cast<const uint2 *>(pg_tile<DT>(p, pair, ks, lane >> 4) + sc_off))
                           : make_uint2(0, 0);
            };
            float acc[W / 2];
#pragma unroll
            for (uint32_t i = 0; i < W / 2; ++i) acc[i] = 0.f;
            auto sweep = [&](auto marked_units) {
                // The marked form takes the units of 32 columns at a time from shared memory, where the warp puts those of
                // the next block once this block's have been read.
                constexpr bool kMarked = decltype(marked_units)::value;
                constexpr uint32_t kLoad = kMarked || W <= 64 ? 32 : 64;
                float *units = unit_stage[warp - 8];
                float next_units[W / 64];
                auto fetch = [&](uint32_t block) {
#pragma unroll
                    for (uint32_t i = 0; i < W / 64; ++i)
                        next_units[i] = block < p.kst * 4 ? p.block_unit[(size_t)block * p.pos_pad + t.n0 + first + i * 32 + lane] : 0.f;
                };
                if constexpr (kMarked) fetch(t.ks0 * 4);
                uint2 sc = scales(t.ks0);
                for (uint32_t ks = t.ks0; ks < t.ks1 && ok; ++ks) {
                    const uint2 sc_next = scales(ks + 1);
#pragma unroll 1
                    for (uint32_t j = 0; j < 4; ++j, ++used) {
                        const uint32_t d = used % C::kD;
                        if constexpr (kMarked) {
                            __syncwarp();  // the block before has been read
#pragma unroll
                            for (uint32_t i = 0; i < W / 64; ++i) units[i * 32 + lane] = next_units[i];
                            fetch(ks * 4 + j + 1);
                            __syncwarp();
                        }
                        if (!__all_sync(0xffffffffu, bar_wait(d_full + d * 8, (used / C::kD) & 1, &dead))) {
                            ok = false;
                            break;
                        }
                        fence_after();
                        const uint32_t word = j & 2 ? sc.y : sc.x;
                        const float s = __half2float(__ushort_as_half((uint16_t)(j & 1 ? word >> 16 : word & 0xffff)));
                        // columns past the tile's belong to the accumulator all the same, and their sums are not stored
#pragma unroll
                        for (uint32_t c = 0; c < W / 2; c += kLoad) {
                            if (c >= columns) break;
                            float v[kLoad];
                            if constexpr (kLoad == 64)
                                tmem_ld64(src + d * W + c, v);
                            else
                                tmem_ld32(src + d * W + c, v);
                            tmem_ld_wait();
                            if (c + kLoad >= columns) {  // all of the accumulator is in registers
                                fence_before();
                                __syncwarp();
                                if (lane == 0) {
                                    if constexpr (G == 2)
                                        bar_turn_leader(report + d * 8);
                                    else
                                        bar_arrive(report + d * 8);
                                }
                            }
                            if constexpr (kMarked) {
#pragma unroll
                                for (uint32_t i = 0; i < kLoad; i += 4) {
                                    const float4 x = *reinterpret_cast<const float4 *>(units + c + i);
                                    v[i] *= x.x;
                                    v[i + 1] *= x.y;
                                    v[i + 2] *= x.z;
                                    v[i + 3] *= x.w;
                                }
                            }
#pragma unroll
                            for (uint32_t i = 0; i < kLoad; i += 2) pg_fma2(acc + c + i, s, v + i);
                        }
                    }
                    sc = sc_next;
                }
            };
            // the units of blocks for all positions of this warp, if one is marked
            if ((marked_tiles[warp - 8] >> (u % p.pos_tiles)) & 1)
                sweep(std::true_type());
            else
                sweep(std::false_type());
            {  // what is left of the units: a factor per column, one for marked tiles
                const bool in_blocks = (marked_tiles[warp - 8] >> (u % p.pos_tiles)) & 1;
                __syncwarp();
#pragma unroll
                for (uint32_t i = 0; i < W / 64; ++i) {
                    const uint32_t at = t.n0 + first + i * 32 + lane;
                    unit_stage[warp - 8][i * 32 + lane] = in_blocks || at >= p.m ? 1.0f : p.unit[at];
                }
                __syncwarp();
            }
            if (ok && row < p.rows) {
                const float so = (p.s_out ? p.s_out[row] : 1.0f) * code_unit(DT);
                const uint32_t n0 = t.n0 + first;
                float *y = p.y + t.sp * p.split_stride + (size_t)n0 * p.rows + row;
#pragma unroll
                for (uint32_t i = 0; i < W / 2; ++i)
                    if (i < columns && n0 + i < p.m) y[(size_t)i * p.rows] = acc[i] * unit_stage[warp - 8][i] * so;
            }
        }
    }
    __syncwarp();
    __syncthreads();
    if constexpr (G == 2) cluster_sync();  // no arrival at, and no product from, a CTA that has left
    if (warp == 1) {
        fence_after();
        if constexpr (G == 2)
            tmem_free_pair(tmem, kCols);
        else
            tmem_free(tmem, kCols);
    }
    if (tid == 0 && dead) *p.error_word = DEV_ERR_WAIT_TIMEOUT;
}

namespace {

template <int DT, uint32_t W, uint32_t G>
ctox_status pg_init(ctox_ctx *ctx, bool *usable) {
    const auto kernel = k_packed_gemm<DT, W, G>;
    cudaFuncAttributes attr;
    CTOX_CUDA(ctx, cudaFuncGetAttributes(&attr, kernel));
    if (W > 64 && attr.numRegs != 128) *usable = false;  // the split in the kernel counts on 128 per thread at launch
    CTOX_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ctx->max_smem_optin - 1024 - 16 * (int)W));
    return CTOX_OK;
}
template <int DT, uint32_t W, uint32_t G>
ctox_status pg_launch(ctox_ctx *ctx, PgParams &p) {
    const auto kernel = k_packed_gemm<DT, W, G>;
    const uint32_t stage = PgCfg<W, G>::kABytes + p.n / G * 256;
    p.stages = ((uint32_t)ctx->max_smem_optin - 2048 - 16 * W) / stage;  // beside the barriers and 16 W bytes of units
    if (p.stages > kPgStages) p.stages = kPgStages;
    const size_t smem = (size_t)p.stages * stage + 1024;
    const uint32_t slots = (uint32_t)ctx->sm_count / G, grid = (p.units < slots ? p.units : slots) * G;
    if constexpr (G == 2)
        CTOX_CUDA(ctx, launch_pdl_cluster(kernel, dim3(grid), dim3(kPgThreads), smem, ctx->stream, 2, p));
    else
        CTOX_CUDA(ctx, launch_pdl(kernel, dim3(grid), dim3(kPgThreads), smem, ctx->stream, p));
    return CTOX_OK;
}
template <int DT>
ctox_status pg_launch(ctox_ctx *ctx, PgParams &p) {
    return p.n > 128 ? pg_launch<DT, 256, 2>(ctx, p) : p.n > 64 ? pg_launch<DT, 128, 1>(ctx, p) : pg_launch<DT, 64, 1>(ctx, p);
}

}  // namespace

ctox_status packed_gemm_init(ctox_ctx *ctx, bool *usable) {
    *usable = true;
    EX((pg_init<0, 64, 1>(ctx, usable)));
    EX((pg_init<1, 64, 1>(ctx, usable)));
    EX((pg_init<0, 128, 1>(ctx, usable)));
    EX((pg_init<1, 128, 1>(ctx, usable)));
    EX((pg_init<0, 256, 2>(ctx, usable)));
    return pg_init<1, 256, 2>(ctx, usable);
}

ctox_status launch_packed_gemm(ctox_matvec *mv, const LongIn &in, uint32_t m, uint64_t row0, uint64_t row_end, float *y,
                               size_t capacity, LongOut *out) {
    ctox_ctx *ctx = mv->ctx;
    const MatvecPart &part = mv->parts[0];
    if (mv->parts.size() != 1 || m == 0 || row_end > mv->rows ||
        (size_t)m * mv->rows > capacity)
        return fail(ctx, CTOX_SHAPE, "packed product: %u positions of a %llu-row matrix", m, (unsigned long long)mv->rows);
    PgParams p{};
    p.w = part.prep;
    p.x = in.x;
    p.unit = in.unit;
    p.block_unit = in.block_unit;
    p.spread = in.spread;
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
    // Tile width and column split by the time of the longest chain of units on an SM, from what a 64-column block of n
    // positions was measured to take (us, one B200, 999 and 37 positions, four matrix shapes): 0.56 at 48, 0.60 at 96,
    // 0.64 at 128 (one CTA); 0.76 at 160, 0.90 at 256 (a pair). A unit costs about a microsecond more for filling its
    // pipeline and writing its sums; a partial sum beyond the first is written and read again at about 5 TB/s.
    double best = 1e30;
    for (uint32_t n = 32; n <= 256; n += n < 128 ? 16 : 32) {
        const uint32_t G = n > 128 ? 2 : 1, slots = (uint32_t)ctx->sm_count / G;
        const double step = G == 2 ? 0.53 + 0.00146 * n : 0.52 + 0.0009 * n;
        const uint32_t tiles = (m + n - 1) / n, tiles_r = (row_tiles + G - 1) / G;
        if (tiles * n > in.pos_pad || p.rt0 % G || tiles > 32) continue;
        for (uint32_t s = 1; s <= p.kst && s <= 16 && s * p.split_stride <= capacity; ++s) {
            const uint32_t units = tiles_r * tiles * s, rounds = (units + slots - 1) / slots;
            const double cost = rounds * (((p.kst + s - 1) / s) * 4 * step + 1.0) + (s - 1) * (0.5 + 1.6e-6 * p.split_stride);
            if (cost < best) {
                best = cost;
                p.n = n;
                p.splits = s;
                p.units = units;
            }
        }
    }
    if (p.n == 0) return fail(ctx, CTOX_SHAPE, "packed product: %u positions exceed the buffer's %u", m, in.pos_pad);
    p.pos_tiles = (m + p.n - 1) / p.n;
    if (p.n > 128) p.rt0 /= 2;
    timing_begin(ctx);
    EX(part.dt ? pg_launch<1>(ctx, p) : pg_launch<0>(ctx, p));
    timing_end(ctx, KC_GEMM, (double)part.prep_bytes + 4.0 * m * ((double)mv->columns + mv->rows),
               2.0 * (double)(row_end - row0) * (double)mv->columns * m);
    *out = LongOut{y, p.rows, p.splits, p.split_stride};
    return CTOX_OK;
}

}  // namespace ctox
