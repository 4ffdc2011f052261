// Persistent tensor-core product for long passes: one CTA per SM, 128 x BN tiles, operands staged by TMA
// (one thread), multiplied by tcgen05.mma (one thread), accumulators double-buffered in tensor memory so
// that four epilogue warps drain a tile while the next one is computed. Large products take pairs of CTAs
// (G = 2, cta_group::2): 256 x 256 tiles, each CTA with half of the rows of either operand, so that an SM draws 32
// instead of 48 KB from L2 per 512 cycles of tensor work.
#include "gemm.cuh"
#include "umma.cuh"

namespace ctox {

constexpr int kGmThreads = 192;  // warp 0: TMA, warp 1: MMA, warps 2-5: epilogue
constexpr uint32_t kGmM = 128, kGmK = 64, kGmStageMax = 8;

ctox_status tensor_map_bf16(ctox_ctx *ctx, CUtensorMap *map, const void *base, uint64_t rows, uint64_t cols, uint64_t ld,
                            uint32_t box_rows, uint32_t box_cols) {
    using Encode = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static Encode encode = nullptr;
    if (!encode) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        CTOX_CUDA(ctx, cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q));
        if (!fn || q != cudaDriverEntryPointSuccess)
            return fail(ctx, CTOX_UNSUPPORTED_OPERATION, "cuTensorMapEncodeTiled is not available");
        encode = (Encode)fn;
    }
    const cuuint64_t dims[2] = {cols, rows}, strides[1] = {ld * 2};
    const cuuint32_t box[2] = {box_cols, box_rows}, step[2] = {1, 1};
    const CUtensorMapSwizzle sw = box_cols * 2 == 128  ? CU_TENSOR_MAP_SWIZZLE_128B
                                  : box_cols * 2 == 64 ? CU_TENSOR_MAP_SWIZZLE_64B
                                                       : CU_TENSOR_MAP_SWIZZLE_32B;
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box, step,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
        return fail(ctx, CTOX_SHAPE, "tensor map of %llu x %llu (ld %llu): error %d", (unsigned long long)rows,
                    (unsigned long long)cols, (unsigned long long)ld, (int)r);
    return CTOX_OK;
}

struct GemmPages {  // cache rows behind an operand (table null: rows as they are)
    const uint32_t *table;
    uint32_t page_tokens, row0;
};
__device__ __forceinline__ int operand_row(const GemmPages &p, uint32_t row) {
    if (!p.table) return (int)row;
    const uint32_t pos = p.row0 + row;
    return (int)(p.table[pos / p.page_tokens] * p.page_tokens + pos % p.page_tokens);
}

// A warp's 32 rows m0 .. of BYTES bytes each, chunk c of this lane's row in w[c], to d + row * pitch: through shared memory, so
// that neighbouring lanes store neighbouring chunks. (A row per lane, each store touched 32 lines: a product over 512
// columns spent most of its 40 us on them.)
constexpr uint32_t kStoreStage = 32 * (128 + 16);  // bytes of shared memory per warp
template <uint32_t BYTES>
__device__ __forceinline__ void store_rows(uint8_t *d, size_t pitch, const uint4 *w, uint32_t rows, uint8_t *stage) {
    constexpr uint32_t C = BYTES / 16, kPitch = BYTES + 16;
    const uint32_t lane = threadIdx.x & 31;
    __syncwarp();  // the rows before have been read
#pragma unroll
    for (uint32_t c = 0; c < C; ++c) *reinterpret_cast<uint4 *>(stage + lane * kPitch + c * 16) = w[c];
    __syncwarp();
#pragma unroll
    for (uint32_t i = 0; i < C; ++i) {
        const uint32_t r = (i * 32 + lane) / C, c = (i * 32 + lane) % C;
        const uint4 x = *reinterpret_cast<const uint4 *>(stage + r * kPitch + c * 16);
        if (r < rows) *reinterpret_cast<uint4 *>(d + r * pitch + c * 16) = x;
    }
}

// 32 columns n0 .. n0 + 32 of the output rows of a warp; m: this lane's row (the warp's 32 rows follow one another). Lanes
// past the last row take part.
__device__ __forceinline__ void gemm_store(const GemmOut &o, float *v, uint32_t m, uint32_t n0, uint32_t M, uint32_t N,
                                           uint8_t *stage) {
    const uint32_t m0 = m - (threadIdx.x & 31), rows = M - m0 < 32 ? M - m0 : 32;  // m0 < M
    if (o.bias) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
            if (n0 + j < N) v[j] += __ldg(o.bias + n0 + j);
    }
    if (o.kind == OUT_CLAMPED_GLU) {
        __nv_bfloat16 *d = (__nv_bfloat16 *)o.d + (size_t)m * o.ld + n0 / 2;
        alignas(16) __nv_bfloat162 h[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
            h[j] = __floats2bfloat162_rn(clamped_glu(v[4 * j], v[4 * j + 1], o.cap, o.slope),
                                         clamped_glu(v[4 * j + 2], v[4 * j + 3], o.cap, o.slope));
        if (n0 + 32 <= N && o.ld % 8 == 0) {
            store_rows<32>((uint8_t *)((__nv_bfloat16 *)o.d + (size_t)m0 * o.ld + n0 / 2), (size_t)o.ld * 2,
                           reinterpret_cast<const uint4 *>(h), rows, stage);
        } else if (m < M) {
#pragma unroll
            for (int j = 0; j < 16; ++j)
                if (n0 + 2 * j < N) d[j] = j & 1 ? h[j / 2].y : h[j / 2].x;
        }
        return;
    }
    if (o.kind == OUT_RELU2) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = v[j] > 0.f ? v[j] * v[j] : 0.f;
    } else if (o.kind == OUT_SOFTCAP) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = o.cap * tanhf(v[j] / o.cap);
    } else if (o.kind == OUT_ROPE) {
        uint32_t w = n0 % o.head_width;  // heads are a multiple of 16 wide: w is even, a pair never straddles two
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
            if (m < M && w >= o.rope0 && w < o.rope0 + o.rope_dims) {
                const float2 cs = o.table[(size_t)m * (o.rope_dims / 2) + ((w - o.rope0) >> 1)];
                const float a = v[j] * cs.x - v[j + 1] * cs.y, b = v[j + 1] * cs.x + v[j] * cs.y;
                v[j] = a;
                v[j + 1] = b;
            }
            w += 2;
            if (w >= o.head_width) w -= o.head_width;
        }
    }
    const bool full = n0 + 32 <= N;
    if (o.split && n0 >= o.split) {
        if (m >= M) return;
        float *d = o.d2 + (size_t)m * o.ld2 + (n0 - o.split);
#pragma unroll
        for (int j = 0; j < 32; ++j)
            if (n0 + j < N) d[j] = v[j];
    } else if (o.bf16) {
        __nv_bfloat16 *d = (__nv_bfloat16 *)o.d + (size_t)m * o.ld + n0;
        if (full && o.ld % 8 == 0) {
            alignas(16) __nv_bfloat162 h[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) h[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
            store_rows<64>((uint8_t *)((__nv_bfloat16 *)o.d + (size_t)m0 * o.ld + n0), (size_t)o.ld * 2,
                           reinterpret_cast<const uint4 *>(h), rows, stage);
        } else if (m < M) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
                if (n0 + j < N) d[j] = __float2bfloat16_rn(v[j]);
        }
    } else {
        float *d = (float *)o.d + (size_t)m * o.ld + n0;
        if (full && o.ld % 4 == 0) {
            store_rows<128>((uint8_t *)((float *)o.d + (size_t)m0 * o.ld + n0), (size_t)o.ld * 4, reinterpret_cast<const uint4 *>(v),
                            rows, stage);
        } else if (m < M) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
                if (n0 + j < N) d[j] = v[j];
        }
    }
}

template <uint32_t BN, uint32_t G>
__global__ void __launch_bounds__(kGmThreads, 1)
    k_gemm(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, GemmPages pa, GemmPages pb,
           uint32_t M, uint32_t N, uint32_t K, uint32_t stages, GemmOut out, int32_t *error_word) {
    using namespace umma;
    constexpr uint32_t kBRows = BN / G, kABytes = kGmM * kGmK * 2, kBBytes = kBRows * kGmK * 2;  // of this CTA
    constexpr uint32_t kBBox = kBRows < 128 ? kBRows : 128, kBoxes = kBRows / kBBox;
    constexpr uint32_t kCols = 2 * BN;
    extern __shared__ uint8_t raw[];
    __shared__ __align__(8) uint64_t bars[2 * kGmStageMax + 5];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int dead;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = G == 2 ? cluster_rank() : 0;
    const uint32_t base = (smem_addr(raw) + 1023) & ~1023u;
    const uint32_t full = smem_addr(bars), empty = full + kGmStageMax * 8, acc_full = empty + kGmStageMax * 8,
                   acc_empty = acc_full + 16, drained = acc_empty + 16;
    if (tid == 0) {
        dead = 0;
        for (uint32_t i = 0; i < stages; ++i) {
            bar_init(full + i * 8, 1);  // at the first CTA of a pair: the copies of both
            bar_init(empty + i * 8, 1);
        }
        for (uint32_t i = 0; i < 2; ++i) {
            bar_init(acc_full + i * 8, 1);
            bar_init(acc_empty + i * 8, 4 * G);
        }
        bar_init(drained, 1);
        bar_init_fence();
        tma_prefetch_map(&map_a);
        tma_prefetch_map(&map_b);
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
    pdl_launch();  // a later kernel's allocation must not come before this one's (see umma.cuh)
    const uint32_t tmem = tmem_slot;
    const uint32_t tiles_m = (M + kGmM * G - 1) / (kGmM * G), tiles_n = (N + BN - 1) / BN, tiles = tiles_m * tiles_n;
    const uint32_t ksteps = (K + kGmK - 1) / kGmK, first = blockIdx.x / G, step = gridDim.x / G;
    pdl_wait();
    if (warp == 0) {
        if (lane == 0) {
            uint32_t issued = 0, s = 0, parity = 1;  // parity of the phase before a ring's first: passes at once
            bool ok = true;
            for (uint32_t t = first; t < tiles && ok; t += step) {
                const uint32_t m0 = (t % tiles_m * G + rank) * kGmM, n0 = t / tiles_m * BN + rank * kBRows;
                const int ra = m0 < M ? operand_row(pa, m0) : (int)m0;
                int rb[kBoxes];
#pragma unroll
                for (uint32_t i = 0; i < kBoxes; ++i) rb[i] = n0 + i * 128 < N ? operand_row(pb, n0 + i * 128) : (int)(n0 + i * 128);
                for (uint32_t k = 0; k < ksteps; ++k, ++issued) {
                    if (!(ok = bar_wait(empty + s * 8, parity, &dead))) break;
                    const uint32_t bar = full + s * 8, dst = base + s * (kABytes + kBBytes);
                    auto load = [&](uint32_t to, const CUtensorMap *map, int row) {
                        if constexpr (G == 2)
                            tma_load_pair(to, map, leader_addr(bar), (int)(k * kGmK), row);
                        else
                            tma_load(to, map, bar, (int)(k * kGmK), row);
                    };
                    if (rank == 0) bar_expect(bar, G * (kABytes + kBBytes));
                    load(dst, &map_a, ra);
#pragma unroll
                    for (uint32_t i = 0; i < kBoxes; ++i) load(dst + kABytes + i * kBBox * kGmK * 2, &map_b, rb[i]);
                    if (++s == stages) {
                        s = 0;
                        parity ^= 1;
                    }
                }
            }
            if (!ok) {  // leave no copy in flight behind; a pair's barrier may lack the other CTA's part, so by time
                if constexpr (G == 2) {
                    const long long t0 = clock64();
                    while (clock64() - t0 < 2000000) {
                    }
                } else {
                    for (uint32_t i = 0; i < stages && i < issued; ++i)
                        bar_drain(full + (issued - 1 - i) % stages * 8, ((issued - 1 - i) / stages) & 1);
                }
            }
        }
    } else if (warp == 1) {
        // The whole warp runs the loop and one lane issues: its values are uniform, so that descriptors need no moves
        // between register files. The second CTA of a pair issues nothing.
        const bool issuer = elect_one();
        uint32_t s = 0, parity = 0, n_tile = 0;
        bool ok = true;
        const uint32_t idesc = idesc_bf16(kGmM * G, BN);
        const uint64_t desc0 = smem_desc(base, 128);
        for (uint32_t t = rank == 0 ? first : tiles; t < tiles && ok; t += step, ++n_tile) {
            const uint32_t acc = n_tile & 1, d = tmem + acc * BN;
            if (!(ok = __all_sync(0xffffffffu, bar_wait<G == 2 ? BAR_PAIR_TURN : BAR_CTA>(acc_empty + acc * 8, ((n_tile >> 1) & 1) ^ 1, &dead)))) break;
            fence_after();
            for (uint32_t k = 0; k < ksteps; ++k) {
                if (!(ok = __all_sync(0xffffffffu, bar_wait(full + s * 8, parity, &dead)))) break;
                fence_after();
                const uint64_t da = desc0 + s * ((kABytes + kBBytes) >> 4), db = da + (kABytes >> 4);
                if (issuer) {
#pragma unroll
                    for (uint32_t i = 0; i < kGmK / 16; ++i) {
                        if constexpr (G == 2)
                            mma_f16_pair(d, da + i * 2, db + i * 2, idesc, k > 0 || i > 0);
                        else
                            mma_f16(d, da + i * 2, db + i * 2, idesc, k > 0 || i > 0);
                    }
                    if constexpr (G == 2)
                        commit_pair(empty + s * 8);
                    else
                        commit(empty + s * 8);
                }
                if (++s == stages) {
                    s = 0;
                    parity ^= 1;
                }
            }
            if (ok && issuer) {
                if constexpr (G == 2)
                    commit_pair(acc_full + acc * 8);
                else
                    commit(acc_full + acc * 8);
            }
        }
        if (!ok && issuer) {
            if constexpr (G == 2)
                commit_pair(drained);
            else
                commit(drained);
            bar_drain(drained, 0);
        }
    } else {
        const uint32_t quarter = warp & 3;  // the lanes of tensor memory this warp may read
        const uint32_t report = G == 2 ? leader_addr(acc_empty) : acc_empty;
        uint8_t *raw_stage = raw + (base - smem_addr(raw)) + stages * (kABytes + kBBytes) + quarter * kStoreStage;
        uint32_t n_tile = 0;
        for (uint32_t t = first; t < tiles; t += step, ++n_tile) {
            const uint32_t acc = n_tile & 1, m = (t % tiles_m * G + rank) * kGmM + quarter * 32 + lane, n0 = t / tiles_m * BN;
            if (!__all_sync(0xffffffffu, bar_wait(acc_full + acc * 8, (n_tile >> 1) & 1, &dead))) break;
            fence_after();
            const uint32_t src = tmem + acc * BN + ((quarter * 32) << 16);
#pragma unroll 1
            for (uint32_t c = 0; c < BN; c += 32) {
                alignas(16) float v[32];
                tmem_ld32(src + c, v);
                tmem_ld_wait();
                if (m - lane < M && n0 + c < N) gemm_store(out, v, m, n0 + c, M, N, raw_stage);
            }
            fence_before();
            __syncwarp();
            if (lane == 0) {
                if constexpr (G == 2)
                    bar_turn_leader(report + acc * 8);
                else
                    bar_arrive(report + acc * 8);
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
    if (tid == 0 && dead) *error_word = DEV_ERR_WAIT_TIMEOUT;
}

namespace {

template <uint32_t BN, uint32_t G>
ctox_status gemm_launch(ctox_ctx *ctx, const GemmOperand &a, const GemmOperand &b, const GemmOut &out) {
    const uint32_t stage_bytes = kGmM * kGmK * 2 + BN / G * kGmK * 2;
    uint32_t stages = ((uint32_t)ctx->max_smem_optin - 2048 - 4 * kStoreStage) / stage_bytes;
    if (stages > kGmStageMax) stages = kGmStageMax;
    const size_t smem = (size_t)stages * stage_bytes + 1024 + 4 * kStoreStage;
    CUtensorMap ma, mb;
    auto encode = [&](CUtensorMap *m, const GemmOperand &o, uint32_t box) {
        return tensor_map_bf16(ctx, m, o.p, o.page_table ? o.store_rows : o.rows, o.cols, o.ld, box, kGmK);
    };
    ctox_status rc = encode(&ma, a, kGmM);
    if (!rc) rc = encode(&mb, b, BN / G < 128 ? BN / G : 128);
    if (rc) return rc;
    CTOX_CUDA(ctx, cudaFuncSetAttribute(k_gemm<BN, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const uint32_t tiles = ((a.rows + kGmM * G - 1) / (kGmM * G)) * ((b.rows + BN - 1) / BN);
    const uint32_t slots = (uint32_t)ctx->sm_count / G, grid = (tiles < slots ? tiles : slots) * G;
    const GemmPages pa{a.page_table, a.page_tokens, a.row0}, pb{b.page_table, b.page_tokens, b.row0};
    if constexpr (G == 2)
        CTOX_CUDA(ctx, launch_pdl_cluster(k_gemm<BN, G>, dim3(grid), dim3(kGmThreads), smem, ctx->stream, 2, ma, mb, pa, pb,
                                          a.rows, b.rows, a.cols, stages, out, ctx->dev_error));
    else
        CTOX_CUDA(ctx, launch_pdl(k_gemm<BN, G>, dim3(grid), dim3(kGmThreads), smem, ctx->stream, ma, mb, pa, pb, a.rows, b.rows,
                                  a.cols, stages, out, ctx->dev_error));
    return CTOX_OK;
}

}  // namespace

ctox_status launch_gemm(ctox_ctx *ctx, const GemmOperand &a, const GemmOperand &b, const GemmOut &out) {
    if (!a.rows || !b.rows) return CTOX_OK;
    if (a.cols != b.cols || a.ld % 8 || b.ld % 8) return fail(ctx, CTOX_SHAPE, "gemm: operand layouts");
    for (const GemmOperand *o : {&a, &b})
        if (o->page_table && (o->page_tokens % 128 || o->row0 % 128))
            return fail(ctx, CTOX_SHAPE, "gemm: pages of %u tokens are not whole tiles", o->page_tokens);
    // tile by rounds over the SMs (an SM's work per round, in columns); a narrower tile has less reuse, hence the constant. A
    // pair's tile is as much work for an SM as the 256-wide one and less traffic: 270 against 320. Measured over the products
    // of two latent-attention layers of width 5120, 2048 tokens, with pairs and without: 1.12 against 1.23 ms (feed-forward
    // of 16384), 0.67 against 0.75 ms (8192), 0.91 and 0.90 of the time with the products too small for pairs among them.
    uint32_t best = 0, best_cost = 0xffffffffu;
    for (uint32_t bn : {512u, 256u, 128u, 64u}) {  // 512: a pair's 256 x 256
        const uint32_t G = bn == 512 ? 2 : 1, w = bn == 512 ? 256 : bn, slots = (uint32_t)ctx->sm_count / G;
        const uint32_t tiles = ((a.rows + kGmM * G - 1) / (kGmM * G)) * ((b.rows + w - 1) / w);
        const uint32_t cost = ((tiles + slots - 1) / slots) * (G == 2 ? 270 : w + 64);
        if (cost < best_cost) {
            best_cost = cost;
            best = bn;
        }
    }
    timing_begin(ctx);
    EX(best == 512   ? (gemm_launch<256, 2>(ctx, a, b, out))
       : best == 256 ? (gemm_launch<256, 1>(ctx, a, b, out))
       : best == 128 ? (gemm_launch<128, 1>(ctx, a, b, out))
                     : (gemm_launch<64, 1>(ctx, a, b, out)));
    timing_end(ctx, KC_GEMM, 2.0 * ((double)a.rows + b.rows) * a.cols + (out.bf16 ? 2.0 : 4.0) * a.rows * b.rows,
               2.0 * a.rows * b.rows * a.cols);
    return CTOX_OK;
}

__global__ void k_rope_table(const float *__restrict__ freq, uint32_t pairs, uint32_t pos0, uint32_t rows,
                             float2 *__restrict__ table) {
    pdl_launch();
    pdl_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows * pairs) return;
    float s, c;
    sincosf((float)(pos0 + i / pairs) * freq[i % pairs], &s, &c);
    table[i] = make_float2(c, s);
}

ctox_status launch_rope_table(ctox_ctx *ctx, const float *freq, uint32_t pairs, uint32_t pos0, uint32_t rows,
                              float2 *table) {
    CTOX_CUDA(ctx, launch_pdl(k_rope_table, dim3((rows * pairs + 255) / 256), dim3(256), 0, ctx->stream, freq, pairs, pos0,
                              rows, table));
    return CTOX_OK;
}

}  // namespace ctox
