// Matrix-vector product of one position with dense bf16 weights, streamed through shared memory (plain decode of the layer
// stacks).
//
// What bounds it: HBM, then what a decode step's chain of launches adds to it (the prologue's round trip and block sums, about 2 us of
// each). 17408 x 5120 and back (178 MB each) take 33 and 28 us in that chain, 5.4 and 6.4 TB/s; the chain of the latent model
// 15.6 ms for 16 tokens against 19.3 with k_dense_matvec, whose loads go through registers, in waves of whole row units.
//
// A CTA per SM takes an equal share of the rows; its 16 warps stand side by side on the columns (as many
// per row as keep a warp's part of the input in registers), and every warp keeps a ring of bulk copies of its own row parts in
// flight. They start before the dependency wait: the weights are constants, so they arrive while the kernels before this one end
// and while the prologue (residual add, norm) forms the input.
#include "dense_device.cuh"
#include "umma.cuh"

#include <mutex>
#include <set>

namespace ctox {

constexpr uint32_t kDsWarps = 16, kDsThreads = kDsWarps * 32;
constexpr uint32_t kDsSteps = 5;    // vectors of eight columns per lane, at most: 40 registers of input
constexpr uint32_t kDsInput = 4;    // vectors of four columns of a normalised input per thread, at most
constexpr uint32_t kDsStages = 16;  // copies in flight per warp, at most
// Shared memory of a launch. A deeper ring holds up the prologue's loads, a shallower one leaves HBM idle meanwhile: 16 decoded tokens of
// an eight-layer model of width 5120 / a request with 32 decoded tokens on one of width 2048 / one of 30 + 30 tokens through four latent layers of
// width 2560 take 16.2 / 15.3 / 8.4 ms with 220 KB, 15.65 / 15.1 / 8.2 with 140, 15.6 / 15.1 / 8.2 with 108, 15.85 / 15.3 / 8.3 with 84.
constexpr size_t kDsRoom = 140 * 1024;
constexpr uint32_t kDsBatch = 4;    // rows summed over the lanes together

struct DenseStream {
    const __nv_bfloat16 *w;
    uint32_t ld, rows;
    uint32_t ks_log2, seg;  // warps per row, vectors of eight columns per warp
    uint32_t stages, stage_bytes;
    uint32_t part_at, x_at;  // byte offsets in shared memory: partial sums [row][warp of the row], input vector
    VecIn in;
    VecOut out;
    LatentAppend ap;
    uint32_t append_positions;
    int32_t *error_word;
};

__device__ __forceinline__ float block_sum(float v, float *red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float s = 0.f;
#pragma unroll
    for (uint32_t i = 0; i < kDsWarps; ++i) s += red[i];
    return s;
}

// The input vector (VecIn with a norm) in xs, zero from its last column to ld. A thread holds four columns of every kDsThreads *
// 4 in registers throughout: the norms' weights, which are constants, from before the dependency wait, the vectors from one
// round trip after it (three dependent trips and the reductions' barriers took 5 to 6 us of a launch). CTA 0 stores the
// stream with its sublayer's output added.
template <int NORM>
struct InputNorm {
    float4 w[kDsInput], wb[kDsInput];
    __device__ __forceinline__ void constants(const VecIn &in) {
        const bool vec = ((uintptr_t)in.w & 15) == 0, vec_b = ((uintptr_t)in.wb & 15) == 0;
#pragma unroll
        for (uint32_t i = 0; i < kDsInput; ++i) {
            const uint32_t c = (i * kDsThreads + threadIdx.x) * 4;
            w[i] = load4(in.w, c, in.cols, vec);
            if (NORM == NORM_LAYER && in.wb) wb[i] = load4(in.wb, c, in.cols, vec_b);
        }
    }
    float4 v[kDsInput], y[kDsInput];
    __device__ __forceinline__ void load(const VecIn &in) {
        const bool vec_x = ((uintptr_t)in.x & 15) == 0, vec_y = ((uintptr_t)in.y & 15) == 0;
#pragma unroll
        for (uint32_t i = 0; i < kDsInput; ++i) {
            const uint32_t c = (i * kDsThreads + threadIdx.x) * 4;
            v[i] = load4(in.x, c, in.cols, vec_x);
            if (in.y) y[i] = load4(in.y, c, in.cols, vec_y);
        }
    }
    __device__ __forceinline__ void form(const VecIn &in, float *xs, uint32_t ld, float (*red)[kDsWarps]) {
        const uint32_t cols = in.cols;
        auto sum4 = [](const float4 &v) { return (v.x + v.y) + (v.z + v.w); };
        auto sq4 = [](const float4 &v) { return (v.x * v.x + v.y * v.y) + (v.z * v.z + v.w * v.w); };
        // v - mean, zero past the last column
        auto centred = [&](const float4 &v, uint32_t c, float mean) {
            return make_float4(c < cols ? v.x - mean : 0.f, c + 1 < cols ? v.y - mean : 0.f, c + 2 < cols ? v.z - mean : 0.f,
                               c + 3 < cols ? v.w - mean : 0.f);
        };
        const float n = (float)cols;
        float s = 0.f, mean = 0.f;
        if (in.y) {
            if (NORM == NORM_LAYER && in.wb) {
#pragma unroll
                for (uint32_t i = 0; i < kDsInput; ++i) s += sum4(y[i]);
                mean = block_sum(s, red[0]) / n;
                s = 0.f;
#pragma unroll
                for (uint32_t i = 0; i < kDsInput; ++i) {
                    y[i] = centred(y[i], (i * kDsThreads + threadIdx.x) * 4, mean);
                    s += sq4(y[i]);
                }
                const float inv = 1.0f / sqrtf(block_sum(s, red[1]) / n + in.eps);
#pragma unroll
                for (uint32_t i = 0; i < kDsInput; ++i)
                    y[i] = make_float4(y[i].x * inv * wb[i].x, y[i].y * inv * wb[i].y, y[i].z * inv * wb[i].z, y[i].w * inv * wb[i].w);
            }
#pragma unroll
            for (uint32_t i = 0; i < kDsInput; ++i) {
                const uint32_t c = (i * kDsThreads + threadIdx.x) * 4;
                v[i] = make_float4(v[i].x + y[i].x, v[i].y + y[i].y, v[i].z + y[i].z, v[i].w + y[i].w);
                if (blockIdx.x == 0 && c < cols) store4(in.x_out, c, cols, v[i]);
            }
        }
        if (NORM == NORM_LAYER) {
            s = 0.f;
#pragma unroll
            for (uint32_t i = 0; i < kDsInput; ++i) s += sum4(v[i]);
            mean = block_sum(s, red[2]) / n;
#pragma unroll
            for (uint32_t i = 0; i < kDsInput; ++i) v[i] = centred(v[i], (i * kDsThreads + threadIdx.x) * 4, mean);
        }
        s = 0.f;
#pragma unroll
        for (uint32_t i = 0; i < kDsInput; ++i) s += sq4(v[i]);
        const float inv = 1.0f / sqrtf(block_sum(s, red[3]) / n + in.eps);
#pragma unroll
        for (uint32_t i = 0; i < kDsInput; ++i) {
            const uint32_t c = (i * kDsThreads + threadIdx.x) * 4;
            if (c < ld)
                *reinterpret_cast<float4 *>(xs + c) = make_float4(v[i].x * inv * w[i].x, v[i].y * inv * w[i].y, v[i].z * inv * w[i].z,
                                                                  v[i].w * inv * w[i].w);
        }
        __syncthreads();
    }
};

// d += a * b, lane by lane of the pair
__device__ __forceinline__ void fma2(float2 &d, float a0, float a1, float b0, float b1) {
    asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%0, %1};\n\t"
        "fma.rn.f32x2 c, a, b, c;\n\tmov.b64 {%0, %1}, c;\n\t}"
        : "+f"(d.x), "+f"(d.y)
        : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}

// NS: vectors per lane; NORM, KIND: of the input and the outputs, one kernel each, since a launch reads its code anew and a decode step is
// a chain of them.
template <int NS, int NORM, int KIND>
__global__ void __launch_bounds__(kDsThreads, 1) k_dense_stream(const __grid_constant__ DenseStream a) {
    using namespace umma;
    if (!a.append_positions) pdl_launch();
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t bars[kDsWarps * kDsStages];
    __shared__ float red[4][kDsWarps];
    __shared__ volatile int dead;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, grid = gridDim.x - a.append_positions;
    if (blockIdx.x >= grid) {
        pdl_wait();
        pdl_launch();
        latent_append_row(a.ap, blockIdx.x - grid, tid, kDsThreads, red[0]);
        return;
    }
    // Rows of this CTA, in whole pairs (a gated or rotated output needs both rows of a pair), then of this warp.
    const uint32_t row_pairs = (a.rows + 1) / 2;
    const uint32_t r0 = 2 * (uint32_t)((uint64_t)blockIdx.x * row_pairs / grid),
                   r1 = min(a.rows, 2 * (uint32_t)((uint64_t)(blockIdx.x + 1) * row_pairs / grid)), n = r1 - r0;
    const uint32_t ks = 1u << a.ks_log2, kp = warp & (ks - 1), rg = warp >> a.ks_log2, groups = kDsWarps >> a.ks_log2;
    const uint32_t first = n * rg / groups, count = n * (rg + 1) / groups - first;  // from r0 on
    const uint32_t vectors = a.ld / 8, v0 = kp * a.seg, len = v0 < vectors ? min(a.seg, vectors - v0) : 0;
    const __nv_bfloat16 *src = a.w + (size_t)(r0 + first) * a.ld + (size_t)v0 * 8;
    const uint32_t my_bars = smem_addr(&bars[warp * kDsStages]), ring = smem_addr(smem) + warp * a.stages * a.stage_bytes;
    const uint32_t todo = len ? count : 0;
    // A row is read once in a pass: its lines are the first to leave L2. With the default priority the weights push out what later
    // kernels read again (cache rows, states, norm weights), which the loads of k_dense_matvec do not: a token's cache attention over 32-bit
    // rows took 31 us instead of 23. A request of 134 + 31 tokens on a latent model (6 layers of width 2048, 32-bit cache) 26.4 -> 24.9 ms,
    // 16 tokens of the eight-layer model of width 5120 16.1 -> 15.6.
    uint64_t once;
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(once));
    auto request = [&](uint32_t row, uint32_t st) {  // one thread
        bar_expect(my_bars + 8 * st, len * 16);
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(
                         ring + st * a.stage_bytes),
                     "l"(src + (size_t)row * a.ld), "r"(len * 16), "r"(my_bars + 8 * st), "l"(once)
                     : "memory");
    };
    // Half of the ring is asked for here; the rest once the input's loads are on their way, which would wait behind it.
    const uint32_t early = min(todo, (a.stages + 1) / 2), late = min(todo, a.stages);
    if (tid == 0) dead = 0;
    if (lane == 0) {
        for (uint32_t s = 0; s < a.stages; ++s) bar_init(my_bars + 8 * s, 1);
        bar_init_fence();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        for (uint32_t s = 0; s < early; ++s) request(s, s);
    }
    // What of the input and the outputs does not depend on earlier kernels: weights of the norms, and of this thread's row (the
    // first kDsThreads rows; the others' are formed at the end) the bias and the turn.
    InputNorm<NORM> norm;
    if constexpr (NORM != NORM_NONE) norm.constants(a.in);
    const RowConstants mine = row_constants<KIND>(a.out, 0, r0 + tid, tid < n ? a.rows : 0);
    __syncthreads();
    pdl_wait();
    if (a.append_positions) pdl_launch();  // see dense.cuh
    // this lane's columns of the input: vector v0 + s * 32 + lane
    float x[NS][8];
    auto take = [&](const float *p, uint32_t end, bool vec) {
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            const uint32_t c = (v0 + s * 32 + lane) * 8;
            const bool mine = s * 32 + lane < len;
            const float4 u = mine ? load4(p, c, end, vec) : make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 v = mine ? load4(p, c + 4, end, vec) : make_float4(0.f, 0.f, 0.f, 0.f);
            x[s][0] = u.x, x[s][1] = u.y, x[s][2] = u.z, x[s][3] = u.w;
            x[s][4] = v.x, x[s][5] = v.y, x[s][6] = v.z, x[s][7] = v.w;
        }
    };
    if constexpr (NORM == NORM_NONE)
        take(a.in.x, a.in.cols, ((uintptr_t)a.in.x & 15) == 0);
    else
        norm.load(a.in);
    if (lane == 0)
        for (uint32_t s = early; s < late; ++s) request(s, s);
    if constexpr (NORM != NORM_NONE) {
        float *xs = reinterpret_cast<float *>(smem + a.x_at);
        norm.form(a.in, xs, a.ld, red);
        take(xs, a.ld, true);
    }
    float *part = reinterpret_cast<float *>(smem + a.part_at);
    uint32_t st = 0, parity = 0, done = 0;
    bool ok = true;
    for (uint32_t i = 0; i < todo && ok; i += kDsBatch) {
        float sum[kDsBatch];
#pragma unroll
        for (uint32_t q = 0; q < kDsBatch; ++q) {
            sum[q] = 0.f;
            if (ok && i + q < todo) {
                ok = __all_sync(0xffffffffu, bar_wait(my_bars + 8 * st, parity, &dead));
                if (ok) {
                    const uint8_t *row = smem + (warp * a.stages + st) * a.stage_bytes + lane * 16;
                    uint4 w[NS];
#pragma unroll
                    for (int s = 0; s < NS; ++s)
                        w[s] = s * 32 + lane < len ? *reinterpret_cast<const uint4 *>(row + s * 512) : make_uint4(0, 0, 0, 0);
                    float2 both = make_float2(0.f, 0.f);
#pragma unroll
                    for (int s = 0; s < NS; ++s) {
                        const uint32_t v[4] = {w[s].x, w[s].y, w[s].z, w[s].w};
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            fma2(both, __uint_as_float(v[k] << 16), __uint_as_float(v[k] & 0xffff0000u), x[s][2 * k], x[s][2 * k + 1]);
                    }
                    sum[q] = both.x + both.y;
                    ++done;
                    __syncwarp();  // the stage has been read
                    if (lane == 0 && i + q + a.stages < todo) {
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        request(i + q + a.stages, st);
                    }
                    if (++st == a.stages) {
                        st = 0;
                        parity ^= 1;
                    }
                }
            }
        }
        // over the lanes: lanes of bit 4 keep rows 2 and 3, of bit 3 the odd one of the two
        const bool hi = lane & 16, odd_row = lane & 8;
        float u = hi ? sum[2] : sum[0], v = hi ? sum[3] : sum[1];
        u += __shfl_xor_sync(0xffffffffu, hi ? sum[0] : sum[2], 16);
        v += __shfl_xor_sync(0xffffffffu, hi ? sum[1] : sum[3], 16);
        float t = odd_row ? v : u;
        t += __shfl_xor_sync(0xffffffffu, odd_row ? u : v, 8);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        const uint32_t r = i + (lane >> 3);
        if ((lane & 7) == 0 && r < todo) part[(first + r) * ks + kp] = t;
    }
    if (!ok) {  // leave no copy in flight behind
        if (lane == 0) atomicExch(a.error_word, DEV_ERR_WAIT_TIMEOUT);
        for (uint32_t i = done; i < min(todo, done + a.stages); ++i) {
            bar_drain(my_bars + 8 * st, parity);
            if (++st == a.stages) {
                st = 0;
                parity ^= 1;
            }
        }
    }
    __syncthreads();
    const uint32_t used = min(ks, (vectors + a.seg - 1) / a.seg);  // warps of a row that have columns
    auto row_sum = [&](uint32_t r) {
        float v = part[r * ks];
        for (uint32_t k = 1; k < used; ++k) v += part[r * ks + k];
        return v;
    };
    const int kind = KIND < 0 ? a.out.kind : KIND;
    const bool paired = kind == OUT_CLAMPED_GLU || kind == OUT_ROPE;
    for (uint32_t r = tid; r < n; r += kDsThreads)
        emit_row<KIND>(a.out, 0, 0, r0 + r, row_sum(r), paired && (r ^ 1u) < n ? row_sum(r ^ 1u) : 0.f,
                       r == tid ? mine : row_constants<KIND>(a.out, 0, r0 + r, a.rows));
}

namespace {

template <int NS, int NORM, int KIND>
ctox_status stream_kernel(ctox_ctx *ctx, const DenseStream &a, uint32_t grid, size_t smem) {
    static std::mutex mu;
    static std::set<int> ready;  // devices on which the kernel may use the shared memory it asks for
    {
        std::lock_guard<std::mutex> lock(mu);
        if (!ready.count(ctx->device)) {
            CTOX_CUDA(ctx, cudaFuncSetAttribute(k_dense_stream<NS, NORM, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDsRoom));
            ready.insert(ctx->device);
        }
    }
    CTOX_CUDA(ctx, launch_pdl(k_dense_stream<NS, NORM, KIND>, dim3(grid), dim3(kDsThreads), smem, ctx->stream, a));
    return CTOX_OK;
}
// The pairs that a layer stack has get a kernel of their own, others the general one of their norm.
template <int NS>
ctox_status stream_launch(ctox_ctx *ctx, const DenseStream &a, uint32_t grid, size_t smem) {
    const int kind = a.out.kind;
    if (a.in.norm == NORM_NONE)
        return kind == OUT_PLAIN ? stream_kernel<NS, NORM_NONE, OUT_PLAIN>(ctx, a, grid, smem) : stream_kernel<NS, NORM_NONE, -1>(ctx, a, grid, smem);
    if (a.in.norm == NORM_RMS)
        return kind == OUT_PLAIN         ? stream_kernel<NS, NORM_RMS, OUT_PLAIN>(ctx, a, grid, smem)
               : kind == OUT_ROPE        ? stream_kernel<NS, NORM_RMS, OUT_ROPE>(ctx, a, grid, smem)
               : kind == OUT_CLAMPED_GLU ? stream_kernel<NS, NORM_RMS, OUT_CLAMPED_GLU>(ctx, a, grid, smem)
                                         : stream_kernel<NS, NORM_RMS, -1>(ctx, a, grid, smem);
    return kind == OUT_PLAIN   ? stream_kernel<NS, NORM_LAYER, OUT_PLAIN>(ctx, a, grid, smem)
           : kind == OUT_RELU2 ? stream_kernel<NS, NORM_LAYER, OUT_RELU2>(ctx, a, grid, smem)
                               : stream_kernel<NS, NORM_LAYER, -1>(ctx, a, grid, smem);
}

// Shape of a launch; false: the matrix is not for this kernel.
bool stream_shape(const ctox_ctx *ctx, const DenseMat &w, const VecIn &in, uint32_t append, DenseStream *a, uint32_t *grid,
                  size_t *smem) {
    if (in.ws_o || (in.norm != NORM_NONE && w.ld > kDsInput * kDsThreads * 4) ||
        (size_t)w.rows * w.ld * 2 < kDenseStreamBytes || (uint32_t)ctx->sm_count <= append)
        return false;
    const uint32_t vectors = w.ld / 8;
    *grid = (uint32_t)ctx->sm_count - append;  // the CTAs that append need an SM of their own
    const uint32_t row_pairs = (w.rows + 1) / 2, most = 2 * ((row_pairs + *grid - 1) / *grid);
    const size_t x_bytes = in.norm == NORM_NONE ? 0 : (size_t)w.ld * 4;
    size_t fixed = 0;
    for (a->ks_log2 = 0;; ++a->ks_log2) {
        a->seg = (vectors + (1u << a->ks_log2) - 1) >> a->ks_log2;
        a->stage_bytes = a->seg * 16;
        fixed = x_bytes + ((size_t)(most << a->ks_log2) * 4 + 15) / 16 * 16;
        const uint32_t fit = fixed < kDsRoom ? (uint32_t)((kDsRoom - fixed) / (kDsWarps * a->stage_bytes)) : 0;
        a->stages = fit < kDsStages ? fit : kDsStages;
        const bool last = (1u << a->ks_log2) == kDsWarps;
        if (a->seg <= kDsSteps * 32 && a->stages >= 2) break;
        if (last) return false;
    }
    const size_t ring = (size_t)kDsWarps * a->stages * a->stage_bytes;
    a->x_at = (uint32_t)ring;
    a->part_at = (uint32_t)(ring + x_bytes);
    *smem = ring + fixed;
    return true;
}

}  // namespace

ctox_status launch_dense_stream(ctox_ctx *ctx, const DenseMat &w, const VecIn &in, const VecOut &out, const LatentAppend *append,
                                bool *taken) {
    DenseStream a{};
    uint32_t grid = 0;
    size_t smem = 0;
    a.append_positions = append ? 1 : 0;
    *taken = stream_shape(ctx, w, in, a.append_positions, &a, &grid, &smem);
    if (!*taken) return CTOX_OK;
    a.w = w.w;
    a.ld = w.ld;
    a.rows = w.rows;
    a.in = in;
    a.out = out;
    if (append) a.ap = *append;
    a.error_word = ctx->dev_error;
    const uint32_t steps = (a.seg + 31) / 32;
    timing_begin(ctx);
    ctox_status rc;
    if (steps <= 3)
        rc = stream_launch<3>(ctx, a, grid + a.append_positions, smem);
    else if (steps == 4)
        rc = stream_launch<4>(ctx, a, grid + a.append_positions, smem);
    else
        rc = stream_launch<5>(ctx, a, grid + a.append_positions, smem);
    if (rc) return rc;
    timing_end(ctx, KC_DENSE_MATVEC, 2.0 * w.rows * w.ld, 2.0 * w.rows * w.ld);
    return CTOX_OK;
}

}  // namespace ctox
