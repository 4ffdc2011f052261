// Tensor-core product of a prepared packed matrix with many positions (passes of the hybrid model that are
// longer than the streaming matvec takes).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "matvec.cuh"

namespace ctox {

// Activations of a long pass: fp16 parts of x * s_in / unit, hi and 2^kLoShift times what hi leaves (lo), as [block of 64 columns][part: hi, lo][position]
// [128 bytes]. The columns of a row are in the slot order of inv_perm (layout.cuh), its 16-byte chunks XOR-swizzled by
// position & 7, so that any run of positions that starts at a multiple of eight is a ready shared-memory operand and one
// contiguous copy. The unit is a power of two: one per position, or one per block where the position is marked as
// `spread` (some block lies so far below the row's largest value that the row's unit would cost it bits).
struct LongIn {
    uint8_t *x;
    float *unit;          // [position]
    float *block_unit;    // [block][pos_pad]: of every position; kUnitTail more are read
    uint8_t *spread;      // [position]; kUnitTail more are read
    uint32_t pos_pad;  // positions of a block's row of the buffer (a multiple of eight): those of the pass and a tile
};
constexpr uint32_t kLongPosTile = 256;  // widest tile of positions
constexpr uint32_t kUnitTail = 128, kLoShift = 11;
inline size_t long_in_bytes(uint32_t blocks_padded, uint32_t pos_pad) { return (size_t)blocks_padded * 2 * pos_pad * 128; }

// Output of such a product: `splits` partial sums [position][rows], to be added up in index order.
struct LongOut {
    float *y;
    uint32_t rows, splits;
    size_t split_stride;  // floats between two partial sums
};

// Makes the kernels ready on the context's device; *usable: false where this build's kernels do not have the registers that
// their warps share out.
ctox_status packed_gemm_init(ctox_ctx *ctx, bool *usable);
// y = W x for m positions; rows row0 .. row_end only (row0 rounded down to a tile of 128). `capacity`: floats
// behind y. Recovery scales are applied; the result is in *out.
ctox_status launch_packed_gemm(ctox_matvec *mv, const LongIn &in, uint32_t m, uint64_t row0, uint64_t row_end, float *y,
                               size_t capacity, LongOut *out);

}  // namespace ctox
