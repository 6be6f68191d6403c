// The packed slab block for 3x3 / padding 1 stacks (packed_slab.cu) as packed.cu and net.cu call it.
#pragma once

#include <stddef.h>
#include <stdint.h>

namespace clb {
namespace slab {
struct __align__(16) Rec {
    int4 off[4];               // tile offsets of taps 2i and 2i + 1, each for the left and the right conv column of a window
    int code[7];               // gate ids folded to 0..7 ...
    int c;                     // (output channel)
    unsigned inv[7];           // ... and their output inversion
    unsigned fresh;            // planes (bit 0: the first) that the record before does not leave in place
    int ch[2];                 // input channels of the tile's planes
    int planes, all_in_tile;   // planes to copy where no record came before
    int word[8];               // the raw selection words (global path)
};
} // namespace slab

// Order of the units of a packed activation between the stages of a network.
enum Order { kRows = 0,      // feature rows [F][U]
             kSlabs = 1,     // [C][U][H * W], pixels row-major
             kSplitSlabs = 2 // [C][U][H][W], a row's even columns before its odd ones (W even): what packed_slab.cu's tile holds
};
__host__ __device__ __forceinline__ int split_position(int pixel, int side) // side: a power of two
{
    const int col = pixel & (side - 1);
    return (pixel & ~(side - 1)) | ((col & 1) ? side >> 1 : 0) | (col >> 1);
}
} // namespace clb

// does the kernel take this block?  (U > 0 slabs of side * side units below 2^31 in all: 268 million samples of 32x32)
bool clb_slab3_covers(int H, int W, int sh, int sw, int ph, int pw, int kh, int kw);
size_t clb_slab3_record_bytes(int C);
// An order of the output channels in which neighbours share input channels: 3 ints each {channel, first plane, second plane | fresh << 16}
// (host; false: a selection that does not fit two planes, whose records keep the channels' own order)
bool clb_slab3_order(const int32_t *sel, int Ci, int C, int32_t *order);
// order: that table on the device, or null
int clb_slab3_records(const uint8_t *ops, const int32_t *sel, const int32_t *order, void *recs, int Ci, int side, int C, cudaStream_t st);
// in: kSlabs or kSplitSlabs; out: any order (kSplitSlabs: side >= 8)
int clb_slab3_block(const void *x, const void *recs, void *y, int Ci, int side, int C, int64_t U, clb::Order in, clb::Order out, cudaStream_t st);

// the input stages of packed.cu with the batch padded to U units of 128 samples; side: of the images, read for kSplitSlabs only
int clb_pack_bits_units(const uint8_t *t, void *packed, int64_t N, int64_t F, int64_t U, int64_t HW, int side, clb::Order order, cudaStream_t st);
int clb_thermometer_pack_units(const void *pixels, int pixels_u8, const float *thresholds, int levels, void *packed, int64_t N, int64_t channels, int64_t HW,
                               int64_t words, int side, clb::Order order, cudaStream_t st);
int clb_packed_rows_to_slabs(const void *rows, void *slabs, int64_t C, int64_t HW, int64_t U, int side, clb::Order order, cudaStream_t st);
// class sums over rows of U units, of whose samples the first B count
int clb_group_popcount_units(const void *x, int32_t *counts, int64_t F, int64_t U, int64_t B, int k, cudaStream_t st);
// the same over the trees of clb_packed_tree on rows of U units, without their outputs; CLB_ERR_SHAPE: run the two apart
int clb_packed_tree_count(const void *x, const int32_t *leaf, const uint8_t *ops, int32_t *counts, int64_t in_dim, int64_t out_dim, int levels, int64_t U,
                          int64_t B, int k, cudaStream_t st);
