// What the permute kernels share, and the permutation of many blocks prepared once (permute.cu): the same
// mapper for every block, blocks of any shape at element offsets of the source and the destination.
#pragma once
#include "ctn_common.h"

namespace ctn {

constexpr int kMaxRank = 16;

struct alignas(16) U128 {
  uint64_t a, b;
};

// staged row pitch in elements: an odd number of 32-bit words (wider types: odd), so that the
// column reads of consecutive rows fall on different banks
constexpr int tile_pitch(int es, int ta) {
  return es >= 4 ? (ta | 1) : es == 2 ? (ta % 4 == 0 ? ta + 2 : ta) : (ta % 8 == 0 ? ta + 4 : ta);
}

// Boxes over any axes are taken from this many elements an SM on.  Fewer elements go one by one where the tiles
// would hold more than FEW_RATIO times their slots: whole rows of divisions but no set-up (f64 [256,256,2,2]
// (0,1,3,2) 3.5 -> 3.1 us, bool [7,151,17,31] (1,0,3,2) 6.6 -> 5.4; at [1000,1000,2,2], 27000 an SM, 18 against 12).
constexpr int64_t PACK_MIN_PER_SM = 4096;
constexpr double FEW_RATIO = 3.3;

// permute_packed.cu: a reduced permutation of rank r (axes merged, innermost moving; strides in elements, those
// of the output by old axis) of n elements of `es` bytes, whose tiles would have tile_slots slots.  False,
// with nothing launched, where the tiles are the better choice.
bool permute_packed(int es, const void *src, void *dst, int r, const int64_t *rshape, const int *rmap,
                    const int64_t *in_stride, const int64_t *out_stride_of_old, int64_t n, int64_t tile_slots, int nsm,
                    cudaStream_t st);

struct BlockPermute;
ctn_status block_permute_create(int dtype, int rank, int64_t nblocks, const uint64_t *old_shapes,
                                const int64_t *src_offs, const int64_t *dst_offs, const uint64_t *mapper,
                                BlockPermute **out);
// enqueues the launches on `st`; holds no device state, so any thread, stream and device may run it
ctn_status block_permute_run(const BlockPermute &p, const void *src, void *dst, cudaStream_t st);
void block_permute_destroy(BlockPermute *p);
}  // namespace ctn
