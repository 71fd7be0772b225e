// Permutation of many blocks prepared once (permute.cu): the same mapper for every block, blocks
// of any shape at element offsets of the source and the destination.
#pragma once
#include "ctn_common.h"

namespace ctn {
struct BlockPermute;
ctn_status block_permute_create(int dtype, int rank, int64_t nblocks, const uint64_t *old_shapes,
                                const int64_t *src_offs, const int64_t *dst_offs, const uint64_t *mapper,
                                BlockPermute **out);
// enqueues the launches on `st`; holds no device state, so any thread, stream and device may run it
ctn_status block_permute_run(const BlockPermute &p, const void *src, void *dst, cudaStream_t st);
void block_permute_destroy(BlockPermute *p);
}  // namespace ctn
