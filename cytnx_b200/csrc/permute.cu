// Tensor permute (materialisation of a lazy permutation) for sm_100a.
//
// Semantics of the reference (src/backend/utils_internal_cpu/Movemem_cpu.cpp:152-191,
// src/backend/utils_internal_gpu/cuMovemem_gpu.cu:60-94): for a row-major tensor of
// old_shape, out has new_shape[i] = old_shape[mapper[i]] and
// out[sum_i new_stride[i] * idx_old[mapper[i]]] = in[idx_old].  Pure data movement,
// bit-exact for every dtype.
//
// B200 design: the permutation is first reduced (size-1 axes dropped, axes that stay
// adjacent merged), then one of two kernels runs:
//  * the innermost axis is preserved -> a row-gather copy in 16-byte vectors where the
//    row length and pointers allow (every warp reads and writes whole contiguous runs);
//  * otherwise a tiled transpose between the input's fastest axes and the output's
//    fastest axes, so both the HBM reads and the HBM writes are coalesced; all remaining
//    axes are batch axes decomposed per tile (k_tile_transpose).  For 1- and 2-byte
//    elements, when the input strides allow a tensor map (16-byte multiples, at most 3
//    batch axes), the tiles are staged by TMA: a persistent CTA double-buffers (128 bytes
//    of the input's fastest axis) x 128 tiles into shared memory with cp.async.bulk.tensor
//    (SWIZZLE_128B, so the column reads of the transpose spread over the banks) and
//    writes 16-byte vectors along the output's fastest axis.  A short output axis (< 16)
//    under a long input axis has a staged kernel of its own, and tensors whose tiles would be
//    mostly empty go in boxes over any axes (permute_packed.cu).
// No per-call allocation or host<->device copy of stride vectors: the reduced
// geometry travels as kernel parameters (the reference mallocs and copies two
// stride arrays per call, cuMovemem_gpu.cu:139-152).

#include <algorithm>
#include <atomic>
#include <cstring>
#include <exception>
#include <memory>
#include <mutex>
#include <vector>

#include "ctn_common.h"
#include "permute.cuh"
#include "tmap.h"

namespace ctn {

template <int N>
struct VecT;
template <>
struct VecT<1> { using T = uint8_t; };
template <>
struct VecT<2> { using T = uint16_t; };
template <>
struct VecT<4> { using T = uint32_t; };
template <>
struct VecT<8> { using T = uint64_t; };
template <>
struct VecT<16> { using T = U128; };

// ---------------------------------------------------------------- row copy
// The last new axis equals the last old axis: rows of contiguous elements on both sides, whose
// order changes.  A CTA writes ROW_THREADS * PER consecutive units (1 to 16 bytes each, whatever
// divides the rows and the base addresses).  Bound by HBM once the index arithmetic is cheap: the
// input offset of a row takes a division per outer axis, so it is computed once per row of the
// chunk, in parallel, into shared memory; a unit then takes one 32-bit division by the row length
// (a multiply-high by floor(2^32 / d) with one correction) and a look-up, and a thread issues all
// its loads before the first store.  Without the table (every unit its own divisions): small tensors, one
// unit a thread, where one unit's latency is all there is, and elements that are rows of their own, of which
// the table would hold one entry each.
// Measured, a division per axis and unit -> this (read + written TB/s): f64 [2048,4,4,1024]
// (0,2,1,3) 5.4 -> 6.6, [2047,5,3,1001] 3.0 -> 6.3; f32 [2047,5,3,1001] 1.5 -> 4.0; int16 0.8 ->
// 2.8, bool 0.4 -> 1.4 (narrow odd rows: bound by the number of element accesses).  Assembling
// 16-byte outputs from shifted input vectors was faster only for rows above 2 KB of 1- or 4-byte
// elements and up to 40 % slower for short rows of 8-byte elements.
constexpr int ROW_THREADS = 256;
constexpr int row_per(int unit) { return unit >= 16 ? 4 : unit >= 4 ? 8 : 16; }  // units per thread
constexpr int ROW_PER_DIRECT = 4;                                                // without the table

struct RowGeom {
  int n;                    // outer axes
  int64_t ext[kMaxRank];    // their extents, innermost first
  int64_t ins[kMaxRank];    // input strides (in units)
  int64_t row;              // units per row
  uint32_t rec;             // floor(2^32 / row), 2^32 - 1 for one unit per row
  int wide;                 // 64-bit row numbers
};

// input offset of a row; 32-bit divisions unless the row numbers need more
__device__ __forceinline__ int64_t row_offset(const RowGeom &g, int64_t row) {
  int64_t off = 0;
  if (!g.wide) {
    uint32_t r = (uint32_t)row;
    for (int i = 0; i + 1 < g.n; ++i) {
      const uint32_t d = (uint32_t)g.ext[i], q = r / d;
      off += (int64_t)(r - q * d) * g.ins[i];
      r = q;
    }
    return off + (int64_t)r * g.ins[g.n - 1];
  }
  for (int i = 0; i + 1 < g.n; ++i) {
    const int64_t q = row / g.ext[i];
    off += (row - q * g.ext[i]) * g.ins[i];
    row = q;
  }
  return off + row * g.ins[g.n - 1];
}

// rows of 2^31 units and more are a mode of their own: a chunk lies in at most two of them, and the columns
// take 64 bits
enum RowMode { ROW_DIRECT, ROW_TABLE, ROW_LONG };

template <typename U, int PER, int MODE>
__global__ void __launch_bounds__(ROW_THREADS) k_row_copy(const U *__restrict__ src, U *__restrict__ dst,
                                                          const __grid_constant__ RowGeom g, int64_t total) {
  extern __shared__ int64_t row_off[];
  constexpr int CHUNK = ROW_THREADS * PER;
  for (int64_t c = (int64_t)blockIdx.x * CHUNK; c < total; c += (int64_t)gridDim.x * CHUNK) {
    const int64_t r0 = g.wide ? c / g.row : (int64_t)((uint32_t)c / (uint32_t)g.row);  // first row of the chunk
    const uint32_t c0 = (uint32_t)(c - r0 * g.row);                                 // and the column it starts at
    const uint32_t cnt = (uint32_t)(total - c < CHUNK ? total - c : CHUNK);
    const uint32_t len = (uint32_t)g.row;
    auto split = [&](uint32_t x, uint32_t &col) -> uint32_t {
      uint32_t q = __umulhi(x, g.rec);
      if (x - q * len >= len) ++q;  // the estimate is short by at most one
      col = x - q * len;
      return q;
    };
    if (MODE == ROW_TABLE) {
      uint32_t last;
      const uint32_t rows = split(c0 + cnt - 1, last) + 1;
      for (uint32_t i = threadIdx.x; i < rows; i += ROW_THREADS) row_off[i] = row_offset(g, r0 + i);
      __syncthreads();
    } else if (MODE == ROW_LONG) {
      if (threadIdx.x < 2) row_off[threadIdx.x] = row_offset(g, r0 + threadIdx.x);
      __syncthreads();
    }
    U v[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const uint32_t e = threadIdx.x + i * ROW_THREADS;
      if (e < cnt) {
        if (MODE == ROW_LONG) {
          const int64_t col = c - r0 * g.row + e;
          v[i] = col < g.row ? src[row_off[0] + col] : src[row_off[1] + col - g.row];
        } else {
          uint32_t col;
          const uint32_t r = split(c0 + e, col);
          v[i] = src[(MODE == ROW_TABLE ? row_off[r] : row_offset(g, r0 + r)) + col];
        }
      }
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const uint32_t e = threadIdx.x + i * ROW_THREADS;
      if (e < cnt) dst[c + e] = v[i];
    }
    if (MODE != ROW_DIRECT) __syncthreads();  // the next chunk reuses the table
  }
}

template <typename U>
static void launch_rows(const void *src, void *dst, const RowGeom &g, int64_t total, int nsm, cudaStream_t st) {
  constexpr int PER = row_per((int)sizeof(U)), CHUNK = ROW_THREADS * PER;
  auto go = [&](auto kern, int per, size_t smem) {
    const int64_t chunk = (int64_t)ROW_THREADS * per, grid = std::min<int64_t>((total + chunk - 1) / chunk, (int64_t)1 << 30);
    kern<<<(unsigned)grid, ROW_THREADS, smem, st>>>((const U *)src, (U *)dst, g, total);
  };
  // small: below one chunk of the table's form an SM, or two where the rows are so short that it gains little
  // (int16 [4,17,1323,16] (2,1,0,3) 3.4 / 2.7 us; f32 [256,4,4,255] (0,2,1,3) 3.5 / 7.7)
  if (total < (int64_t)nsm * CHUNK * (g.row <= 2 ? 2 : 1)) go(k_row_copy<U, 1, ROW_DIRECT>, 1, 0);
  else if (g.row == 1) go(k_row_copy<U, ROW_PER_DIRECT, ROW_DIRECT>, ROW_PER_DIRECT, 0);
  else if (g.row < (int64_t)1 << 31) go(k_row_copy<U, PER, ROW_TABLE>, PER, (size_t)(CHUNK / g.row + 2) * sizeof(int64_t));
  else go(k_row_copy<U, PER, ROW_LONG>, PER, 2 * sizeof(int64_t));
}

// ---------------------------------------------------------------- tiled transpose
// Input fastest axis "a" (new position pa), output fastest axis "b" (old axis with
// input stride sb), for the staged kernel below.
struct TransGeom {
  int nbatch_dims;
  int64_t na, nb;           // sizes of axes a and b
  int64_t in_stride_b;      // input stride of axis b
  int64_t batch;            // number of batch points
  int64_t bshape[kMaxRank]; // batch axes (new order, row-major over them)
  int64_t bin[kMaxRank];    // their input strides
  int64_t bout[kMaxRank];   // their output strides
};

// General tiled transpose, any element size, strides and extents.  The reduced axes fall into
// three groups: A, contiguous in the input (the input's fastest axis and, while the product is
// below the wanted run, the axes next to it in the input), B, contiguous in the output (the
// output's fastest axis and its neighbours likewise), and the batch axes.  A CTA moves one tile
// of TA x TB elements: it reads runs of TA along A, stages them in shared memory and writes
// runs of TB along B.  Grouping axes keeps the runs long when the last axes are short (a site
// tensor's physical legs, a 37-element leg), and the tile's shape (powers of two, TA * TB = CAP)
// follows the groups' extents.  A group ends where the next axis belongs to the other one: two short innermost
// axes that are each other's neighbours leave most of a tile empty, and permute_packed takes such tensors.
// These kernels are bound by instruction issue before HBM (a 32-lane access moves 32 elements of
// a narrow type only), so a tile's shape is a compile-time constant: a row costs one offset and
// one 64-bit multiply-add, an element its load, its store and the shared-memory round trip.  All
// loads of a thread (CAP / 256 elements) are issued before the first store.  Element accesses
// throughout: nothing is asked of the alignment of rows, strides or base pointers.
// Measured (TB/s read + written), the 32 x 32 kernel this replaced -> this one: f64
// [2048,3,3,2048] reversed 5.9 -> 6.4, [2047,3,3,2045] 5.3 -> 6.1, [4000000,5] 1.6 -> 6.2; f32
// [2047,3,3,2045] 3.4 -> 5.5, [1021,3,37,509] (3,1,0,2) 1.8 -> 4.5, and the aligned
// [2048,3,3,2048], which a TMA-staged kernel moved at 4.7, 6.1; int16 ragged 0.9-1.8 -> 3.6-3.9.
constexpr int TILE_THREADS = 256;
// elements per tile, by measurement ([2048,3,3,2048] reversed): f64 1024 / 2048 elements 110 / 94
// us, f32 2048 / 4096 63 / 49 us; 16-byte elements and small tensors 1024 (four loads per thread)
constexpr int TILE_SMALL = 1024;
constexpr int tile_cap(int es) { return es == 1 ? 8192 : es <= 4 ? 4096 : es == 8 ? 2048 : 1024; }
constexpr int TILE_TA_MIN = 2, TILE_TA_MAX = 1024;  // tile widths along A (TB = CAP / TA likewise >= 2)

template <int R, typename IT>
struct TilePerm {
  int64_t src, dst;            // element offsets of the permuted block
  IT ext[R], ins[R], outs[R];  // axes: A group (innermost first), B group (innermost first), batch
  IT na, nb;                   // extents of the groups
  IT tiles_a, tiles_b;
  int8_t n_a, n_b, n_x;        // axes per group
  int8_t log_ta;               // the tile's width along A
};

// offset of index x of the group whose axes are k0 .. k0 + n - 1 (innermost first)
template <int R, typename IT>
__device__ __forceinline__ IT group_offset(const TilePerm<R, IT> &g, const IT *st, int k0, int n, IT x) {
  IT o = 0;
  for (int k = k0; k + 1 < k0 + n; ++k) {
    const IT d = g.ext[k];
    const IT q = x / d;
    o += (x - q * d) * st[k];
    x = q;
  }
  return o + x * st[k0 + n - 1];
}

template <typename T, int CAP, int TA, typename IT>
struct TileSmem {
  static constexpr int TB = CAP / TA;
  static constexpr int PITCH = tile_pitch((int)sizeof(T), TA);
  T tile[TB * PITCH];
  IT off[TA + TB];  // [0, TA): output offsets of the tile's a, [TA, TA + TB): input offsets of its b
};

template <typename T, int CAP, int TA, int R, typename IT>
__device__ __forceinline__ void tile_transpose(const TilePerm<R, IT> &g, IT t, const T *__restrict__ src,
                                               T *__restrict__ dst, void *smem) {
  using SM = TileSmem<T, CAP, TA, IT>;
  constexpr int TB = SM::TB, PITCH = SM::PITCH;
  constexpr int WA = TA < 32 ? TA : 32, HA = TA / WA, RA = TILE_THREADS / WA;  // reading: lanes along A, rows of b
  constexpr int WB = TB < 32 ? TB : 32, HB = TB / WB, RB = TILE_THREADS / WB;  // writing: lanes along B, rows of a
  constexpr int NRA = TB / RA > 0 ? TB / RA : 1, NRB = TA / RB > 0 ? TA / RB : 1;
  static_assert(NRA * HA * TILE_THREADS >= CAP && NRB * HB * TILE_THREADS >= CAP, "tile coverage");
  SM &sm = *reinterpret_cast<SM *>(smem);
  const int tid = threadIdx.x;
  IT r = t / g.tiles_a;
  const IT a0 = (t - r * g.tiles_a) * (IT)TA;
  const IT q = r / g.tiles_b;
  const IT b0 = (r - q * g.tiles_b) * (IT)TB;
  r = q;
  IT in_off = a0, out_off = b0;
  for (int i = 0; i < g.n_x; ++i) {
    const int k = g.n_a + g.n_b + i;
    const IT d = g.ext[k];
    const IT qq = i + 1 < g.n_x ? r / d : 0;
    const IT c = r - qq * d;
    in_off += c * g.ins[k];
    out_off += c * g.outs[k];
    r = qq;
  }
  const int ca = (int)(g.na - a0 < (IT)TA ? g.na - a0 : (IT)TA);
  const int cb = (int)(g.nb - b0 < (IT)TB ? g.nb - b0 : (IT)TB);
  const bool one_a = g.n_a == 1, one_b = g.n_b == 1;  // single axes: offsets are multiples of one stride
  const IT sa = g.outs[0], sb = g.ins[g.n_a];
  if (!(one_a && one_b)) {
    for (int i = tid; i < TA + TB; i += TILE_THREADS) {
      if (i < TA) sm.off[i] = one_a ? 0 : group_offset(g, g.outs, 0, g.n_a, (IT)(a0 + (IT)i));
      else sm.off[i] = one_b ? 0 : group_offset(g, g.ins, g.n_a, g.n_b, (IT)(b0 + (IT)(i - TA)));
    }
    __syncthreads();
  }
  {
    const int lane = tid % WA, row0 = tid / WA;
    const T *s = src + g.src + (int64_t)in_off + lane;
    T v[NRA][HA];
#pragma unroll
    for (int i = 0; i < NRA; ++i) {
      const int b = row0 + i * RA;
      const IT o = one_b ? (b0 + (IT)b) * sb : sm.off[TA + (TB % RA == 0 ? b : b % TB)];
#pragma unroll
      for (int h = 0; h < HA; ++h)
        if (b < cb && lane + h * WA < ca) v[i][h] = s[(int64_t)o + h * WA];
    }
#pragma unroll
    for (int i = 0; i < NRA; ++i) {
      const int b = row0 + i * RA;
#pragma unroll
      for (int h = 0; h < HA; ++h)
        if (b < cb && lane + h * WA < ca) sm.tile[b * PITCH + lane + h * WA] = v[i][h];
    }
  }
  __syncthreads();
  {
    const int lane = tid % WB, row0 = tid / WB;
    T *o = dst + g.dst + (int64_t)out_off + lane;
#pragma unroll
    for (int i = 0; i < NRB; ++i) {
      const int a = row0 + i * RB;
      const IT oo = one_a ? (a0 + (IT)a) * sa : sm.off[TA % RB == 0 ? a : a % TA];
#pragma unroll
      for (int h = 0; h < HB; ++h)
        if (a < ca && lane + h * WB < cb) o[(int64_t)oo + h * WB] = sm.tile[(lane + h * WB) * PITCH + a];
    }
  }
}

template <typename T, int CAP, int TA, typename IT>
__global__ void __launch_bounds__(TILE_THREADS) k_tile_transpose(const T *__restrict__ src, T *__restrict__ dst,
                                                                 const __grid_constant__ TilePerm<kMaxRank, IT> g,
                                                                 int64_t ntiles) {
  __shared__ __align__(16) unsigned char smem[sizeof(TileSmem<T, CAP, TA, IT>)];
  for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    tile_transpose<T, CAP, TA>(g, (IT)t, src, dst, smem);
    __syncthreads();  // the next tile reuses the stage and the offsets
  }
}

// Geometry of a reduced permutation whose innermost axis moves (reduce_perm's axes; strides in
// elements).  Groups stop growing at `want` elements.  Returns the number of tiles of `cap`
// elements.
template <int R, typename IT>
static int64_t tile_geometry(int es, int cap, int want, int r, const int64_t *rshape, const int *rmap, const int64_t *in_stride,
                             const int64_t *out_stride_of_old, TilePerm<R, IT> &g) {
  const int a = r - 1, b = rmap[r - 1];
  bool used[kMaxRank] = {false};
  int order[kMaxRank], n = 0;
  int grp_b[kMaxRank], nb = 0;
  int64_t eb = rshape[b], ea = rshape[a];
  grp_b[nb++] = b;
  used[b] = used[a] = true;
  for (int i = r - 2; i >= 0 && rmap[i] != a && eb < want; --i) {  // output neighbours of b
    grp_b[nb++] = rmap[i];
    used[rmap[i]] = true;
    eb *= rshape[rmap[i]];
  }
  order[n++] = a;
  for (int j = r - 2; j >= 0 && !used[j] && ea < want; --j) {  // input neighbours of a
    order[n++] = j;
    used[j] = true;
    ea *= rshape[j];
  }
  g.n_a = (int8_t)n;
  for (int i = 0; i < nb; ++i) order[n++] = grp_b[i];
  g.n_b = (int8_t)nb;
  int64_t batch = 1;
  for (int i = r - 1; i >= 0; --i)
    if (!used[rmap[i]]) {
      order[n++] = rmap[i];
      batch *= rshape[rmap[i]];
    }
  g.n_x = (int8_t)(n - g.n_a - g.n_b);
  for (int k = 0; k < n; ++k) {
    g.ext[k] = (IT)rshape[order[k]];
    g.ins[k] = (IT)in_stride[order[k]];
    g.outs[k] = (IT)out_stride_of_old[order[k]];
  }
  g.na = (IT)ea;
  g.nb = (IT)eb;
  // the width that covers the plane with the least work, elements (padding included) times what the
  // runs of a tile cost unless they hold their whole group.  Written runs (along b) below 256 bytes, or
  // 64 elements of the small types, leave sectors in part: per element 1.15 to 1.4 times the time at
  // half of that, 1.5 to 2 at a quarter.  Read runs (along a) below 64 bytes or 8 elements: 1.1 to 1.5 at
  // half of that (what is left of a line is still in L2 for the next tile).  Among equals (within a
  // part in 64, the last tiles of a long axis) the squarest tile.
  // f32 (33, 606061) (1, 0), fewest tiles 16 wide against 64 wide: 62.7 / 38.6 us; (68, 294117): 54.6 / 43.6.
  int64_t best = -1, best_skew = 0;
  const int64_t full_a = std::max(8, 64 / es), full_b = std::min(64, 256 / es);
  for (int l = 1; (1 << l) <= TILE_TA_MAX; ++l) {
    const int64_t ta = (int64_t)1 << l, tb = cap / ta;
    if (ta < TILE_TA_MIN || tb < TILE_TA_MIN || tb > TILE_TA_MAX) continue;
    const int64_t cost_a = ta >= ea || ta >= full_a ? 16 : 2 * ta >= full_a ? 32 : 48;
    const int64_t cost_b = tb >= eb || tb >= full_b ? 16 : 2 * tb >= full_b ? 22 : 4 * tb >= full_b ? 28 : 48;
    const int64_t cost = ((ea + ta - 1) / ta) * ((eb + tb - 1) / tb) * cost_a * cost_b;
    const int64_t skew = std::max(ta, tb) / std::min(ta, tb);
    if (best < 0 || cost < best - best / 64 || (cost <= best + best / 64 && skew < best_skew)) {
      best = cost;
      best_skew = skew;
      g.log_ta = (int8_t)l;
    }
  }
  const int64_t ta = (int64_t)1 << g.log_ta, tb = cap / ta;
  const int64_t tiles_a = (ea + ta - 1) / ta, tiles_b = (eb + tb - 1) / tb;
  g.tiles_a = (IT)tiles_a;
  g.tiles_b = (IT)tiles_b;
  return tiles_a * tiles_b * batch;
}

template <typename T, int CAP, typename IT>
static void launch_tile(const void *src, void *dst, const TilePerm<kMaxRank, IT> &g, int64_t ntiles, cudaStream_t st) {
  const unsigned grid = (unsigned)std::min<int64_t>(ntiles, (int64_t)1 << 30);
  auto go = [&](auto kern) { kern<<<grid, TILE_THREADS, 0, st>>>((const T *)src, (T *)dst, g, ntiles); };
  switch (g.log_ta) {
    case 1: if constexpr (CAP / 2 <= TILE_TA_MAX) go(k_tile_transpose<T, CAP, 2, IT>); break;
    case 2: if constexpr (CAP / 4 <= TILE_TA_MAX) go(k_tile_transpose<T, CAP, 4, IT>); break;
    case 3: if constexpr (CAP / 8 <= TILE_TA_MAX) go(k_tile_transpose<T, CAP, 8, IT>); break;
    case 4: if constexpr (CAP / 16 <= TILE_TA_MAX) go(k_tile_transpose<T, CAP, 16, IT>); break;
    case 5: go(k_tile_transpose<T, CAP, 32, IT>); break;
    case 6: go(k_tile_transpose<T, CAP, 64, IT>); break;
    case 7: go(k_tile_transpose<T, CAP, 128, IT>); break;
    case 8: go(k_tile_transpose<T, CAP, 256, IT>); break;
    case 9: go(k_tile_transpose<T, CAP, 512, IT>); break;
    default: if constexpr (CAP > 1024) go(k_tile_transpose<T, CAP, 1024, IT>); break;
  }
}

// ---------------------------------------------------------------- many blocks in one launch
// The blocks of a block-sparse tensor are permuted together: a launch per block costs 2-3 us of
// host and device time each, against well under 1 us of work for a block of a few thousand
// elements.  A CTA finds its block by a binary search over the tile counts and moves one tile of
// TILE_SMALL elements of it, with the same tiles as a single tensor's (a block's shape is known
// only at run time, so the widths are a switch here) or a run of a copied block.  The
// descriptors travel as kernel parameters: no device table to upload, so a first call can be
// captured in a graph and a prepared permutation can run on any device, stream and thread.
// Measured: 128 blocks of an XXZ wavefunction at D=1024 520 -> 17 us for the whole Python call,
// several thousand blocks of a Hubbard wavefunction 10 ms -> 58 us, the environment update that
// stages its operands this way 3.3 -> 0.19 ms.
constexpr int BLOCK_RANK = 4;     // reduced axes a descriptor holds; others take their own launch
constexpr int BLOCK_BATCH = 340;  // descriptors per launch: 32 KB of parameters
constexpr int BLOCK_BATCH_SMALL = 40;
// bytes from which a block takes its own launch: there the launch's 2-3 us are hidden, and the
// larger tiles of a single tensor move 6.4 instead of 5.4 TB/s
constexpr int64_t BLOCK_OWN_BYTES = 8 << 20;

// times a block's elements that its tiles may hold before it is copied element by element, the output
// contiguous and the input read where it lies (short innermost axes that are each other's neighbours: a warp
// then reads whole lines all the same).  60 f64 blocks, tiles / elements: [60,50,2,2] (0,1,3,2), 256 times, 448 /
// 5.8 us; [100,12,12] (0,2,1), 7 times, 17.6 / 7.4; [100,16,16], 4 times, 17.8 / 10.9; [100,24,24], 1.8 times,
// 18.1 / 18.7.
constexpr int BLOCK_SPARSE = 3;

template <int N>
struct BlockBatch {
  int32_t n;
  uint32_t tile0[N + 1];  // first tile of each block
  TilePerm<BLOCK_RANK, uint32_t> p[N];
};
static_assert(sizeof(BlockBatch<BLOCK_BATCH>) <= 32764, "kernel parameter limit");

template <typename T>
constexpr size_t block_smem() {
  size_t m = 0;
  for (int ta = 2; ta <= TILE_SMALL / 2; ta *= 2) {
    const size_t tb = TILE_SMALL / ta, pitch = tile_pitch((int)sizeof(T), ta);
    const size_t b = (tb * pitch * sizeof(T) + 15) / 16 * 16 + (ta + tb) * 4;
    m = b > m ? b : m;
  }
  return m;
}

template <typename T, int N>
__global__ void __launch_bounds__(TILE_THREADS) k_permute_blocks(const T *__restrict__ src, T *__restrict__ dst,
                                                                 const __grid_constant__ BlockBatch<N> bb) {
  __shared__ __align__(16) unsigned char smem[block_smem<T>()];
  const uint32_t tile = blockIdx.x;
  int lo = 0, hi = bb.n - 1;
  while (lo < hi) {  // last block with tile0 <= tile
    const int mid = (lo + hi + 1) >> 1;
    if (bb.tile0[mid] <= tile) lo = mid;
    else hi = mid - 1;
  }
  const TilePerm<BLOCK_RANK, uint32_t> &g = bb.p[lo];
  const uint32_t t = tile - bb.tile0[lo];
  switch (g.log_ta) {
    case 0: {  // element by element: ext[0] along the output's innermost axis, n_x axes outside it; na in all
      constexpr int PER = TILE_SMALL / TILE_THREADS;
      T v[PER];
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const uint32_t u = t * TILE_SMALL + threadIdx.x + i * TILE_THREADS;
        if (u >= g.na) break;
        uint32_t row = g.n_x ? u / g.ext[0] : 0, in = (u - row * g.ext[0]) * g.ins[0];
        for (int k = 1; k <= g.n_x; ++k) {
          const uint32_t q = k < g.n_x ? row / g.ext[k] : 0;
          in += (row - q * g.ext[k]) * g.ins[k];
          row = q;
        }
        v[i] = src[g.src + in];
      }
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const uint32_t u = t * TILE_SMALL + threadIdx.x + i * TILE_THREADS;
        if (u < g.na) dst[g.dst + u] = v[i];
      }
      break;
    }
    case 1: tile_transpose<T, TILE_SMALL, 2>(g, t, src, dst, smem); break;
    case 2: tile_transpose<T, TILE_SMALL, 4>(g, t, src, dst, smem); break;
    case 3: tile_transpose<T, TILE_SMALL, 8>(g, t, src, dst, smem); break;
    case 4: tile_transpose<T, TILE_SMALL, 16>(g, t, src, dst, smem); break;
    case 5: tile_transpose<T, TILE_SMALL, 32>(g, t, src, dst, smem); break;
    case 6: tile_transpose<T, TILE_SMALL, 64>(g, t, src, dst, smem); break;
    case 7: tile_transpose<T, TILE_SMALL, 128>(g, t, src, dst, smem); break;
    case 8: tile_transpose<T, TILE_SMALL, 256>(g, t, src, dst, smem); break;
    default: tile_transpose<T, TILE_SMALL, 512>(g, t, src, dst, smem);
  }
}

// Short output axis (nb < 16) under a long input axis (na >= 256): a CTA stages a tile of
// TA = 256 x APT consecutive a by all nb b of one batch point in shared memory.  Reads:
// nb coalesced input rows, all APT x nb loads of a thread issued together.  Writes: b follows a
// directly in the output, so the tile is ONE contiguous output run of cnt_a x nb elements,
// written in 16-byte vectors when the run starts on a 16-byte boundary (f64 [5,4000000]: 6.5
// TB/s against 6.2 in tiles; with other axes between a and b the tiles, which join short axes,
// are faster).  NB bounds nb at compile time so the staging registers stay few (occupancy
// carries the bytes in flight).
constexpr int STAGED_THREADS = 256;
// CTAs that the registers have to leave room for: without the bound the compiler took 58 registers instead of
// 40 for bool and nb 7 ([7,5000000]: 30 us against 25)
constexpr int staged_ctas(int es, int nb, int apt) {
  const int words = nb * apt * (es > 4 ? es / 4 : 1);  // a thread's staged elements
  return es <= 8 && words <= 16 ? (words <= 4 ? 8 : words <= 8 ? 7 : 6) : words <= 32 ? 4 : words <= 64 ? 2 : 1;
}

template <typename T, int NB, int APT, typename IT>
__global__ void __launch_bounds__(STAGED_THREADS, staged_ctas((int)sizeof(T), NB, APT)) k_transpose_staged(const T *__restrict__ src, T *__restrict__ dst,
                                                                     TransGeom g) {
  extern __shared__ __align__(16) unsigned char staged_smem[];
  T *tile = reinterpret_cast<T *>(staged_smem);
  constexpr int TA = STAGED_THREADS * APT;
  const int nb = (int)g.nb;
  const int tid = threadIdx.x;
  const IT tiles_a = (IT)((g.na + TA - 1) / TA);
  const IT total = (IT)((g.na + TA - 1) / TA * g.batch);
  for (IT t = blockIdx.x; t < total; t += gridDim.x) {
    IT bidx = t / tiles_a;
    const int64_t a0 = (int64_t)(t - bidx * tiles_a) * TA;
    int64_t in_off = 0, out_off = 0;
    for (int i = g.nbatch_dims - 1; i >= 0; --i) {
      const IT d = (IT)g.bshape[i];
      const IT q = bidx / d;
      const IT c = bidx - q * d;
      in_off += (int64_t)c * g.bin[i];
      out_off += (int64_t)c * g.bout[i];
      bidx = q;
    }
    const int cnt_a = (int)(g.na - a0 < TA ? g.na - a0 : TA);
    const T *s = src + in_off + a0;
    T v[APT][NB];
#pragma unroll
    for (int p = 0; p < APT; ++p)
#pragma unroll
      for (int b = 0; b < NB; ++b)
        if (b < nb && p * STAGED_THREADS + tid < cnt_a) v[p][b] = s[(int64_t)b * g.in_stride_b + p * STAGED_THREADS + tid];
    __syncthreads();  // the previous tile's writers are done reading the stage
#pragma unroll
    for (int p = 0; p < APT; ++p)
#pragma unroll
      for (int b = 0; b < NB; ++b)
        if (b < nb && p * STAGED_THREADS + tid < cnt_a) tile[(p * STAGED_THREADS + tid) * nb + b] = v[p][b];
    __syncthreads();
    const int cnt = cnt_a * nb;  // elements staged
    T *o = dst + out_off + a0 * nb;
    if (sizeof(T) < 16 && (reinterpret_cast<uintptr_t>(o) & 15) == 0) {
      constexpr int V = 16 / sizeof(T);
      const int nv = cnt / V;
      const uint4 *s4 = reinterpret_cast<const uint4 *>(tile);
      uint4 *o4 = reinterpret_cast<uint4 *>(o);
      for (int i = tid; i < nv; i += STAGED_THREADS) o4[i] = s4[i];
      for (int i = nv * V + tid; i < cnt; i += STAGED_THREADS) o[i] = tile[i];
    } else {
      for (int i = tid; i < cnt; i += STAGED_THREADS) o[i] = tile[i];
    }
  }
}

// Launches k_transpose_staged when the geometry suits it (na >= 256, nb < 16, the stage
// within 48 KB); returns false otherwise.
template <typename T, int NB>
static bool launch_staged_nb(const void *src, void *dst, const TransGeom &g, int nsm, cudaStream_t st) {
  int apt = NB <= 8 ? 2 : 1;
  if ((size_t)STAGED_THREADS * apt * g.nb * sizeof(T) > 48 * 1024) apt = 1;
  const size_t smem = (size_t)STAGED_THREADS * apt * g.nb * sizeof(T);
  if (smem > 48 * 1024) return false;
  const int64_t ta = (int64_t)STAGED_THREADS * apt;
  const int64_t total = (g.na + ta - 1) / ta * g.batch;
  const int64_t blocks = std::min<int64_t>(total, (int64_t)nsm * 64);
  const bool narrow = total + blocks < ((int64_t)1 << 32);  // 32-bit tile arithmetic
  if (apt == 2 && narrow)
    k_transpose_staged<T, NB, 2, uint32_t><<<(unsigned)blocks, STAGED_THREADS, smem, st>>>((const T *)src, (T *)dst, g);
  else if (apt == 2)
    k_transpose_staged<T, NB, 2, int64_t><<<(unsigned)blocks, STAGED_THREADS, smem, st>>>((const T *)src, (T *)dst, g);
  else if (narrow)
    k_transpose_staged<T, NB, 1, uint32_t><<<(unsigned)blocks, STAGED_THREADS, smem, st>>>((const T *)src, (T *)dst, g);
  else
    k_transpose_staged<T, NB, 1, int64_t><<<(unsigned)blocks, STAGED_THREADS, smem, st>>>((const T *)src, (T *)dst, g);
  return true;
}

template <typename T>
static bool launch_staged(const void *src, void *dst, const TransGeom &g, int nsm, cudaStream_t st) {
  if (g.na < STAGED_THREADS || g.nb >= 16 || g.nb < 2) return false;
  if (g.nb <= 2) return launch_staged_nb<T, 2>(src, dst, g, nsm, st);
  if (g.nb <= 4) return launch_staged_nb<T, 4>(src, dst, g, nsm, st);
  if (g.nb <= 8) return launch_staged_nb<T, 8>(src, dst, g, nsm, st);
  return launch_staged_nb<T, 16>(src, dst, g, nsm, st);
}

static int sm_count() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

// ---------------------------------------------------------------- TMA-staged transpose
// Tile: TA = 128 / ES elements of axis a (one 128-byte swizzle row) x TB = 128 of axis b.
// The tensor map views the input as [batch2][batch1][batch0][b][a] (a fastest); the
// shared-memory image of a box row b is 128 bytes whose 16-byte chunks are XOR-swizzled
// with (b & 7).  The 256 threads write the tile as 16-byte output vectors (16 / ES
// consecutive b of one a), TA * TB * ES / 4096 of them each.
// b rows per staged tile: 16 KB tiles (int16 4.37 -> 4.83 TB/s against 64 rows)
constexpr int TMA_TB = 128;
constexpr int TMA_THREADS = 256;
constexpr long long TMA_SPIN = 1ll << 26;  // mbarrier probes before giving up

struct TmaGeom {
  int64_t na, nb;
  int64_t tiles_a, tiles_b, batch;
  int nbatch;
  int64_t bshape[3];  // batch extents (tensor-map order: innermost first)
  int64_t bout[3];    // their output strides (elements)
  int64_t out_stride_a;
  unsigned *err;      // host memory (tma_err_word)
  long long spins;    // mbarrier probes of a tile's wait
};

__device__ __forceinline__ uint32_t smem32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// rotate a 128-bit value (little-endian words) left by `bits` (0..127)
__device__ __forceinline__ uint4 rotl128(uint4 x, int bits) {
  const int w = bits >> 5, s = bits & 31;
  if (w & 2) {
    uint32_t t = x.x; x.x = x.z; x.z = t;
    t = x.y; x.y = x.w; x.w = t;
  }
  if (w & 1) {
    const uint32_t t = x.w;
    x.w = x.z; x.z = x.y; x.y = x.x; x.x = t;
  }
  uint4 y;
  y.x = __funnelshift_l(x.w, x.x, s);
  y.y = __funnelshift_l(x.x, x.y, s);
  y.z = __funnelshift_l(x.y, x.z, s);
  y.w = __funnelshift_l(x.z, x.w, s);
  return y;
}

// IT: integer type of the tile and batch index arithmetic (32-bit when it fits)
template <int ES, typename IT>
__global__ void __launch_bounds__(TMA_THREADS) k_transpose_tma(const __grid_constant__ CUtensorMap in_map,
                                                              uint8_t *__restrict__ dst, TmaGeom g) {
  constexpr int TA = 128 / ES;
  constexpr int TILE = TMA_TB * 128;                   // bytes per staged tile
  constexpr int VEC = 16 / ES;                         // elements per output vector
  constexpr int CHUNKS = TMA_TB / VEC;                 // output vectors per a (along b)
  constexpr int AROWS = TMA_THREADS / CHUNKS;          // a rows written per pass
  __shared__ __align__(1024) uint8_t buf[2][TILE];
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ int stop;
  const IT tiles_a = (IT)g.tiles_a;
  const IT ntile = (IT)(g.tiles_a * g.tiles_b);
  const IT total = (IT)(g.tiles_a * g.tiles_b * g.batch);
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem32(&bar[0])));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem32(&bar[1])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    stop = 0;
  }
  __syncthreads();
  struct C5 {
    int x0, x1, x2, x3, x4;
  };
  auto coords = [&](IT t) -> C5 {
    IT bidx = t / ntile;
    const IT tt = t - bidx * ntile;
    const IT tb = tt / tiles_a, ta = tt - tb * tiles_a;
    C5 c{(int)(ta * TA), (int)(tb * TMA_TB), 0, 0, 0};
    if (g.nbatch > 0) {
      const IT d = (IT)g.bshape[0];
      const IT q = bidx / d;
      c.x2 = (int)(bidx - q * d);
      bidx = q;
    }
    if (g.nbatch > 1) {
      const IT d = (IT)g.bshape[1];
      const IT q = bidx / d;
      c.x3 = (int)(bidx - q * d);
      bidx = q;
    }
    if (g.nbatch > 2) c.x4 = (int)bidx;
    return c;
  };
  auto issue = [&](IT t, int slot) {
    const C5 c = coords(t);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem32(&bar[slot])), "r"(TILE)
                 : "memory");
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, "
        "%6}], [%7];" ::"r"(smem32(buf[slot])),
        "l"(reinterpret_cast<uint64_t>(&in_map)), "r"(c.x0), "r"(c.x1), "r"(c.x2), "r"(c.x3), "r"(c.x4),
        "r"(smem32(&bar[slot]))
        : "memory");
  };
  IT t = blockIdx.x;
  if (threadIdx.x == 0 && t < total) issue(t, 0);
  uint32_t phase[2] = {0, 0};
  int i = 0;
  for (; t < total; ++i, t += gridDim.x) {
    const int slot = i & 1;
    const IT tn = t + gridDim.x;
    if (threadIdx.x == 0) {
      if (tn < total) issue(tn, slot ^ 1);  // that buffer was released by the last __syncthreads
      bool ok = false;
      for (long long k = 0; k < g.spins && !ok; ++k) {
        uint32_t r;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(r)
            : "r"(smem32(&bar[slot])), "r"(phase[slot])
            : "memory");
        ok = r != 0;
      }
      if (!ok) {
        *g.err = 1u;  // seen by the host when the kernel has ended
        stop = 1;
      }
    }
    __syncthreads();
    if (stop) break;
    phase[slot] ^= 1;
    const C5 c = coords(t);
    int64_t out_base = 0;
    if (g.nbatch > 0) out_base += (int64_t)c.x2 * g.bout[0];
    if (g.nbatch > 1) out_base += (int64_t)c.x3 * g.bout[1];
    if (g.nbatch > 2) out_base += (int64_t)c.x4 * g.bout[2];
    const uint8_t *tile = buf[slot];
    // A warp covers CW output vectors (along b) of 32 / CW a rows.  Staged row bl sits at
    // bl * 128 bytes with its 16-byte chunks XOR-swizzled by (bl & 7), so the rows that the
    // CW lanes of one a row read at step e must differ in (bl & 7) to reach different
    // banks: lane ch reads its VEC rows in an order rotated by `rot` and the assembled
    // vector is rotated back in registers.  Every staged load of the warp is then one
    // shared-memory wavefront (8 distinct chunks, or lanes sharing a 32-bit word).
    constexpr int CW = CHUNKS < 8 ? CHUNKS : 8;   // output vectors per a row within a warp
    constexpr int WG = CHUNKS / CW;               // warps per a row
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ch_lo = lane % CW;
    const int ch = (warp % WG) * CW + ch_lo, ar = (warp / WG) * (32 / CW) + lane / CW;
    const int rot = VEC >= 8 ? (ch_lo * (8 / CW)) & (VEC - 1) : (ch_lo >> 1) & (VEC - 1);
#pragma unroll
    for (int a_off = 0; a_off < TA; a_off += AROWS) {
      const int al = a_off + ar;  // local a
      const int64_t ag = c.x0 + al, bg0 = c.x1 + ch * VEC;
      if (al >= TA || ag >= g.na || bg0 >= g.nb) continue;
      using T = typename VecT<ES>::T;
      union {
        T e[VEC];
        uint4 q;
      } v;
      const int byte = al * ES;
#pragma unroll
      for (int e = 0; e < VEC; ++e) {
        const int bl = ch * VEC + ((e + rot) & (VEC - 1));  // local b = staged row
        const int sw = (((byte >> 4) ^ (bl & 7)) << 4) | (byte & 15);
        v.e[e] = *reinterpret_cast<const T *>(tile + bl * 128 + sw);
      }
      v.q = rotl128(v.q, rot * ES * 8);  // element j of the vector is staged row ch * VEC + j
      T *o = reinterpret_cast<T *>(dst) + (out_base + ag * g.out_stride_a + bg0);
      const int nvalid = g.nb - bg0 < VEC ? (int)(g.nb - bg0) : VEC;
      if (nvalid == VEC && ((reinterpret_cast<uintptr_t>(o) & 15) == 0)) {
        *reinterpret_cast<uint4 *>(o) = v.q;
      } else {
        for (int e = 0; e < nvalid; ++e) o[e] = v.e[e];
      }
    }
    __syncthreads();  // this buffer may be refilled
  }
  // an early stop leaves its tile's copy in flight, and the next one's if it was issued: wait for them (bounded)
  if (threadIdx.x == 0 && stop) {
    for (int s2 = 0; s2 < 2; ++s2)
      for (long long k = 0; k < TMA_SPIN && (s2 == (i & 1) || t + gridDim.x < total); ++k) {
        uint32_t r;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(r)
            : "r"(smem32(&bar[s2])), "r"(phase[s2])
            : "memory");
        if (r) break;
      }
  }
}

// The word that a wait which ran out raises: 4 bytes of pinned host memory for the life of the process, which
// every device can write, so the host sees it without a copy or a synchronisation.  Made on first use, also
// under a stream capture (an allocation is legal there in the relaxed mode), by one thread.
static std::atomic<unsigned *> tma_word{nullptr};
static unsigned *tma_err_word() {
  unsigned *w = tma_word.load(std::memory_order_acquire);
  if (w) return w;
  static std::mutex mu;
  std::lock_guard<std::mutex> lk(mu);
  if ((w = tma_word.load(std::memory_order_acquire))) return w;
  void *p = nullptr;
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) return nullptr;
  const cudaError_t e = cudaHostAlloc(&p, sizeof(unsigned), cudaHostAllocPortable | cudaHostAllocMapped);
  cudaThreadExchangeStreamCaptureMode(&mode);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  w = static_cast<unsigned *>(p);
  *w = 0;
  tma_word.store(w, std::memory_order_release);
  return w;
}
// CTN_ERR_TIMEOUT, once, after a permutation that gave up (asynchronously, like any launch's error)
static ctn_status tma_status() {
  unsigned *w = tma_word.load(std::memory_order_acquire);
  if (w && *(volatile unsigned *)w && __atomic_exchange_n(w, 0u, __ATOMIC_RELAXED)) {
    set_error("ctn_permute: an earlier permutation gave up waiting for a staged tile; its output is incomplete");
    return CTN_ERR_TIMEOUT;
  }
  return CTN_OK;
}

// TMA path for the transpose case; returns false (nothing launched) when the geometry
// does not fit a tensor map
template <int ES>
static bool try_transpose_tma(const void *src, void *dst, int r, const int64_t *rshape, const int *rmap,
                              const int64_t *in_stride, const int64_t *out_stride, cudaStream_t st, ctn_status *res,
                              long long spins = TMA_SPIN) {
  constexpr int TA = 128 / ES;
  const int a = r - 1, b = rmap[r - 1];
  if (r - 2 > 3) return false;
  int64_t nel = 1;
  for (int i = 0; i < r; ++i) nel *= rshape[i];
  if (nel * ES < (1 << 20)) return false;  // small tensors: the plain tile kernel (no tensor map to encode)
  if ((reinterpret_cast<uintptr_t>(src) & 15) != 0) return false;
  int pa = 0;
  for (int i = 0; i < r; ++i)
    if (rmap[i] == a) pa = i;
  TmaGeom g;
  g.na = rshape[a];
  g.nb = rshape[b];
  g.out_stride_a = out_stride[pa];
  g.tiles_a = (g.na + TA - 1) / TA;
  g.tiles_b = (g.nb + TMA_TB - 1) / TMA_TB;
  g.nbatch = 0;
  g.batch = 1;
  cuuint64_t dims[5] = {1, 1, 1, 1, 1}, strides[4] = {0, 0, 0, 0};
  dims[0] = (cuuint64_t)g.na;
  dims[1] = (cuuint64_t)g.nb;
  strides[0] = (cuuint64_t)(in_stride[b] * ES);
  for (int i = r - 1; i >= 0; --i) {  // batch axes, innermost output axis first
    const int j = rmap[i];
    if (j == a || j == b) continue;
    dims[2 + g.nbatch] = (cuuint64_t)rshape[j];
    strides[1 + g.nbatch] = (cuuint64_t)(in_stride[j] * ES);
    g.bshape[g.nbatch] = rshape[j];
    g.bout[g.nbatch] = out_stride[i];
    g.nbatch++;
    g.batch *= rshape[j];
  }
  for (int i = 0; i < 1 + g.nbatch; ++i)
    if (strides[i] % 16 != 0 || strides[i] >= (1ull << 40)) return false;
  for (int i = 1 + g.nbatch; i < 4; ++i) strides[i] = strides[g.nbatch] * (cuuint64_t)dims[1 + g.nbatch];
  for (int i = 0; i < 5; ++i)
    if (dims[i] > (1ull << 31)) return false;
  if (g.tiles_a * g.tiles_b * g.batch > (1ll << 40)) return false;
  g.err = tma_err_word();
  if (!g.err) return false;
  g.spins = spins;
  CUtensorMap map;
  const cuuint32_t box[5] = {(cuuint32_t)TA, (cuuint32_t)TMA_TB, 1, 1, 1};
  const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  const CUtensorMapDataType dt = ES == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_UINT16;
  const EncodeTiledFn enc = encode_tiled();
  if (!enc) return false;
  if (enc(&map, dt, 5, const_cast<void *>(src), dims, strides, box, estr,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return false;
  const int64_t total = g.tiles_a * g.tiles_b * g.batch;
  const int64_t blocks = std::min<int64_t>(total, (int64_t)sm_count() * 8);
  if (total + 2 * blocks < ((int64_t)1 << 32))  // t and t + grid stay below 2^32
    k_transpose_tma<ES, uint32_t><<<(unsigned)blocks, TMA_THREADS, 0, st>>>(map, (uint8_t *)dst, g);
  else
    k_transpose_tma<ES, int64_t><<<(unsigned)blocks, TMA_THREADS, 0, st>>>(map, (uint8_t *)dst, g);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error("CUDA error %s in k_transpose_tma", cudaGetErrorString(e));
    *res = CTN_ERR_CUDA;
  } else {
    *res = CTN_OK;
  }
  return true;
}


// Reduce (drop size-1 axes, merge axes that stay adjacent).  Returns reduced rank.
static int reduce_perm(int rank, const uint64_t *old_shape, const uint64_t *mapper, int64_t *rshape,
                       int *rmap) {
  // keep old axes with extent > 1
  int keep_idx[kMaxRank];
  int nk = 0;
  int old_to_k[kMaxRank];
  for (int j = 0; j < rank; ++j) {
    old_to_k[j] = -1;
    if (old_shape[j] != 1) {
      old_to_k[j] = nk;
      keep_idx[nk++] = j;
    }
  }
  int64_t kshape[kMaxRank];
  for (int k = 0; k < nk; ++k) kshape[k] = (int64_t)old_shape[keep_idx[k]];
  int kmap[kMaxRank];
  int nm = 0;
  for (int i = 0; i < rank; ++i)
    if (old_to_k[mapper[i]] >= 0) kmap[nm++] = old_to_k[mapper[i]];
  // merge: old axes k and k+1 merge if k+1 immediately follows k in the new order
  int group_of[kMaxRank];
  int ng = 0;
  int64_t gshape[kMaxRank];
  for (int k = 0; k < nk; ++k) {
    bool merge = false;
    if (k > 0) {
      for (int i = 0; i + 1 < nm; ++i)
        if (kmap[i] == k - 1 && kmap[i + 1] == k) merge = true;
    }
    if (merge) {
      group_of[k] = ng - 1;
      gshape[ng - 1] *= kshape[k];
    } else {
      group_of[k] = ng;
      gshape[ng++] = kshape[k];
    }
  }
  int r = 0;
  for (int i = 0; i < nm; ++i) {
    int g = group_of[kmap[i]];
    if (r == 0 || rmap[r - 1] != g) rmap[r++] = g;
  }
  for (int g = 0; g < ng; ++g) rshape[g] = gshape[g];
  return ng;
}

template <int ES>
static ctn_status launch_perm(const void *src, void *dst, int rank, const uint64_t *old_shape,
                              const uint64_t *mapper, cudaStream_t st) {
  using T = typename VecT<ES>::T;
  int64_t n = 1;
  for (int i = 0; i < rank; ++i) n *= (int64_t)old_shape[i];
  if (n == 0) return CTN_OK;
  int64_t rshape[kMaxRank];
  int rmap[kMaxRank];
  int r = reduce_perm(rank, old_shape, mapper, rshape, rmap);
  bool ident = true;
  for (int i = 0; i < r; ++i) ident &= (rmap[i] == i);
  if (r <= 1 || ident) {
    CTN_CUDA(cudaMemcpyAsync(dst, src, (size_t)n * ES, cudaMemcpyDeviceToDevice, st));
    return CTN_OK;
  }
  int64_t in_stride[kMaxRank];
  int64_t acc = 1;
  for (int j = r - 1; j >= 0; --j) {
    in_stride[j] = acc;
    acc *= rshape[j];
  }
  int64_t out_shape[kMaxRank], out_stride[kMaxRank];
  for (int i = 0; i < r; ++i) out_shape[i] = rshape[rmap[i]];
  acc = 1;
  for (int i = r - 1; i >= 0; --i) {
    out_stride[i] = acc;
    acc *= out_shape[i];
  }
  const int nsm = sm_count();
  if (rmap[r - 1] == r - 1) {
    const int64_t L = rshape[r - 1];
    const int64_t bytes_row = L * ES;
    const uintptr_t al = reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst);
    int vb = ES;  // unit bytes
    for (int cand = 16; cand > ES; cand /= 2)
      if (bytes_row % cand == 0 && al % cand == 0) {
        vb = cand;
        break;
      }
    const int64_t unit = vb / ES, row = L / unit, total = n / unit;
    // each row is one unit: a permutation of units, whose innermost axis moves, and a tiled transpose reads
    // whole lines of them where a copy row by row takes a line for each (row copy -> this: int16
    // [4,271049,24,2] (2,0,1,3) 272 -> 42 us, f64 [512,3,3,512,2] (3,1,2,0,4) 16.2 -> 9.6, f32 [2000,2000,4] (1,0,2)
    // 31.4 -> 19.8); below 1024 units an SM the copy, one unit a thread (f64 [12,5746,2] (1,0,2) 3.6 -> 2.2)
    if (row == 1 && total >= nsm * 1024) {
      uint64_t ushape[kMaxRank], umap[kMaxRank];
      for (int i = 0; i + 1 < r; ++i) {
        ushape[i] = (uint64_t)rshape[i];
        umap[i] = (uint64_t)rmap[i];
      }
      switch (vb) {
        case 16: return launch_perm<16>(src, dst, r - 1, ushape, umap, st);
        case 8: return launch_perm<8>(src, dst, r - 1, ushape, umap, st);
        case 4: return launch_perm<4>(src, dst, r - 1, ushape, umap, st);
        default: return launch_perm<2>(src, dst, r - 1, ushape, umap, st);
      }
    }
    RowGeom g;
    g.n = 0;
    g.row = row;
    for (int i = r - 2; i >= 0; --i) {  // innermost outer axis first
      g.ext[g.n] = out_shape[i];
      g.ins[g.n++] = in_stride[rmap[i]] / unit;  // exact: multiples of a row
    }
    g.rec = g.row > 1 ? (uint32_t)((1ull << 32) / (uint64_t)g.row) : 0xFFFFFFFFu;
    g.wide = total >= ((int64_t)1 << 32) - 65536;
    switch (vb) {
      case 16: launch_rows<U128>(src, dst, g, total, nsm, st); break;
      case 8: launch_rows<uint64_t>(src, dst, g, total, nsm, st); break;
      case 4: launch_rows<uint32_t>(src, dst, g, total, nsm, st); break;
      case 2: launch_rows<uint16_t>(src, dst, g, total, nsm, st); break;
      default: launch_rows<uint8_t>(src, dst, g, total, nsm, st);
    }
    CTN_CHECK_LAUNCH();
    return CTN_OK;
  }
  // TMA staging pays for 1- and 2-byte elements ([2048,3,3,2048] reversed: int16 31 us against 38
  // us in element accesses, bool 17 against 35); for 4-byte elements the element tiles are faster
  // (49 against 64 us), and a short output axis (< 16) wastes most of a staged tile
  if (ES <= 2 && rshape[rmap[r - 1]] >= 16) {
    ctn_status res = CTN_OK;
    if (try_transpose_tma<(ES <= 2 ? ES : 2)>(src, dst, r, rshape, rmap, in_stride, out_stride, st, &res)) return res;
  }
  const int a = r - 1;        // input fastest (old axis)
  const int b = rmap[r - 1];  // old axis that is output fastest
  int pa = 0;
  for (int i = 0; i < r; ++i)
    if (rmap[i] == a) pa = i;
  // a short output axis right behind a long one: the staged tile is one run of the output
  if (rshape[b] < 16 && rshape[a] >= STAGED_THREADS && out_stride[pa] == rshape[b]) {
    TransGeom g;
    g.na = rshape[a];
    g.nb = rshape[b];
    g.in_stride_b = in_stride[b];
    g.nbatch_dims = 0;
    g.batch = 1;
    for (int i = 0; i < r; ++i) {
      const int j = rmap[i];
      if (j == a || j == b) continue;
      g.bshape[g.nbatch_dims] = rshape[j];
      g.bin[g.nbatch_dims] = in_stride[j];
      g.bout[g.nbatch_dims] = out_stride[i];
      g.nbatch_dims++;
      g.batch *= rshape[j];
    }
    if (launch_staged<T>(src, dst, g, nsm, st)) {
      CTN_CHECK_LAUNCH();
      return CTN_OK;
    }
  }
  int64_t out_stride_of_old[kMaxRank];
  for (int i = 0; i < r; ++i) out_stride_of_old[rmap[i]] = out_stride[i];
  constexpr int WANT = ES == 1 ? 128 : 64;
  // tiles that are mostly empty (short axes that are each other's neighbours, which neither group can join)
  // give way to boxes over any axes
  auto packed = [&](int64_t ntiles, int cap, int64_t na) {
    // bytes whose tiles read runs of 16 and less: a warp's access takes a line for every few bytes, twice the
    // slots' worth (bool [1653,8,2,1653,4] (0,2,4,3,1), tiles half full: 768 us, boxes 321; one thread per output row 452)
    const int64_t slots = ntiles * cap * (ES == 1 && na <= 16 ? 2 : 1);
    if (n >= nsm * PACK_MIN_PER_SM)
      return permute_packed(ES, src, dst, r, rshape, rmap, in_stride, out_stride_of_old, n, slots, nsm, st);
    if ((double)slots < FEW_RATIO * (double)n) return false;
    RowGeom g;  // few elements: each a row of its own
    g.n = r;
    g.row = 1;
    g.rec = 0xFFFFFFFFu;
    g.wide = 0;
    for (int i = 0; i < r; ++i) {
      g.ext[i] = out_shape[r - 1 - i];
      g.ins[i] = in_stride[rmap[r - 1 - i]];
    }
    launch_rows<T>(src, dst, g, n, nsm, st);
    return true;
  };
  // 32-bit index arithmetic (a division costs several times less) when every offset fits
  if (n < ((int64_t)1 << 31)) {
    TilePerm<kMaxRank, uint32_t> g;
    g.src = g.dst = 0;
    int64_t ntiles = tile_geometry(ES, tile_cap(ES), WANT, r, rshape, rmap, in_stride, out_stride_of_old, g);
    // fewer than two tiles per SM: the latency of one tile is all there is, so smaller tiles, and
    // axes joined only where a group would be very short (a joined group needs an offset table)
    const bool small = ntiles < 2 * nsm;
    if (small) ntiles = tile_geometry(ES, TILE_SMALL, 16, r, rshape, rmap, in_stride, out_stride_of_old, g);
    if (packed(ntiles, small ? TILE_SMALL : tile_cap(ES), (int64_t)g.na)) {
    } else if (small) {
      launch_tile<T, TILE_SMALL>(src, dst, g, ntiles, st);
    } else {
      launch_tile<T, tile_cap(ES)>(src, dst, g, ntiles, st);
    }
  } else {
    TilePerm<kMaxRank, uint64_t> g;
    g.src = g.dst = 0;
    const int64_t ntiles = tile_geometry(ES, tile_cap(ES), WANT, r, rshape, rmap, in_stride, out_stride_of_old, g);
    if (!packed(ntiles, tile_cap(ES), (int64_t)g.na)) launch_tile<T, tile_cap(ES)>(src, dst, g, ntiles, st);
  }
  CTN_CHECK_LAUNCH();
  return CTN_OK;
}

static ctn_status permute_impl(const void *src, void *dst, int dtype, int rank,
                               const uint64_t *old_shape, const uint64_t *mapper, cudaStream_t st) {
  const size_t es = ctn_dtype_size(dtype);
  CTN_REQUIRE(es != 0, "ctn_permute: unknown dtype %d", dtype);
  CTN_TRY(tma_status());
  CTN_REQUIRE(rank >= 0 && rank <= kMaxRank, "ctn_permute: rank %d out of range", rank);
  bool seen[kMaxRank] = {false};
  for (int i = 0; i < rank; ++i) {
    CTN_REQUIRE(mapper[i] < (uint64_t)rank && !seen[mapper[i]], "ctn_permute: invalid mapper");
    seen[mapper[i]] = true;
  }
  if (rank == 0) {
    CTN_CUDA(cudaMemcpyAsync(dst, src, es, cudaMemcpyDeviceToDevice, st));
    return CTN_OK;
  }
  switch (es) {
    case 1: return launch_perm<1>(src, dst, rank, old_shape, mapper, st);
    case 2: return launch_perm<2>(src, dst, rank, old_shape, mapper, st);
    case 4: return launch_perm<4>(src, dst, rank, old_shape, mapper, st);
    case 8: return launch_perm<8>(src, dst, rank, old_shape, mapper, st);
    case 16: return launch_perm<16>(src, dst, rank, old_shape, mapper, st);
  }
  set_error("ctn_permute: unsupported element size");
  return CTN_ERR_UNSUPPORTED;
}

// one int16 transpose whose waits give up at once
static ctn_status selftest_tma_timeout(cudaStream_t st) {
  const int64_t n = 1024, shape[2] = {n, n}, stride[2] = {n, 1};
  const int rmap[2] = {1, 0};
  CTN_TRY(tma_status());
  char *buf = nullptr;
  CTN_CUDA(cudaMalloc(&buf, 4 * n * n));
  ctn_status rc = CTN_OK;
  const bool launched = try_transpose_tma<2>(buf, buf + 2 * n * n, 2, shape, rmap, stride, stride, st, &rc, 0);
  if (cudaStreamSynchronize(st) != cudaSuccess && rc == CTN_OK) rc = CTN_ERR_CUDA;
  cudaFree(buf);
  CTN_TRY(rc);
  CTN_TRY(tma_status());
  set_error(launched ? "ctn_selftest_permute_timeout: nothing was reported" : "ctn_selftest_permute_timeout: no tensor maps here");
  return launched ? CTN_ERR_INVALID : CTN_ERR_UNSUPPORTED;
}

struct BlockPermute {
  struct Own {  // a block with a launch of its own
    int64_t src, dst;
    std::vector<uint64_t> shape;
  };
  int dtype = 0, rank = 0;
  size_t es = 0;
  std::vector<uint64_t> mapper;
  std::vector<Own> own;
  std::vector<std::unique_ptr<BlockBatch<BLOCK_BATCH>>> batches;
};

ctn_status block_permute_create(int dtype, int rank, int64_t nblocks, const uint64_t *old_shapes,
                                const int64_t *src_offs, const int64_t *dst_offs, const uint64_t *mapper,
                                BlockPermute **out) {
  const size_t es = ctn_dtype_size(dtype);
  CTN_REQUIRE(es != 0, "ctn_permute_blocks: unknown dtype %d", dtype);
  std::unique_ptr<BlockPermute> p(new BlockPermute());
  p->dtype = dtype;
  p->rank = rank;
  p->es = es;
  if (nblocks > 0) {
    CTN_REQUIRE(rank >= 0 && rank <= kMaxRank, "ctn_permute: rank %d out of range", rank);
    bool seen[kMaxRank] = {false};
    for (int i = 0; i < rank; ++i) {
      CTN_REQUIRE(mapper[i] < (uint64_t)rank && !seen[mapper[i]], "ctn_permute: invalid mapper");
      seen[mapper[i]] = true;
    }
    p->mapper.assign(mapper, mapper + rank);
  }
  for (int64_t b = 0; b < nblocks; ++b) {
    const uint64_t *shape = old_shapes + b * rank;
    int64_t n = 1;
    for (int i = 0; i < rank; ++i) n *= (int64_t)shape[i];
    if (n == 0) continue;
    int64_t rshape[kMaxRank];
    int rmap[kMaxRank];
    const int r = reduce_perm(rank, shape, mapper, rshape, rmap);
    if (nblocks == 1 || r > BLOCK_RANK || n * (int64_t)es >= BLOCK_OWN_BYTES) {
      p->own.push_back({src_offs[b], dst_offs[b], std::vector<uint64_t>(shape, shape + rank)});
      continue;
    }
    TilePerm<BLOCK_RANK, uint32_t> g{};
    int64_t in_stride[kMaxRank], out_stride_of_old[kMaxRank], acc = 1;
    for (int j = r - 1; j >= 0; --j) {
      in_stride[j] = acc;
      acc *= rshape[j];
    }
    acc = 1;
    for (int i = r - 1; i >= 0; --i) {
      out_stride_of_old[rmap[i]] = acc;
      acc *= rshape[rmap[i]];
    }
    int64_t tiles = 0;
    const bool moves = r > 1 && rmap[r - 1] != r - 1;
    if (moves) tiles = tile_geometry((int)es, TILE_SMALL, 16, r, rshape, rmap, in_stride, out_stride_of_old, g);
    if (!moves || tiles * TILE_SMALL > BLOCK_SPARSE * n) {  // rows that keep their order, or tiles mostly empty
      g.log_ta = 0;
      g.na = (uint32_t)n;
      g.n_x = (int8_t)std::max(0, r - 1);
      g.ext[0] = g.ins[0] = 1;
      for (int k = 0; k < r; ++k) {  // innermost of the output first
        g.ext[k] = (uint32_t)rshape[rmap[r - 1 - k]];
        g.ins[k] = (uint32_t)in_stride[rmap[r - 1 - k]];
      }
      tiles = (n + TILE_SMALL - 1) / TILE_SMALL;
    }
    g.src = src_offs[b];
    g.dst = dst_offs[b];
    if (p->batches.empty() || p->batches.back()->n == BLOCK_BATCH ||
        (int64_t)p->batches.back()->tile0[p->batches.back()->n] + tiles >= ((int64_t)1 << 31)) {
      p->batches.emplace_back(new BlockBatch<BLOCK_BATCH>());
      p->batches.back()->n = 0;
      p->batches.back()->tile0[0] = 0;
    }
    BlockBatch<BLOCK_BATCH> &bb = *p->batches.back();
    bb.p[bb.n] = g;
    bb.tile0[bb.n + 1] = bb.tile0[bb.n] + (uint32_t)tiles;
    ++bb.n;
  }
  *out = p.release();
  return CTN_OK;
}

template <typename T>
static ctn_status launch_batches(const BlockPermute &p, const void *src, void *dst, cudaStream_t st) {
  for (const auto &b : p.batches) {
    const unsigned grid = b->tile0[b->n];
    if (b->n <= BLOCK_BATCH_SMALL) {  // few blocks: 4 KB of parameters
      BlockBatch<BLOCK_BATCH_SMALL> s;
      s.n = b->n;
      std::copy(b->tile0, b->tile0 + b->n + 1, s.tile0);
      std::copy(b->p, b->p + b->n, s.p);
      k_permute_blocks<T, BLOCK_BATCH_SMALL><<<grid, TILE_THREADS, 0, st>>>((const T *)src, (T *)dst, s);
    } else {
      k_permute_blocks<T, BLOCK_BATCH><<<grid, TILE_THREADS, 0, st>>>((const T *)src, (T *)dst, *b);
    }
    CTN_CHECK_LAUNCH();
  }
  return CTN_OK;
}

ctn_status block_permute_run(const BlockPermute &p, const void *src, void *dst, cudaStream_t st) {
  CTN_TRY(tma_status());
  for (const auto &o : p.own)
    CTN_TRY(permute_impl((const char *)src + o.src * p.es, (char *)dst + o.dst * p.es, p.dtype, p.rank, o.shape.data(),
                         p.mapper.data(), st));
  switch (p.es) {
    case 1: return launch_batches<uint8_t>(p, src, dst, st);
    case 2: return launch_batches<uint16_t>(p, src, dst, st);
    case 4: return launch_batches<uint32_t>(p, src, dst, st);
    case 8: return launch_batches<uint64_t>(p, src, dst, st);
    default: return launch_batches<U128>(p, src, dst, st);
  }
}

void block_permute_destroy(BlockPermute *p) { delete p; }

}  // namespace ctn

extern "C" ctn_status ctn_permute(const void *src, void *dst, int dtype, int rank,
                                  const uint64_t *old_shape, const uint64_t *mapper, void *stream) {
  return ctn::permute_impl(src, dst, dtype, rank, old_shape, mapper, ctn::as_stream(stream));
}

extern "C" ctn_status ctn_selftest_permute_timeout(void *stream) { return ctn::selftest_tma_timeout(ctn::as_stream(stream)); }

// the descriptors' memory may not be there: a status, not an exception across the C boundary
template <class F>
static ctn_status no_throw(F f) {
  try {
    return f();
  } catch (const std::exception &e) {
    ctn::set_error("ctn_permute_blocks: %s", e.what());
    return CTN_ERR_INVALID;
  }
}

extern "C" ctn_status ctn_permute_blocks(const void *src, void *dst, int dtype, int rank,
                                         int64_t nblocks, const uint64_t *old_shapes,
                                         const int64_t *src_offs, const int64_t *dst_offs,
                                         const uint64_t *mapper, void *stream) {
  return no_throw([&]() -> ctn_status {
    ctn::BlockPermute *p = nullptr;
    CTN_TRY(ctn::block_permute_create(dtype, rank, nblocks, old_shapes, src_offs, dst_offs, mapper, &p));
    const std::unique_ptr<ctn::BlockPermute, void (*)(ctn::BlockPermute *)> own(p, ctn::block_permute_destroy);
    return ctn::block_permute_run(*p, src, dst, ctn::as_stream(stream));
  });
}

struct ctn_permute_plan {
  ctn::BlockPermute *p = nullptr;
  ~ctn_permute_plan() { ctn::block_permute_destroy(p); }
};

extern "C" ctn_status ctn_permute_plan_create(int dtype, int rank, int64_t nblocks, const uint64_t *old_shapes,
                                              const int64_t *src_offs, const int64_t *dst_offs,
                                              const uint64_t *mapper, ctn_permute_plan **plan) {
  CTN_REQUIRE(plan, "ctn_permute_plan_create: null argument");
  return no_throw([&]() -> ctn_status {
    std::unique_ptr<ctn_permute_plan> h(new ctn_permute_plan());
    CTN_TRY(ctn::block_permute_create(dtype, rank, nblocks, old_shapes, src_offs, dst_offs, mapper, &h->p));
    *plan = h.release();
    return CTN_OK;
  });
}
extern "C" ctn_status ctn_permute_plan_run(const ctn_permute_plan *plan, const void *src, void *dst, void *stream) {
  CTN_REQUIRE(plan, "ctn_permute_plan_run: null plan");
  return ctn::block_permute_run(*plan->p, src, dst, ctn::as_stream(stream));
}
extern "C" void ctn_permute_plan_destroy(ctn_permute_plan *plan) { delete plan; }
