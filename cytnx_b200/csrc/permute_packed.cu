// Permutation in boxes over any axes (the "packed" tiles), for the tensors whose input and output runs share axes.
#include <algorithm>

#include "ctn_common.h"
#include "permute.cuh"

namespace ctn {

// ---------------------------------------------------------------- packed tiles
// The tiles above need the input's run and the output's run to be made of different axes.  Where the
// two innermost axes are neighbours (physical legs swapped, [N, 2, 2] (0, 2, 1)) neither group can
// grow past the other, every batch point is a tile of its own and most of its slots stay empty.
// Here a tile is a box over any axes: those that make up a run of the input, those that make up a run
// of the output, and as much of the next ones as the stage holds, whichever side they lie on.
// Thread i handles elements i, i + 256, ... of the box, in the input's order when it reads and in the
// output's order when it writes; what that takes (two offsets inside the box, two places in the stage)
// is the same for every tile, so a CTA works it out once, keeps it in registers and walks over many
// tiles, for which only the box's origin changes.  At most one axis a side is cut into chunks; the
// last chunk of an axis is told from the others by the element's coordinate along it.
// Bound by HBM for elements of 8 bytes and more, by instruction issue below (one element per lane).
// Measured, tiles of k_tile_transpose -> boxes (the kernel that moved such tensors before the tiles did, one
// thread per output row): [2048,2048,2,2] (0,1,3,2) f64 10220 -> 50 us (124), f32 13290 -> 32 (104), bool
// 25700 -> 27 (109); f32 [940,249,5,7] (0,1,3,2) 743 -> 16 (26), [600,1997,4,4,3] (3,1,0,4,2) 4510 -> 118
// (262), [200000,24,24] (0,2,1) 652 -> 210 (420).
// Registers, not threads, carry the bytes in flight: two or three CTAs an SM without spills beat three or four
// with them (50 against 66 us for the first of these); a grid of the resident CTAs, so that the set-up is paid once.
constexpr int PACK_THREADS = 256;
constexpr int pack_per(int es) { return es >= 16 ? 4 : 8; }     // elements per thread
constexpr int pack_ctas(int es) { return es == 8 ? 2 : 3; }     // resident CTAs per SM (registers)
// elements of 4 bytes and less below this many an SM: two a thread, eight CTAs an SM (a box's latency is most of
// the time: bool [5,16,17,25,25] (1,3,2,4,0) 8.6 -> 6.3 us, f32 [183,4,7,4,33] (1,3,0,4,2) 7.4 -> 5.9; 8-byte
// elements, f64 [4000,20,20] (0,2,1), 6.7 -> 7.2)
constexpr int64_t PACK_SMALL_PER_SM = 16384;
constexpr int PACK_WHOLE = 1 << 30;
// Boxes are taken where the tiles would hold PACK_RATIO times their slots, boxes that an axis's end cuts
// counted 1 + PACK_CUT times (coordinates are worked out for each of their elements).  Over 80 drawn shapes, tiles /
// boxes: f64 [200000,24,24], 3.0 times, 537 / 334 us; int16 [12,24,16,1522,5] (2,4,0,3,1), 1.6 times, 82 / 68; f32
// [30000,48,48], 1.0 times, 111 / 187; f64 [8000,65,65], 0.4 times (two axes cut), 120 / 239.
constexpr double PACK_RATIO = 1.5, PACK_CUT = 2.0;

// x / d for x below 2^16 and d from 2 to 2^16 / 2: the high word of x * (2^32 / d + 1)
struct SmallDiv {
  uint32_t d, m;
};
static SmallDiv small_div(int d) { return {(uint32_t)d, (uint32_t)((1ull << 32) / (uint64_t)d) + 1}; }
__host__ __device__ __forceinline__ uint32_t quotient(const SmallDiv &s, uint32_t x) {
  return (uint32_t)(((uint64_t)x * s.m) >> 32);
}

// one axis of the box in an enumeration of its elements
template <typename IT>
struct PackAxis {
  SmallDiv te;     // its extent in the box
  IT stride;       // in the tensor that the enumeration follows
  uint32_t place;  // in the stage
};

template <typename IT>
struct PackPerm {
  int n_t, n_x, n_s;          // axes of the box, batch axes, axes cut into chunks that do not divide them (at most 2)
  int vol, smem;              // elements of the box and of the stage
  PackAxis<IT> in[kMaxRank];  // innermost of the input first
  PackAxis<IT> out[kMaxRank];  // innermost of the output first
  IT bext[kMaxRank], bin[kMaxRank], bout[kMaxRank];  // batch axes, innermost of the output first
  struct Cut {
    int batch, te;                // its batch axis, its chunk
    IT ext;
    SmallDiv in_step, out_step;  // elements per step of the axis in the two enumerations (d == 1: every element)
    SmallDiv mod;
  } cut[2];
};

template <typename IT>
struct PackOrigin {
  IT in, out;
  int lim[2];  // what is left along the cut axes, PACK_WHOLE for a whole chunk
};

template <typename IT>
__host__ __device__ __forceinline__ PackOrigin<IT> pack_origin(const PackPerm<IT> &g, IT t) {
  PackOrigin<IT> p{0, 0, {PACK_WHOLE, PACK_WHOLE}};
  for (int k = 0; k < g.n_x; ++k) {
    const IT d = g.bext[k];
    const IT q = k + 1 < g.n_x ? t / d : 0;
    const IT c = t - q * d;
    p.in += c * g.bin[k];
    p.out += c * g.bout[k];
    t = q;
    for (int s = 0; s < 2; ++s)
      if (s < g.n_s && g.cut[s].batch == k) {
        const IT left = g.cut[s].ext - c * (IT)g.cut[s].te;
        p.lim[s] = left < (IT)g.cut[s].te ? (int)left : PACK_WHOLE;
      }
  }
  return p;
}

// offsets inside the box and places in the stage of elements x0, x0 + 256, ... of an enumeration
template <int PER, typename IT>
__host__ __device__ __forceinline__ void pack_elements(const PackAxis<IT> (&axes)[kMaxRank], int n_t, int x0, IT (&off)[PER],
                                                       uint32_t (&place)[PER]) {
  uint32_t x[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    x[i] = (uint32_t)(x0 + i * PACK_THREADS);
    off[i] = 0;
    place[i] = 0;
  }
#pragma unroll 1
  for (int k = 0; k < n_t; ++k) {
    const PackAxis<IT> a = axes[k];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const uint32_t q = quotient(a.te, x[i]), c = x[i] - q * a.te.d;
      off[i] += (IT)c * a.stride;
      place[i] += c * a.place;
      x[i] = q;
    }
  }
}

// whether element x of an enumeration (the input's or the output's) lies inside a tile cut by the end of an axis
template <bool OUT, typename IT>
__host__ __device__ __forceinline__ bool pack_inside(const PackPerm<IT> &g, const PackOrigin<IT> &p, int x) {
  bool ok = true;
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    if (p.lim[s] == PACK_WHOLE) continue;
    const SmallDiv &step = OUT ? g.cut[s].out_step : g.cut[s].in_step;
    const uint32_t y = step.d == 1 ? (uint32_t)x : quotient(step, (uint32_t)x);
    ok = ok && (int)(y - quotient(g.cut[s].mod, y) * g.cut[s].mod.d) < p.lim[s];
  }
  return ok;
}

template <typename T, int PER, int CTAS, typename IT>
__global__ void __launch_bounds__(PACK_THREADS, CTAS) k_tile_packed(const T *__restrict__ src, T *__restrict__ dst,
                                                                    const __grid_constant__ PackPerm<IT> g, int64_t ntiles) {
  extern __shared__ __align__(16) unsigned char pack_smem[];
  T *stage = reinterpret_cast<T *>(pack_smem);
  __shared__ PackOrigin<IT> origin[2];
  const int tid = threadIdx.x;
  int64_t t = blockIdx.x;
  if (t >= ntiles) return;
  if (tid < 2) origin[tid] = pack_origin(g, (IT)(t + tid * (int64_t)gridDim.x));
  IT in_off[PER], out_off[PER];
  uint32_t place[PER];  // in the stage: where the element is read << 16 | where it is written
  {
    uint32_t w[PER];
    pack_elements<PER>(g.in, g.n_t, tid, in_off, w);
    pack_elements<PER>(g.out, g.n_t, tid, out_off, place);
#pragma unroll
    for (int i = 0; i < PER; ++i) place[i] = place[i] << 16 | (w[i] & 0xFFFF);
  }
  T v[PER] = {};
  auto load = [&](const PackOrigin<IT> &p) {
    const T *s = src + (int64_t)p.in;
    const bool whole = p.lim[0] == PACK_WHOLE && p.lim[1] == PACK_WHOLE;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int x = tid + i * PACK_THREADS;
      if (x < g.vol && (whole || pack_inside<false>(g, p, x))) v[i] = s[(int64_t)in_off[i]];
    }
  };
  __syncthreads();
  PackOrigin<IT> cur = origin[0];
  load(cur);
  for (int slot = 0; t < ntiles; slot ^= 1) {
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int x = tid + i * PACK_THREADS;
      if (x < g.vol) stage[place[i] & 0xFFFF] = v[i];  // past a cut axis's end: anything, and not read
    }
    __syncthreads();
    t += gridDim.x;
    const PackOrigin<IT> next = origin[slot ^ 1];
    if (t < ntiles) load(next);  // in flight while this tile is written
    if (tid == 0) origin[slot] = pack_origin(g, (IT)(t + gridDim.x));
    T *o = dst + (int64_t)cur.out;
    const bool whole = cur.lim[0] == PACK_WHOLE && cur.lim[1] == PACK_WHOLE;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int x = tid + i * PACK_THREADS;
      if (x < g.vol && (whole || pack_inside<true>(g, cur, x))) o[(int64_t)out_off[i]] = stage[place[i] >> 16];
    }
    cur = next;
    __syncthreads();  // the stage and the origin's slot are free
  }
}

// The box for a reduced permutation, at most `cap` elements: the side with the shorter run takes its next
// axis, by doubling, until the box is full.  Returns the number of boxes.
template <typename IT>
static int64_t pack_geometry(int es, int cap, int r, const int64_t *rshape, const int *rmap, const int64_t *in_stride,
                             const int64_t *out_stride_of_old, PackPerm<IT> &g) {
  int64_t te[kMaxRank], vol = 1;
  for (int j = 0; j < r; ++j) te[j] = 1;
  int in_order[kMaxRank], out_order[kMaxRank];  // innermost first
  for (int i = 0; i < r; ++i) {
    in_order[i] = r - 1 - i;
    out_order[i] = rmap[r - 1 - i];
  }
  bool done[2] = {false, false};
  while (!done[0] || !done[1]) {
    int64_t run[2];
    int cand[2];
    for (int s = 0; s < 2; ++s) {
      const int *order = s ? out_order : in_order;
      int i = 0;
      run[s] = 1;
      while (i < r && te[order[i]] == rshape[order[i]]) run[s] *= rshape[order[i++]];
      cand[s] = i < r ? order[i] : -1;
      if (i < r) run[s] *= te[order[i]];
      else done[s] = true;
    }
    if (done[0] && done[1]) break;
    const int s = done[0] ? 1 : done[1] ? 0 : run[1] < run[0];
    const int j = cand[s];
    const int64_t rest = vol / te[j], grown = std::min(std::min(rshape[j], 2 * te[j]), (int64_t)cap / rest);
    if (grown <= te[j]) {
      done[s] = true;
      continue;
    }
    te[j] = grown;
    vol = rest * grown;
  }
  vol = 1;
  for (int j = 0; j < r; ++j) {  // equal chunks
    const int64_t chunks = (rshape[j] + te[j] - 1) / te[j];
    te[j] = (rshape[j] + chunks - 1) / chunks;
    vol *= te[j];
  }
  g.vol = (int)vol;
  // places in the stage: the input's order, its innermost runs padded
  uint32_t place[kMaxRank], in_step[kMaxRank], out_step[kMaxRank], step = 1, at = 1;
  g.n_t = 0;
  for (int i = 0; i < r; ++i) {
    const int j = in_order[i];
    if (te[j] == 1) continue;
    place[j] = at;
    in_step[j] = step;
    at *= g.n_t == 0 ? (uint32_t)tile_pitch(es, (int)te[j]) : (uint32_t)te[j];
    step *= (uint32_t)te[j];
    g.in[g.n_t++] = {small_div((int)te[j]), (IT)in_stride[j], place[j]};
  }
  g.smem = (int)at;
  int n = 0;
  step = 1;
  for (int i = 0; i < r; ++i) {
    const int j = out_order[i];
    if (te[j] == 1) continue;
    g.out[n++] = {small_div((int)te[j]), (IT)out_stride_of_old[j], place[j]};
    out_step[j] = step;
    step *= (uint32_t)te[j];
  }
  int64_t ntiles = 1;
  g.n_x = g.n_s = 0;
  for (int i = 0; i < r; ++i) {
    const int j = out_order[i];
    const int64_t chunks = (rshape[j] + te[j] - 1) / te[j];
    if (chunks == 1) continue;
    if (rshape[j] % te[j] != 0)
      g.cut[g.n_s++] = {g.n_x, (int)te[j], (IT)rshape[j], small_div((int)in_step[j]), small_div((int)out_step[j]),
                        small_div((int)te[j])};
    g.bext[g.n_x] = (IT)chunks;
    g.bin[g.n_x] = (IT)(te[j] * in_stride[j]);
    g.bout[g.n_x++] = (IT)(te[j] * out_stride_of_old[j]);
    ntiles *= chunks;
  }
  return ntiles;
}

template <typename T, int ES, int PER, int CTAS, typename IT>
static bool launch_packed(const void *src, void *dst, int r, const int64_t *rshape, const int *rmap, const int64_t *in_stride,
                          const int64_t *out_stride_of_old, int64_t tile_slots, int nsm, cudaStream_t st) {
  PackPerm<IT> g;
  const int64_t boxes = pack_geometry(ES, PACK_THREADS * PER, r, rshape, rmap, in_stride, out_stride_of_old, g);
  double whole = 1.0;  // share of the boxes that no axis cuts
  for (int s = 0; s < g.n_s; ++s) whole *= 1.0 - 1.0 / (double)g.bext[g.cut[s].batch];
  const double cost = (double)boxes * PACK_THREADS * PER * (1.0 + PACK_CUT * (1.0 - whole));
  if ((double)tile_slots < PACK_RATIO * cost) return false;
  const unsigned grid = (unsigned)std::min<int64_t>(boxes, (int64_t)nsm * CTAS);
  k_tile_packed<T, PER, CTAS, IT><<<grid, PACK_THREADS, (size_t)g.smem * sizeof(T), st>>>((const T *)src, (T *)dst, g, boxes);
  return true;
}

template <typename T, int ES>
static bool packed(const void *src, void *dst, int r, const int64_t *rshape, const int *rmap, const int64_t *in_stride,
                   const int64_t *out_stride_of_old, int64_t n, int64_t tile_slots, int nsm, cudaStream_t st) {
  constexpr int PER = pack_per(ES), CTAS = pack_ctas(ES);
  auto go = [&](auto launch) { return launch(src, dst, r, rshape, rmap, in_stride, out_stride_of_old, tile_slots, nsm, st); };
  if (n >= (int64_t)1 << 31) return go(launch_packed<T, ES, PER, CTAS, uint64_t>);
  if constexpr (ES <= 4)
    if (n < nsm * PACK_SMALL_PER_SM) return go(launch_packed<T, ES, 2, 8, uint32_t>);
  return go(launch_packed<T, ES, PER, CTAS, uint32_t>);
}

bool permute_packed(int es, const void *src, void *dst, int r, const int64_t *rshape, const int *rmap,
                    const int64_t *in_stride, const int64_t *out_stride_of_old, int64_t n, int64_t tile_slots, int nsm,
                    cudaStream_t st) {
  if ((double)tile_slots < PACK_RATIO * (double)n) return false;
  auto go = [&](auto f) { return f(src, dst, r, rshape, rmap, in_stride, out_stride_of_old, n, tile_slots, nsm, st); };
  switch (es) {
    case 1: return go(packed<uint8_t, 1>);
    case 2: return go(packed<uint16_t, 2>);
    case 4: return go(packed<uint32_t, 4>);
    case 8: return go(packed<uint64_t, 8>);
    default: return go(packed<U128, 16>);
  }
}

}  // namespace ctn
