// Grouped FP64 GEMM on the B200 FP64 tensor pipe (DMMA, mma.sync m16n8k16 .f64).
//
// One launch computes every output block of a block-sparse contraction:
//   C_t = sum_{p in pairs(t)} op(A_p) * op(B_p)     (row-major C_t, m_t x n_t)
// which is what BlockUniTensor::contract issues as one Matmul (non-MKL build,
// src/BlockUniTensor.cpp:1180-1223) or one Gemm_Batch group entry (MKL build,
// :1114-1177) per block pair; the reference's GPU Gemm_Batch is a serial loop of
// cublasDgemm calls (src/backend/linalg_internal_gpu/cuGemm_Batch_internal.cu:23-64).
// Here a CTA owns one tile (64x64, 64x32 or 32x32) of one output block and walks the whole K range of
// all its pairs, so every output element is written exactly once (no atomics, no
// zero-fill pass; tasks with no pair write zeros, matching Init's zeros blocks).
// Operands are read in place from the block storage with per-pair leading
// dimensions and an optional transpose, staged through shared memory by a
// 2-stage cp.async pipeline.  FP64 has no tcgen05 kind, so the legacy-warp DMMA
// instruction is the FP64 tensor path on sm_100a.
#include <algorithm>
#include <vector>

#include "ctn_common.h"
#include "gemm_f64.cuh"

namespace ctn {

namespace {
constexpr int BK = F64_BK;  // k depth of a stage; tiles are BM x BN = 64 x 64, 64 x 32 or 32 x 32
constexpr int PAD = 4;
constexpr int NTHREADS = 128;

// 8 bytes global -> shared (a shared-window address); cp_async8_zfill copies nothing and writes
// zeros when `bytes` is 0
__device__ __forceinline__ void cp_async8(uint32_t smem, const void *gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(smem), "l"(gmem));
}
__device__ __forceinline__ void cp_async8_zfill(uint32_t smem, const void *gmem, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(smem), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// D(16x8) += A(16x16) B(16x8), FP64, one warp.  Fragments (groupID g = lane/4,
// t = lane%4): a[i] = A[g + 8*(i&1)][t + 4*(i>>1)], b[i] = B[t + 4*i][g],
// c[0..1] = C[g][2t..2t+1], c[2..3] = C[g+8][2t..2t+1].
__device__ __forceinline__ void dmma_16x8x16(double (&c)[4], const double (&a)[8], const double (&b)[4]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7,%8,%9,%10,%11}, "
      "{%12,%13,%14,%15}, {%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]), "d"(b[0]),
        "d"(b[1]), "d"(b[2]), "d"(b[3]));
}

// Shared-memory tiles keep the operand's contiguous global axis contiguous, so the
// cp.async writes are conflict-free; the +4 double padding makes every fragment read
// pattern below conflict-free as well (bank = 8*x + 2*y for the 4x4 lanes of a phase).
template <bool TA, bool TB, int BM, int BN>
struct SmemT {
  double A[2][TA ? BK : BM][(TA ? BM : BK) + PAD];
  double B[2][TB ? BN : BK][(TB ? BK : BN) + PAD];
};

// One operand's side of the load cursor: this thread's share of the W x BK slices of the current
// pair.  KC: k is the contiguous axis of the source (and of the stage), else the rows are.  All that
// does not change from slice to slice is set up once per pair, so that an element costs its copy
// and one 64-bit add: the loads' index arithmetic (20 instructions an element) was three quarters
// of the instructions of the main loop and kept the DMMA pipe at 76 %.
template <bool KC, int W, int PITCH>
struct SliceCursor {
  static constexpr int LINE = KC ? BK : W;          // contiguous elements of a line of the stage
  static constexpr int LPP = NTHREADS / LINE;       // lines copied per pass
  static constexpr int PASSES = (KC ? W : BK) / LPP;
  static constexpr uint32_t DST = LPP * PITCH * 8;  // bytes between passes in the stage
  const double *p;  // this thread's element of pass 0 of the next slice
  int64_t step;     // elements between passes
  int64_t adv;      // elements between slices
  __device__ __forceinline__ static int line() { return threadIdx.x / LINE; }
  __device__ __forceinline__ static int pos() { return threadIdx.x % LINE; }
  __device__ __forceinline__ static uint32_t offset() { return (uint32_t)(line() * PITCH + pos()) * 8; }
  __device__ __forceinline__ void start(const double *src, int ld, int r0) {
    p = KC ? src + (int64_t)(r0 + line()) * ld + pos() : src + (int64_t)line() * ld + r0 + pos();
    step = LPP * (int64_t)ld;
    adv = KC ? BK : BK * (int64_t)ld;
  }
  // whole slice: all W rows and BK k inside the block
  __device__ __forceinline__ void load(uint32_t dst) {
    const double *q = p;
#pragma unroll
    for (int i = 0; i < PASSES; ++i, q += step) cp_async8(dst + i * DST, q);
    p += adv;
  }
  // `rows` rows and `k` k left in the block: rows past it are not loaded (they only reach output
  // rows that are not stored), k past it is zero-filled (from `any`, which is not read)
  __device__ __forceinline__ void load_edge(uint32_t dst, int rows, int k, const double *any) {
    const double *q = p;
#pragma unroll
    for (int i = 0; i < PASSES; ++i, q += step) {
      const int l = line() + i * LPP, x = pos();
      const bool ok = (KC ? x : l) < k;
      if ((KC ? l : x) < rows) cp_async8_zfill(dst + i * DST, ok ? q : any, ok ? 8 : 0);
    }
    p += adv;
  }
};

// Each of the 4 warps computes a (BM / 2) x (BN / 2) quarter of the tile: 64 x 64 tiles 2 x 4
// m16n8 products per k step, 64 x 32 tiles 2 x 2, 32 x 32 tiles (plans of small blocks, where 64 rows are
// mostly padding) 1 x 2.  Bound by the DMMA pipe, which runs at 128 cycles a product and SM quarter, and by
// how well the other warps' instructions hide behind it.  Two-site FP64 matvec, with the loads'
// arithmetic inside the stage and 64 x 64 tiles -> this: D=4096 635 -> 555 us, D=3000 283 -> 249,
// D=2048 126 -> 105, D=1500 61 -> 52, D=1024 33.0 -> 31.8.  Warps with tiles and stages of their own, which
// skip the padding (1.11 instead of 1.36 times the useful products at D=4096), were slower (637 us
// and more: ten warps per SM do not hide their own load instructions).
template <bool TA, bool TB, int BM, int BN>
__global__ void __launch_bounds__(NTHREADS) k_gemm_grouped_f64(
    const double *__restrict__ A, const double *__restrict__ B, double *__restrict__ C,
    const GemmTaskD *__restrict__ tasks, const GemmPairD *__restrict__ pairs,
    const GemmTileD *__restrict__ tiles, int64_t ntiles) {
  constexpr int MI = BM / 32;  // m16 products per warp
  constexpr int NJ = BN / 16;  // n8 products per warp
  __shared__ __align__(16) SmemT<TA, TB, BM, BN> sm;
  using CA = SliceCursor<!TA, BM, (TA ? BM : BK) + PAD>;
  using CB = SliceCursor<TB, BN, (TB ? BK : BN) + PAD>;
  const uint32_t da0 = (uint32_t)__cvta_generic_to_shared(&sm.A[0][0][0]) + CA::offset();
  const uint32_t db0 = (uint32_t)__cvta_generic_to_shared(&sm.B[0][0][0]) + CB::offset();
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2, t4 = lane & 3;
  for (int64_t ti = blockIdx.x; ti < ntiles; ti += gridDim.x) {
    const GemmTileD tile = tiles[ti];
    const GemmTaskD task = tasks[tile.task];
    const int m0 = tile.m0, n0 = tile.n0;
    const int mr = task.m - m0, nr = task.n - n0;  // rows and columns of the block from here on
    const int quarter = threadIdx.x >> 5;
    const int wm = (quarter >> 1) * (BM / 2), wn = (quarter & 1) * (BN / 2);
    double acc[MI][NJ][4];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[i][j][r] = 0.0;

    // flattened (pair, k) iteration with a 2-deep cp.async pipeline; the next pair's descriptor is
    // fetched when a pair begins
    const GemmPairD *next = pairs + task.pair_begin, *const last = next + task.pair_count;
    GemmPairD np;
    int kleft = 0;
    CA ca;
    CB cb;
    auto fetch = [&] {  // the next pair with work
      np.k = 0;
      while (next < last) {
        np = *next++;
        if (np.k > 0) break;
      }
    };
    auto begin_pair = [&] {
      kleft = np.k > 0 ? np.k : 0;
      if (kleft) {
        ca.start(A + np.a_off, np.lda, m0);
        cb.start(B + np.b_off, np.ldb, n0);
        fetch();
      }
    };
    fetch();
    begin_pair();
    const bool rows_whole = mr >= BM && nr >= BN;
    auto issue = [&](int slot) -> bool {
      const bool have = kleft > 0;
      if (have) {
        const uint32_t da = da0 + (uint32_t)slot * (uint32_t)sizeof(sm.A[0]);
        const uint32_t db = db0 + (uint32_t)slot * (uint32_t)sizeof(sm.B[0]);
        if (rows_whole && kleft >= BK) {
          ca.load(da);
          cb.load(db);
        } else {
          ca.load_edge(da, mr, kleft, A);
          cb.load_edge(db, nr, kleft, B);
        }
        kleft -= BK;
        if (kleft <= 0) begin_pair();
      }
      cp_async_commit();
      return have;
    };
    int buf = 0;
    bool have = issue(0);
    while (have) {
      const bool have_next = issue(buf ^ 1);
      cp_async_wait<1>();
      __syncthreads();
      double a[MI][8], b[NJ][4];
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int r = wm + i * 16 + g + 8 * (e & 1), k = t4 + 4 * (e >> 1);
          a[i][e] = TA ? sm.A[buf][k][r] : sm.A[buf][r][k];
        }
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int k = t4 + 4 * e, cidx = wn + j * 8 + g;
          b[j][e] = TB ? sm.B[buf][cidx][k] : sm.B[buf][k][cidx];
        }
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) dmma_16x8x16(acc[i][j], a[i], b[j]);
      __syncthreads();
      buf ^= 1;
      have = have_next;
    }
    cp_async_wait<0>();
    double *Cp = C + task.c_off;
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int r0 = m0 + wm + i * 16 + g;
        const int c0 = n0 + wn + j * 8 + 2 * t4;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = r0 + h * 8;
          if (r < task.m) {
            if (c0 < task.n) Cp[(int64_t)r * task.ldc + c0] = acc[i][j][2 * h];
            if (c0 + 1 < task.n) Cp[(int64_t)r * task.ldc + c0 + 1] = acc[i][j][2 * h + 1];
          }
        }
      }
    __syncthreads();
  }
}

// Plans whose products are all scalar times vector (k == 1 and n == 1 in every pair, or m == 1):
// C_t = sum_p A_p * b_p.  The contraction of a U(1) tensor with an MPO is of this kind, its legs
// having one state per charge.  A GEMM tile would pad k to 16 and n to 32 columns (D=1024
// environment update: 52 us of tensor-pipe work for 3 MB of data); here each thread walks the
// pairs of its elements, so the kernel is bound by the operands' reads.  Same products, added in
// the same order.  D=1024 environment update 181 -> 172 us, energy and gradient of a 16-site MPS at
// D=192 27.2 -> 25.4 ms (both then bound by the host).
constexpr int SCALED_PER = 4, SCALED_CHUNK = 256 * SCALED_PER;

template <bool COL>  // COL: column vectors A_p (n == 1), else row vectors B_p (m == 1)
__global__ void __launch_bounds__(256) k_scaled_sum(const double *__restrict__ A, const double *__restrict__ B,
                                                    double *__restrict__ C, const GemmTaskD *__restrict__ tasks,
                                                    const GemmPairD *__restrict__ pairs,
                                                    const GemmTileD *__restrict__ tiles) {
  const GemmTileD tile = tiles[blockIdx.x];
  const GemmTaskD task = tasks[tile.task];
  const int len = COL ? task.m : task.n;
  const int e0 = tile.m0 + threadIdx.x;
  double s[SCALED_PER];
#pragma unroll
  for (int i = 0; i < SCALED_PER; ++i) s[i] = 0.0;
  for (int p = 0; p < task.pair_count; ++p) {
    const GemmPairD pr = pairs[task.pair_begin + p];
    if (pr.k <= 0) continue;
    const double c = COL ? B[pr.b_off] : A[pr.a_off];
    const double *x = COL ? A + pr.a_off : B + pr.b_off;
#pragma unroll
    for (int i = 0; i < SCALED_PER; ++i)
      if (e0 + i * 256 < len) s[i] = fma(x[e0 + i * 256], c, s[i]);
  }
  double *o = C + task.c_off;
#pragma unroll
  for (int i = 0; i < SCALED_PER; ++i)
    if (e0 + i * 256 < len) o[e0 + i * 256] = s[i];
}
}  // namespace

void build_tiles_f64(const std::vector<GemmTaskD> &tasks, const std::vector<GemmPairD> &pairs,
                     std::vector<GemmTileD> &tiles, int bm, int bn) {
  tiles.clear();
  std::vector<std::pair<double, GemmTileD>> tmp;
  for (size_t t = 0; t < tasks.size(); ++t) {
    const GemmTaskD &tk = tasks[t];
    double kt = 0;
    for (int p = 0; p < tk.pair_count; ++p) kt += std::max(0, pairs[tk.pair_begin + p].k);
    for (int m0 = 0; m0 < tk.m; m0 += bm)
      for (int n0 = 0; n0 < tk.n; n0 += bn) {
        GemmTileD g;
        g.task = (int32_t)t;
        g.m0 = m0;
        g.n0 = n0;
        tmp.push_back({kt + 1.0, g});
      }
  }
  // longest-first so the tail of the grid is made of cheap tiles
  std::stable_sort(tmp.begin(), tmp.end(), [](const auto &a, const auto &b) { return a.first > b.first; });
  tiles.reserve(tmp.size());
  for (auto &x : tmp) tiles.push_back(x.second);
}

void build_chunks_f64(const std::vector<GemmTaskD> &tasks, bool col, std::vector<GemmTileD> &tiles) {
  tiles.clear();
  for (size_t t = 0; t < tasks.size(); ++t) {
    const int64_t len = col ? tasks[t].m : tasks[t].n;
    for (int64_t e = 0; e < len; e += SCALED_CHUNK) tiles.push_back({(int32_t)t, (int32_t)e, 0});
  }
}

ctn_status launch_scaled_sum_f64(const double *A, const double *B, double *C, const GemmTaskD *d_tasks,
                                 const GemmPairD *d_pairs, const GemmTileD *d_tiles, int64_t ntiles, bool col,
                                 cudaStream_t st) {
  if (ntiles == 0) return CTN_OK;
  if (col) k_scaled_sum<true><<<(unsigned)ntiles, 256, 0, st>>>(A, B, C, d_tasks, d_pairs, d_tiles);
  else k_scaled_sum<false><<<(unsigned)ntiles, 256, 0, st>>>(A, B, C, d_tasks, d_pairs, d_tiles);
  CTN_CHECK_LAUNCH();
  return CTN_OK;
}

namespace {
template <bool TA, bool TB, int BM, int BN>
ctn_status launch_gemm(const double *A, const double *B, double *C, const GemmTaskD *d_tasks, const GemmPairD *d_pairs,
                       const GemmTileD *d_tiles, int64_t ntiles, int nsm, cudaStream_t st) {
  const int64_t grid = std::min<int64_t>(ntiles, (int64_t)nsm * 12);
  k_gemm_grouped_f64<TA, TB, BM, BN><<<(unsigned)grid, NTHREADS, 0, st>>>(A, B, C, d_tasks, d_pairs, d_tiles, ntiles);
  CTN_CHECK_LAUNCH();
  return CTN_OK;
}
template <bool TA, bool TB>
ctn_status launch_tiles(const double *A, const double *B, double *C, const GemmTaskD *d_tasks, const GemmPairD *d_pairs,
                        const GemmTileD *d_tiles, int64_t ntiles, int bm, int bn, int nsm, cudaStream_t st) {
  if (bn == 64) return launch_gemm<TA, TB, 64, 64>(A, B, C, d_tasks, d_pairs, d_tiles, ntiles, nsm, st);
  if (bm == 32) return launch_gemm<TA, TB, 32, 32>(A, B, C, d_tasks, d_pairs, d_tiles, ntiles, nsm, st);
  return launch_gemm<TA, TB, 64, 32>(A, B, C, d_tasks, d_pairs, d_tiles, ntiles, nsm, st);
}
}  // namespace

ctn_status launch_gemm_f64(const double *A, const double *B, double *C, const GemmTaskD *d_tasks,
                           const GemmPairD *d_pairs, const GemmTileD *d_tiles, int64_t ntiles, int flags,
                           int bm, int bn, cudaStream_t st) {
  if (ntiles == 0) return CTN_OK;
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  switch (flags & 3) {
    case 0: return launch_tiles<false, false>(A, B, C, d_tasks, d_pairs, d_tiles, ntiles, bm, bn, nsm, st);
    case 1: return launch_tiles<true, false>(A, B, C, d_tasks, d_pairs, d_tiles, ntiles, bm, bn, nsm, st);
    case 2: return launch_tiles<false, true>(A, B, C, d_tasks, d_pairs, d_tiles, ntiles, bm, bn, nsm, st);
    default: return launch_tiles<true, true>(A, B, C, d_tasks, d_pairs, d_tiles, ntiles, bm, bn, nsm, st);
  }
}

}  // namespace ctn

extern "C" size_t ctn_gemm_grouped_scratch_bytes(int64_t ntasks, int64_t npairs) {
  // tasks + pairs + tiles (upper bound: tiles counted at execution; reserve generously)
  (void)ntasks;
  (void)npairs;
  return 0;
}
