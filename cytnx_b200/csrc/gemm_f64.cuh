// Device-side task tables of the grouped FP64 GEMM and the owning host object.
#pragma once
#include <algorithm>
#include <cstdint>
#include <vector>

#include "ctn_common.h"

namespace ctn {

// Which tile a plan takes (times of whole launches):
// * 32 x 32 where 64 x 32 tiles execute more than 1.12 times their products (blocks of up to a few hundred
//   rows: D=2048 two-site matvec 102 us against 110) or are fewer than six an SM (dense 512^3 17 us against
//   21, 100 x 100 x 2048 60 against 79);
// * 64 x 64, which load each operand element for more products, where that costs next to no padding, there
//   are six an SM of them and more than one slice of k to load (dense 4096 x 4096 x 64 82 us against 92, 4096^2 x
//   2048 2050 against 2150; with one slice 14 an SM: 8192^2 x 8 154 against 180, 2048^2 x 8 14.0 against 12.8).
//   The two-site blocks at D=4096 (1.10 times the products) lose by them: 562 us against 535;
// * 64 x 32 else.
constexpr double F64_NARROW_PADDING = 1.12, F64_WIDE_PADDING = 1.03;
constexpr size_t F64_TILES_PER_SM = 6, F64_TILES_PER_SM_ONE_SLICE = 14;
constexpr int F64_BK = 16;  // k depth of a slice

struct GemmTaskD {
  int64_t c_off;
  int32_t m, n, ldc;
  int32_t pair_begin, pair_count;
  int32_t pad_;
};
struct GemmPairD {
  int64_t a_off, b_off;
  int32_t k, lda, ldb, flags;  // flags bit0: A stored [k][m]; bit1: B stored [n][k]
};
struct GemmTileD {
  int32_t task;
  int32_t m0, n0;
};

void build_tiles_f64(const std::vector<GemmTaskD> &tasks, const std::vector<GemmPairD> &pairs,
                     std::vector<GemmTileD> &tiles, int bm, int bn);
ctn_status launch_gemm_f64(const double *A, const double *B, double *C, const GemmTaskD *d_tasks,
                           const GemmPairD *d_pairs, const GemmTileD *d_tiles, int64_t ntiles, int flags,
                           int bm, int bn, cudaStream_t st);

// the element runs of k_scaled_sum (vectors of m elements when col, else of n)
void build_chunks_f64(const std::vector<GemmTaskD> &tasks, bool col, std::vector<GemmTileD> &tiles);
ctn_status launch_scaled_sum_f64(const double *A, const double *B, double *C, const GemmTaskD *d_tasks,
                                 const GemmPairD *d_pairs, const GemmTileD *d_tiles, int64_t ntiles, bool col,
                                 cudaStream_t st);

// Host tables + their device copy (uploaded once, on the first launch on a device).
struct GroupedGemmF64 {
  std::vector<GemmTaskD> tasks;
  std::vector<GemmPairD> pairs;
  std::vector<GemmTileD> tiles;
  void *d_mem = nullptr;
  int d_dev = -1;
  double flops = 0.0;
  int flags = 0;          // operand orientation shared by every pair of the plan
  int bm = 64, bn = 32;   // tile: 64 x 64, 64 x 32 or 32 x 32
  bool mixed = false;     // pairs disagree on the orientation (rejected at run time)
  int scaled = 0;         // 1: every product is a column vector times a scalar, 2: a row vector, 0: GEMM

  // whether all products are scalar times a contiguous vector (k_scaled_sum)
  bool scaled_sum(bool col) const {
    for (const auto &t : tasks) {
      if (col ? t.n != 1 || t.ldc != 1 : t.m != 1) return false;
      for (int p = 0; p < t.pair_count; ++p) {
        const GemmPairD &pr = pairs[t.pair_begin + p];
        if (pr.k > 1) return false;
        if (col ? !(pr.flags & 1) && pr.lda != 1 : (pr.flags & 2) && pr.ldb != 1) return false;
      }
    }
    return !tasks.empty();
  }

  // products the tiles execute, with K padded to the 16-deep stages
  double executed(int tm, int tn) const {
    double w = 0.0;
    for (const auto &t : tasks) {
      double kp = 0.0;
      for (int p = 0; p < t.pair_count; ++p)
        kp += (double)((std::max(0, pairs[t.pair_begin + p].k) + F64_BK - 1) / F64_BK * F64_BK);
      w += (double)((t.m + tm - 1) / tm) * tm * (double)((t.n + tn - 1) / tn) * tn * kp;
    }
    return w;
  }
  void finalize() {
    scaled = scaled_sum(true) ? 1 : scaled_sum(false) ? 2 : 0;
    if (scaled) {
      build_chunks_f64(tasks, scaled == 1, tiles);
    } else {
      auto count = [&](int m, int n) {
        size_t c = 0;
        for (const auto &t : tasks) c += (size_t)((t.m + m - 1) / m) * (size_t)((t.n + n - 1) / n);
        return c;
      };
      int slices = 0;  // of the longest task
      for (const auto &t : tasks) {
        int c = 0;
        for (int p = 0; p < t.pair_count; ++p) c += (std::max(0, pairs[t.pair_begin + p].k) + F64_BK - 1) / F64_BK;
        slices = std::max(slices, c);
      }
      const size_t wide = 148 * (slices <= 1 ? F64_TILES_PER_SM_ONE_SLICE : F64_TILES_PER_SM);
      if (executed(64, 32) > F64_NARROW_PADDING * executed(32, 32) || count(64, 32) < 148 * F64_TILES_PER_SM) bm = 32;
      else if (executed(64, 64) <= F64_WIDE_PADDING * executed(64, 32) && count(64, 64) >= wide) bn = 64;
      build_tiles_f64(tasks, pairs, tiles, bm, bn);
    }
    flags = pairs.empty() ? 0 : (pairs[0].flags & 3);
    mixed = false;
    for (const auto &p : pairs) mixed |= ((p.flags & 3) != flags);
    flops = 0.0;
    for (const auto &t : tasks)
      for (int p = 0; p < t.pair_count; ++p)
        flops += 2.0 * t.m * (double)t.n * (double)pairs[t.pair_begin + p].k;
  }
  size_t table_bytes() const {
    return tasks.size() * sizeof(GemmTaskD) + pairs.size() * sizeof(GemmPairD) +
           tiles.size() * sizeof(GemmTileD) + 64;
  }
  ctn_status upload(cudaStream_t st) {
    int dev = 0;
    CTN_CUDA(cudaGetDevice(&dev));
    if (d_mem && d_dev == dev) return CTN_OK;
    if (d_mem) {
      cudaFree(d_mem);
      d_mem = nullptr;
    }
    CTN_CUDA(cudaMalloc(&d_mem, table_bytes()));
    d_dev = dev;
    char *p = (char *)d_mem;
    if (!tasks.empty()) CTN_CUDA(cudaMemcpyAsync(p, tasks.data(), tasks.size() * sizeof(GemmTaskD), cudaMemcpyHostToDevice, st));
    p += tasks.size() * sizeof(GemmTaskD);
    if (!pairs.empty()) CTN_CUDA(cudaMemcpyAsync(p, pairs.data(), pairs.size() * sizeof(GemmPairD), cudaMemcpyHostToDevice, st));
    p += pairs.size() * sizeof(GemmPairD);
    if (!tiles.empty()) CTN_CUDA(cudaMemcpyAsync(p, tiles.data(), tiles.size() * sizeof(GemmTileD), cudaMemcpyHostToDevice, st));
    // pageable host memory: make sure the copies finished before the vectors can change
    CTN_CUDA(cudaStreamSynchronize(st));
    return CTN_OK;
  }
  ctn_status run(const double *A, const double *B, double *C, cudaStream_t st) {
    if (mixed) {
      set_error("grouped GEMM: all pairs of one plan must share the operand orientation flags");
      return CTN_ERR_UNSUPPORTED;
    }
    CTN_TRY(upload(st));
    const char *p = (const char *)d_mem;
    const GemmTaskD *dt = (const GemmTaskD *)p;
    const GemmPairD *dp = (const GemmPairD *)(p + tasks.size() * sizeof(GemmTaskD));
    const GemmTileD *dl = (const GemmTileD *)(p + tasks.size() * sizeof(GemmTaskD) + pairs.size() * sizeof(GemmPairD));
    if (scaled) return launch_scaled_sum_f64(A, B, C, dt, dp, dl, (int64_t)tiles.size(), scaled == 1, st);
    return launch_gemm_f64(A, B, C, dt, dp, dl, (int64_t)tiles.size(), flags, bm, bn, st);
  }
  ~GroupedGemmF64() {
    if (d_mem) cudaFree(d_mem);
  }
};

}  // namespace ctn
