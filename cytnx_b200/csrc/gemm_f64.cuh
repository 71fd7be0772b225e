// Device-side task tables of the grouped FP64 GEMM and the owning host object.
#pragma once
#include <algorithm>
#include <cstdint>
#include <vector>

#include "ctn_common.h"

namespace ctn {

// 32 x 32 tiles when 64 x 32 tiles execute more than this many times their products: blocks of up
// to a few hundred rows (D=2048 two-site matvec 105 us against 113), the wider tiles where their
// padding is small (D=4096: 555 us against 567).  64 x 64 tiles were slower throughout (580 us).
constexpr double F64_NARROW_PADDING = 1.12;

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
                           int bm, cudaStream_t st);

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
  int bm = 64;            // rows of a tile of 32 columns
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
      for (int p = 0; p < t.pair_count; ++p) kp += (double)((std::max(0, pairs[t.pair_begin + p].k) + 15) / 16 * 16);
      w += (double)((t.m + tm - 1) / tm) * tm * (double)((t.n + tn - 1) / tn) * tn * kp;
    }
    return w;
  }
  void finalize() {
    scaled = scaled_sum(true) ? 1 : scaled_sum(false) ? 2 : 0;
    if (scaled) {
      build_chunks_f64(tasks, scaled == 1, tiles);
    } else {
      bm = executed(64, 32) > F64_NARROW_PADDING * executed(32, 32) ? 32 : 64;
      build_tiles_f64(tasks, pairs, tiles, bm, 32);
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
    return launch_gemm_f64(A, B, C, dt, dp, dl, (int64_t)tiles.size(), flags, bm, st);
  }
  ~GroupedGemmF64() {
    if (d_mem) cudaFree(d_mem);
  }
};

}  // namespace ctn
