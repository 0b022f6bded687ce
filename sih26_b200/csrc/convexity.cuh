// The dense convexity test of a QP's Hessian on the device: check_convexity
// (src/qp/convexity.cpp:30-134), an LDL' factorisation without interchanges that stops at the first
// pivot below -slack.
//
// Every entry takes the reference's operations in its order: w_ic starts as q_ic and loses
// (l_ik l_ck) d_k for k = 0, 1, ... one rounded operation at a time (no fused add), l_ij = w_ij / d_j;
// so the pivots, and with them the verdict, are the reference's to the bit. The order within an entry
// is all that it fixes: the factorisation runs right-looking in panels of kPanel columns, and every
// entry below a panel takes the panel's kPanel terms at once, from shared memory.
//
// Per panel: each block factors the diagonal kPanel x kPanel block for itself (a chain of kPanel
// divisions, ~10 us, with nothing to wait for), solves its share of the rows below (a thread a row,
// its panel entries in registers), a grid barrier, updates its tiles of the lower triangle, a grid
// barrier. Bound by the panels' chains: n = 2,000 has 63 of them; the 8e9 FP64 operations of the updates
// are well under a millisecond of the chip. A call with an 800 x 2,000 QP took 110-130 ms with the
// factorisation on 16 host threads, most of it there, and takes 13-15 with it here.
#pragma once

#include "device_common.cuh"

namespace sih26 {

constexpr int kPanel = 32;
constexpr int kTile = 64;

struct ConvexityRun {
  double* w;        // n x n, row-major; the lower triangle is used
  double* l;        // n x kPanel: the panel's columns of L, rows below the diagonal block
  int n;
  double slack;
  int* column;      // out: the first column whose pivot is below -slack, or -1
  double* pivot;    // out: that pivot
  GridBarrier bar;
};

// w gets sense * Q from the lower triangle in CSC (row >= column).
__global__ void hessian_scatter(const int* cs, const int* ri, const double* val, int n, double sense, double* w) {
  const int stride = gridDim.x * blockDim.x;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += stride)
    for (int k = cs[j]; k < cs[j + 1]; ++k) w[(size_t)ri[k] * n + j] = sense * val[k];
}

__device__ __forceinline__ double minus_term(double w, double li, double lc, double d) {
  return __dsub_rn(w, __dmul_rn(__dmul_rn(li, lc), d));
}

__global__ void __launch_bounds__(kThreads, 1) convexity_kernel(ConvexityRun R) {
  __shared__ double diag[kPanel][kPanel + 1];  // the diagonal block: L below, work on and above
  __shared__ double d[kPanel];
  __shared__ double li[kTile][kPanel + 1], lc[kTile][kPanel + 1];
  __shared__ int bad;
  const int n = R.n, tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  for (int j0 = 0; j0 < n; j0 += kPanel) {
    const int pw = n - j0 < kPanel ? n - j0 : kPanel;
    // the diagonal block, redundantly in every block: warp r holds rows r, r + kWarps, ...
    for (int e = tid; e < kPanel * kPanel; e += kThreads) {
      const int r = e / kPanel, c = e % kPanel;
      diag[r][c] = r < pw && c <= r ? __ldcg(R.w + (size_t)(j0 + r) * n + j0 + c) : 0.0;
    }
    if (tid == 0) bad = -1;
    __syncthreads();
    for (int j = 0; j < pw; ++j) {
      const double pivot = diag[j][j];
      if (pivot < -R.slack) {
        if (tid == 0) bad = j;
        break;  // every thread reads the same pivot
      }
      const bool zero = pivot <= R.slack;
      if (tid == 0) d[j] = zero ? 0.0 : pivot;
      __syncthreads();
      if (tid > j && tid < pw) diag[tid][j] = zero ? 0.0 : diag[tid][j] / pivot;
      __syncthreads();
      if (!zero) {
        for (int r = j + 1 + warp; r < pw; r += kWarps) {
          const int c = lane;
          if (c > j && c <= r) diag[r][c] = minus_term(diag[r][c], diag[r][j], diag[c][j], pivot);
        }
      }
      __syncthreads();
    }
    __syncthreads();
    if (bad >= 0) {
      if (blockIdx.x == 0 && tid == 0) {
        *R.column = j0 + bad;
        *R.pivot = diag[bad][bad];
      }
      return;  // every block takes the same branch
    }
    const int below = j0 + pw;
    if (below >= n) break;
    // the rows below: l_ij for the panel's columns, a thread per row
    for (int i = below + blockIdx.x * kThreads + tid; i < n; i += gridDim.x * kThreads) {
      double row[kPanel];
#pragma unroll
      for (int c = 0; c < kPanel; ++c) row[c] = __ldcg(R.w + (size_t)i * n + j0 + c);
#pragma unroll
      for (int j = 0; j < kPanel; ++j) {
        const double dj = d[j];
        // 0 stands for a pivot within the slack; one that is not a number (inf - inf) goes on as in the reference
        const double l = dj != 0.0 ? row[j] / dj : 0.0;
        row[j] = l;
        if (dj != 0.0) {
#pragma unroll
          for (int c = j + 1; c < kPanel; ++c) row[c] = minus_term(row[c], l, diag[c][j], dj);
        }
      }
#pragma unroll
      for (int c = 0; c < kPanel; ++c) R.l[(size_t)i * kPanel + c] = row[c];
    }
    if (!grid_barrier(R.bar)) return;
    // the lower triangle behind the panel, tile by tile
    const int rest = n - below, tiles = (rest + kTile - 1) / kTile, count = tiles * (tiles + 1) / 2;
    for (int t = blockIdx.x; t < count; t += gridDim.x) {
      int ti = static_cast<int>((sqrtf(8.0f * t + 1.0f) - 1.0f) * 0.5f);
      while ((ti + 1) * (ti + 2) / 2 <= t) ++ti;
      while (ti * (ti + 1) / 2 > t) --ti;
      const int tc = t - ti * (ti + 1) / 2;
      const int i0 = below + ti * kTile, c0 = below + tc * kTile;
      __syncthreads();
      for (int e = tid; e < kTile * kPanel; e += kThreads) {
        const int r = e / kPanel, k = e % kPanel;
        li[r][k] = i0 + r < n ? __ldcg(R.l + (size_t)(i0 + r) * kPanel + k) : 0.0;
        lc[r][k] = c0 + r < n ? __ldcg(R.l + (size_t)(c0 + r) * kPanel + k) : 0.0;
      }
      __syncthreads();
      const int c = tid & (kTile - 1), r0 = tid / kTile;  // kThreads / kTile rows at a time
      constexpr int kStep = kThreads / kTile, kRows = kTile / kStep;
      double w[kRows];
#pragma unroll
      for (int q = 0; q < kRows; ++q) {
        const int i = i0 + r0 + q * kStep;
        w[q] = i < n && c0 + c <= i ? __ldcg(R.w + (size_t)i * n + c0 + c) : 0.0;
      }
      for (int k = 0; k < kPanel; ++k) {
        const double b = lc[c][k], dk = d[k];
#pragma unroll
        for (int q = 0; q < kRows; ++q) w[q] = minus_term(w[q], li[r0 + q * kStep][k], b, dk);
      }
#pragma unroll
      for (int q = 0; q < kRows; ++q) {
        const int i = i0 + r0 + q * kStep;
        if (i < n && c0 + c <= i) __stcg(R.w + (size_t)i * n + c0 + c, w[q]);
      }
    }
    if (!grid_barrier(R.bar)) return;
  }
  if (blockIdx.x == 0 && tid == 0) *R.column = -1;
}

}  // namespace sih26
