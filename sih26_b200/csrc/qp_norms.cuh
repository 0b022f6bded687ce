// The QP step sizes' two power iterations (qp_condat_vu.cpp:64-134) on the device, in the reference's order
// of operations: sums over a vector in ascending order by one thread, a row's products in ascending column
// order, every product and sum rounded by itself. The estimates are the host's bits.
//
// One launch of two clusters, one for A and one for Q, beside the host's layout of the problem. Bound by the
// vector sums, a chain of n additions of 8 cycles, 21 of them (n = 25,000: 2.2 ms); the host's iterations
// took 11 ms there (250,000 nonzeros).
#pragma once

#include <cooperative_groups.h>

#include "device_common.cuh"

namespace sih26 {

constexpr int kNormTeam = 8;  // blocks of a cluster

struct NormMatrix {
  int rows;
  const int* ptr;
  const int* idx;
  const double* val;
};

struct NormRun {
  NormMatrix first, second;  // v -> first v -> second first v; Q has no second
  int n;                     // length of v; 0: nothing to do, the estimate is 0
  int square;                // 1: A (the square root of |A'A v|), 0: Q (|v'Qv|)
  double* v;                 // [n] the start, overwritten
  double* w;                 // [first.rows]
  double* scalar;            // [2] norm, estimate
};

// sum_j a[j] b[j], j ascending; the first block's threads call it and thread 0 has the sum.
__device__ __forceinline__ double ordered_dot(const double* a, const double* b, int n) {
  constexpr int kChunk = 1024;
  __shared__ double product[2][kChunk];
  const auto fill = [&](int c) {
    // thread 0's warp only adds
    for (int t = (int)threadIdx.x - 32; t < kChunk; t += kThreads - 32) {
      const long long j = (long long)c * kChunk + t;
      if (t >= 0 && j < n) product[c & 1][t] = __dmul_rn(__ldcg(a + j), __ldcg(b + j));
    }
  };
  double s = 0.0;
  const int chunks = n / kChunk + (n % kChunk != 0);
  if (threadIdx.x >= 32) fill(0);
  __syncthreads();
  for (int c = 0; c < chunks; ++c) {
    if (threadIdx.x >= 32) {
      if (c + 1 < chunks) fill(c + 1);
    } else if (threadIdx.x == 0) {
      const double* p = product[c & 1];
      const int count = min(kChunk, n - c * kChunk);
#pragma unroll 16
      for (int t = 0; t < count; ++t) s = __dadd_rn(s, p[t]);
    }
    __syncthreads();
  }
  return s;
}

// out = M in: rows of up to kShort entries a thread each, longer ones a warp each (the lanes form the
// products of 32 entries, lane 0's order adds them).
__device__ __forceinline__ void ordered_rows(const NormMatrix& m, const double* in, double* out, int rank) {
  constexpr int kShort = 64;
  const int lane = threadIdx.x & 31;
  const int thread = rank * kThreads + threadIdx.x, threads = kNormTeam * kThreads;
  for (unsigned r = thread; r < (unsigned)m.rows; r += threads) {
    const int b = __ldg(m.ptr + r), e = __ldg(m.ptr + r + 1);
    if (e - b > kShort) continue;
    double s = 0.0;
#pragma unroll 8
    for (int k = b; k < e; ++k) s = __dadd_rn(s, __dmul_rn(__ldg(m.val + k), __ldcg(in + __ldg(m.idx + k))));
    out[r] = s;
  }
  // every warp looks through rows of its own, a stride apart, so that long ones side by side spread
  const int warp = thread >> 5, warps = threads >> 5;
  for (unsigned r0 = warp; r0 < (unsigned)m.rows; r0 += 32 * warps) {
    const unsigned r = r0 + lane * warps;
    const bool is_long = r < (unsigned)m.rows && __ldg(m.ptr + r + 1) - __ldg(m.ptr + r) > kShort;
    for (unsigned todo = __ballot_sync(0xffffffffu, is_long); todo != 0u; todo &= todo - 1u) {
      const unsigned q = r0 + (__ffs(todo) - 1) * warps;
      // unsigned: the batch behind the last may pass 2^31 - 1
      const unsigned b = __ldg(m.ptr + q), e = __ldg(m.ptr + q + 1);
      const auto product = [&](unsigned k) {
        return k < e ? __dmul_rn(__ldg(m.val + k), __ldcg(in + __ldg(m.idx + k))) : 0.0;
      };
      double s = 0.0, next = product(b + lane);
      for (unsigned k = b; k < e; k += 32) {
        const double mine = next;
        next = product(k + 32 + lane);
        // past the end the lanes hold zeros, which add nothing
#pragma unroll
        for (int l = 0; l < 32; ++l) s = __dadd_rn(s, __shfl_sync(0xffffffffu, mine, l));
      }
      if (lane == 0) out[q] = s;
    }
  }
}

__global__ void __cluster_dims__(kNormTeam, 1, 1) __launch_bounds__(kThreads) qp_norm_kernel(NormRun a, NormRun q) {
  const NormRun& r = blockIdx.x < kNormTeam ? a : q;
  const auto team = cooperative_groups::this_cluster();
  const int rank = blockIdx.x % kNormTeam;
  const int thread = rank * kThreads + threadIdx.x, threads = kNormTeam * kThreads;
  if (r.n == 0) return;
  double *v = r.v, *w = r.w;
  for (int it = 0; it < 20; ++it) {
    if (rank == 0) {
      const double sum = ordered_dot(v, v, r.n);
      if (threadIdx.x == 0) __stcg(r.scalar, __dsqrt_rn(sum));
    }
    team.sync();
    const double norm = __ldcg(r.scalar);
    if (norm <= 0.0) return;  // every block alike; the estimate stays 0
    for (unsigned j = thread; j < (unsigned)r.n; j += threads) v[j] = __ddiv_rn(__ldcg(v + j), norm);
    team.sync();
    ordered_rows(r.first, v, w, rank);
    team.sync();
    if (r.square) {
      ordered_rows(r.second, w, v, rank);
    } else {
      if (it == 19 && rank == 0) {
        const double next = ordered_dot(w, v, r.n);
        if (threadIdx.x == 0) __stcg(r.scalar + 1, fabs(next));
      }
      double* t = v;
      v = w;
      w = t;
    }
    team.sync();
  }
  if (r.square && rank == 0) {
    const double next = ordered_dot(v, v, r.n);
    if (threadIdx.x == 0) __stcg(r.scalar + 1, __dsqrt_rn(__dsqrt_rn(next)));
  }
}

}  // namespace sih26
