// KKT residuals of a given point for an LP already in device memory, computed without
// allocating anything (sankhya_pdhg_gpu_residuals_noalloc in include/sankhya_pdhg_gpu.h).
//
// Who needs this: a caller that must not allocate device memory once it is running -- an
// application whose device memory is owned by its own pool or arena and forbids raw
// cudaMalloc/cudaFree, a service that fixes its device-memory budget at start-up, or a
// latency-critical loop where cudaMalloc/cudaFree's implicit device synchronisation is not
// acceptable. Such a caller still wants to check an answer on the device, with the same
// residual definitions the solver uses.
//
// All scratch lives in one file-scope device array, g_noalloc_scratch, of fixed size
// (kScratchDoubles doubles = 4 MiB). Every GPU that loads this library holds it until the
// process exits. Its layout: block partials of the two reduction passes, an error word, then
// one FP64 activity slot per row, so a call accepts at most kMaxRows rows.
//
// Every call uses the same array and leaves its contents behind; each call clears what must
// start at zero (the activity accumulators and the error word) before using it. Calls whose
// work overlaps on the GPU (different streams, or different host threads without ordering)
// race on the array and give wrong answers; order them on one stream.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <string>

#include "entry_chunks.cuh"
#include "sankhya_pdhg_gpu.h"

namespace sih26 {
extern thread_local std::string g_last_error;
}

namespace {

constexpr int kThreads = 256;
constexpr int kMaxBlocks = 800;        // what the partials hold
constexpr int kGridBlocks = 148 * 4;  // the largest grid: kColumnBlocksPerSm blocks on every SM
constexpr int kSlots = 5;
constexpr size_t kScratchDoubles = (size_t)1 << 19;  // 4 MiB
constexpr size_t kPartialDoubles = 8192;
static_assert(2 * (size_t)kMaxBlocks * kSlots <= kPartialDoubles, "the partials outgrow their part of the scratch");
constexpr size_t kErrorDoubles = 32;  // one 256-byte line for the error word
constexpr size_t kMaxRows = kScratchDoubles - kPartialDoubles - kErrorDoubles;
static_assert(kMaxRows == SANKHYA_PDHG_NOALLOC_MAX_ROWS, "header and scratch layout disagree");

static __device__ __align__(256) double g_noalloc_scratch[kScratchDoubles];

struct View {
  double* col_partials;  // [kMaxBlocks][kSlots]
  double* row_partials;  // [kMaxBlocks][kSlots]
  unsigned* error;       // nonzero: an index was out of range
  unsigned* arrived;     // row blocks done
  double* activity;      // [m]
};

__host__ __device__ inline View carve(double* base) {
  View v;
  v.col_partials = base;
  v.row_partials = base + (size_t)kMaxBlocks * kSlots;
  v.error = reinterpret_cast<unsigned*>(base + kPartialDoubles);
  v.arrived = v.error + 1;
  v.activity = base + kPartialDoubles + kErrorDoubles;
  return v;
}

// An absent bound is +-inf or |v| >= 1e30; anything else, NaN included, is a finite bound, as
// is_finite_bound (include/sankhya/types.hpp:32-39) decides.
__device__ inline bool finite_bound(double v) { return !(fabs(v) >= 1e30); }
__device__ inline double dmax(double a, double b) { return (a < b) ? b : a; }
__device__ inline double dmin(double a, double b) { return (b < a) ? b : a; }

// Block totals of NS slots, in every thread's v on return. The tree is fixed (warps by xor,
// then one warp over the warp totals), so a total depends only on the threads' values.
template <int NS, int kBlock>
__device__ inline void block_total(double (&v)[NS], unsigned max_mask, double (*sh)[NS]) {
  const auto fold = [&](int from) {
    for (int off = from; off > 0; off >>= 1) {
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        const double o = __shfl_xor_sync(0xffffffffu, v[s], off);
        v[s] = ((max_mask >> s) & 1u) ? dmax(v[s], o) : v[s] + o;
      }
    }
  };
  constexpr int kW = kBlock / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  fold(16);
  if (lane == 0) {
#pragma unroll
    for (int s = 0; s < NS; ++s) sh[warp][s] = v[s];
  }
  __syncthreads();
#pragma unroll
  for (int s = 0; s < NS; ++s) v[s] = sh[lane & (kW - 1)][s];
  fold(kW / 2);
}

// Column terms of the reference's evaluate() (src/pdhg/pdhg.cpp:172-199, 239-256) for the
// reduced cost d = c + A'y of column j.
// slots: 0 dual violation^2, 1 bound contribution, 2 complementarity (max), 3 c'x, 4 ||c||^2
constexpr unsigned kColumnMax = 1u << 2;
__device__ __forceinline__ void column_terms(const sankhya_pdhg_problem& p, int j, double xj, double c,
                                             double d, double (&acc)[5]) {
  const double lo = p.col_lower[j], hi = p.col_upper[j];
  if (d > 0.0) {
    if (finite_bound(lo)) acc[1] += d * lo; else acc[0] += d * d;
  } else if (d < 0.0) {
    if (finite_bound(hi)) acc[1] += d * hi; else acc[0] += d * d;
  }
  if (lo != hi) {
    const double ls = finite_bound(lo) ? xj - lo : INFINITY;
    const double us = finite_bound(hi) ? hi - xj : INFINITY;
    acc[2] = dmax(acc[2], fabs(d) * dmin(ls, us));
  }
  acc[3] += c * xj;
  acc[4] += c * c;
}

// Row terms (pdhg.cpp:152-170, 205-222, 227-238) for the activity a of row i. slots: 0 primal
// violation^2, 1 support, 2 row dual violation^2, 3 complementarity (max), 4 ||b||^2
constexpr unsigned kRowMax = 1u << 3;
__device__ __forceinline__ void row_terms(const sankhya_pdhg_problem& p, int i, double a, double y,
                                          double (&acc)[5]) {
  const double lo = p.row_lower[i], hi = p.row_upper[i];
  double viol = 0.0;
  if (finite_bound(lo)) viol = dmax(viol, lo - a);
  if (finite_bound(hi)) viol = dmax(viol, a - hi);
  acc[0] += viol * viol;
  if (y > 0.0) {
    if (finite_bound(hi)) acc[1] += y * hi; else acc[2] += y * y;
  } else if (y < 0.0) {
    if (finite_bound(lo)) acc[1] += y * lo; else acc[2] += y * y;
  }
  if (lo != hi) {
    const double ls = finite_bound(lo) ? a - lo : INFINITY;
    const double us = finite_bound(hi) ? hi - a : INFINITY;
    acc[3] = dmax(acc[3], fabs(y) * dmin(ls, us));
  }
  const double b = finite_bound(lo) ? lo : (finite_bound(hi) ? hi : 0.0);
  acc[4] += b * b;
}

// The residual block in the order of sankhya_pdhg_residuals from the column and row totals
// (NaN everywhere when an index was out of range).
__device__ inline void write_residuals(const double (&c)[5], const double (&r)[5], bool bad, double* out) {
  if (bad) {
    for (int k = 0; k < 9; ++k) out[k] = NAN;
    return;
  }
  const double bound_norm = sqrt(r[4]), cost_norm = sqrt(c[4]);
  const double abs_primal = sqrt(r[0]);
  const double abs_dual = sqrt(c[0] + r[2]);
  const double pobj = c[3], dobj = c[1] - r[1];
  const double gap = fabs(pobj - dobj);
  out[0] = abs_primal / (1.0 + bound_norm);
  out[1] = abs_dual / (1.0 + cost_norm);
  out[2] = gap / (1.0 + fabs(pobj) + fabs(dobj));
  out[3] = pobj;
  out[4] = dobj;
  out[5] = abs_primal;
  out[6] = abs_dual;
  out[7] = gap / dmax(1.0, fabs(pobj));
  out[8] = dmax(c[2], r[3]);
}

// Entries [kb, ke) of column j, clamped to the arrays whatever col_starts holds.
__device__ __forceinline__ void column_range(const sankhya_pdhg_problem& p, int j, int& kb, int& ke) {
  kb = p.col_starts[j];
  ke = p.col_starts[j + 1];
  kb = kb < 0 ? 0 : (kb > p.num_nonzeros ? p.num_nonzeros : kb);
  ke = ke < kb ? kb : (ke > p.num_nonzeros ? p.num_nonzeros : ke);
}

// One column by one thread: scatters A x into `activity` and returns d + A'y of the column, the terms added to
// d in order (pdhg.cpp:172-199: the cost comes first, so it cancels against them one by one).
__device__ inline double column_by_thread(const sankhya_pdhg_problem& p, int kb, int ke, double xj, double d,
                                          double sense, const double* row_dual, double* activity,
                                          unsigned* error) {
  for (int k = kb; k < ke; ++k) {
    const int i = p.row_indices[k];
    if ((unsigned)i >= (unsigned)p.num_rows) {
      atomicOr(error, 1u);
      continue;
    }
    const double a = p.values[k];
    atomicAdd(activity + i, a * xj);
    d += a * (-sense * row_dual[i]);  // y = -sense * row_dual (pdhg.cpp:660)
  }
  return d;
}

// The whole check in one block, for LPs of at most kSmallRows rows whose columns and nonzeros a
// block gets through before the three launches of the path below are done: the activity lives in
// shared memory, nothing is cleared in or read back from the scratch. Bound by latency: one
// launch and a few dependent loads. 60 x 150 with 600 nonzeros: 8.2 us against 13 for the three
// kernels (and 16 for the four of before); 3,200 nonzeros, columns and rows together: 10.3 against
// 13; 9,400: 16.4 against 14, so the line lies between, at kSmallWork.
constexpr int kSmallThreads = 512;
constexpr int kSmallRows = 4096;
constexpr int kSmallWork = 6000;  // nonzeros + columns + rows
__global__ void __launch_bounds__(kSmallThreads) small_kernel(sankhya_pdhg_problem p, const double* x,
                                                              const double* row_dual, double* out) {
  __shared__ double activity[kSmallRows];
  __shared__ double sh[2][kSmallThreads / 32][5];
  __shared__ unsigned error;
  const double sense = p.maximize ? -1.0 : 1.0;
  for (int i = threadIdx.x; i < p.num_rows; i += kSmallThreads) activity[i] = 0.0;
  if (threadIdx.x == 0) error = 0u;
  __syncthreads();
  double c[5] = {0, 0, 0, 0, 0}, r[5] = {0, 0, 0, 0, 0};
  for (int j = threadIdx.x; j < p.num_cols; j += kSmallThreads) {
    int kb, ke;
    column_range(p, j, kb, ke);
    const double xj = x[j], cost = sense * p.cost[j];
    const double d = column_by_thread(p, kb, ke, xj, cost, sense, row_dual, activity, &error);
    column_terms(p, j, xj, cost, d, c);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < p.num_rows; i += kSmallThreads)
    row_terms(p, i, activity[i], -sense * row_dual[i], r);
  block_total<5, kSmallThreads>(c, kColumnMax, sh[0]);
  block_total<5, kSmallThreads>(r, kRowMax, sh[1]);
  if (threadIdx.x == 0) write_residuals(c, r, error != 0u, out);
}

__global__ void clear_kernel(double* base, int m) {
  const View v = carve(base);
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += stride) v.activity[i] = 0.0;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *v.error = 0u;
    *v.arrived = 0u;
  }
}

// Columns: scatter A x into the activity slots; reduced costs and the column terms. A warp takes
// 32 consecutive columns at a time, whose entries are one contiguous range of the arrays: it
// reads kChunk of them coalesced (kChunk / 32 independent loads a lane), finds each entry's
// column by a binary search over the lanes' column ends, sends the activity terms off as
// reductions and parks the terms of A'y in shared memory, where each lane sums its own column
// in order. Bound by the scattered accesses of every entry (a 32-byte sector of row_dual, an L2
// reduction): with the reductions left out the 3M-nonzero check took 39 us, with them 57 (four
// resident blocks and chunks of 128; three of 256 took 60, two of 512 58), against 180 with one
// thread walking each column and a serial fold of the partials.
// The next two kernels are launched to overlap the end of the one before them (5 us off the three
// launches); each waits for it before it touches the scratch.
constexpr int kChunk = 128;
constexpr int kColumnBlocksPerSm = 4;
__global__ void __launch_bounds__(kThreads, kColumnBlocksPerSm) column_kernel(sankhya_pdhg_problem p, const double* x,
                                                          const double* row_dual, double* base) {
  const View v = carve(base);
  __shared__ double terms[kThreads / 32][kChunk];
  __shared__ double sh[kThreads / 32][5];
  const double sense = p.maximize ? -1.0 : 1.0;
  double acc[5] = {0, 0, 0, 0, 0};
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* park = terms[warp];
  cudaGridDependencySynchronize();
  const int groups = p.num_cols / 32 + (p.num_cols % 32 != 0);
  for (int g = blockIdx.x * (kThreads / 32) + warp; g < groups; g += gridDim.x * (kThreads / 32)) {
    const int j = g * 32 + lane;
    const bool mine = j < p.num_cols;
    int kb = 0, ke = 0;
    double xj = 0.0, cost = 0.0;
    if (mine) {
      column_range(p, j, kb, ke);
      xj = x[j];
      cost = sense * p.cost[j];
    }
    double d = cost;
    const int last = __shfl_sync(0xffffffffu, ke, (p.num_cols - g * 32 < 32 ? p.num_cols - g * 32 : 32) - 1);
    if (!mine) kb = ke = last;
    const int first = __shfl_sync(0xffffffffu, kb, 0);
    const int before = __shfl_up_sync(0xffffffffu, ke, 1);
    if (__all_sync(0xffffffffu, lane == 0 || before == kb)) {
      for (int c0 = first, c1; c0 < last; c0 = c1) {
        c1 = sih26::chunk_end<kChunk>(c0, last);
        // the lanes' positions are unsigned: those past the range's end may lie past 2^31 - 1
        const unsigned k0 = (unsigned)c0 + lane, end = c1;
        int row[kChunk / 32];
        double a[kChunk / 32];
#pragma unroll
        for (int t = 0; t < kChunk / 32; ++t) {
          const unsigned k = k0 + 32 * t;
          row[t] = k < end ? p.row_indices[k] : 0;
          a[t] = k < end ? p.values[k] : 0.0;
        }
        double y[kChunk / 32];
#pragma unroll
        for (int t = 0; t < kChunk / 32; ++t) {
          const unsigned k = k0 + 32 * t;
          const bool good = (unsigned)row[t] < (unsigned)p.num_rows;
          if (k < end && !good) atomicOr(v.error, 1u);
          y[t] = k < end && good ? row_dual[row[t]] : 0.0;
        }
#pragma unroll
        for (int t = 0; t < kChunk / 32; ++t) {
          const unsigned k = k0 + 32 * t;
          // the lane whose column holds entry k: the number of columns that end at or before k
          int owner = 0;
#pragma unroll
          for (int step = 16; step > 0; step >>= 1)
            if ((unsigned)__shfl_sync(0xffffffffu, ke, owner + step - 1) <= k) owner += step;
          const double xo = __shfl_sync(0xffffffffu, xj, owner & 31);
          if (k < end) {
            if ((unsigned)row[t] < (unsigned)p.num_rows) atomicAdd(v.activity + row[t], a[t] * xo);
            park[lane + 32 * t] = a[t] * (-sense * y[t]);  // y = -sense * row_dual (pdhg.cpp:660)
          }
        }
        __syncwarp();
        const int b = kb > c0 ? kb : c0, e = ke < c1 ? ke : c1;
        for (int k = b; k < e; ++k) d += park[k - c0];
        __syncwarp();
      }
    } else if (mine) {
      // column starts that are not in order: each lane reads its own column
      d = column_by_thread(p, kb, ke, xj, cost, sense, row_dual, v.activity, v.error);
    }
    if (mine) column_terms(p, j, xj, cost, d, acc);
  }
  block_total<5, kThreads>(acc, kColumnMax, sh);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int s = 0; s < 5; ++s) v.col_partials[(size_t)blockIdx.x * kSlots + s] = acc[s];
  }
}

// Rows, then the last block to arrive folds both passes' partials (each thread the same blocks
// in the same order whichever block is last) and writes the residual block: as a kernel of its own
// with one folding thread that step took 155 us, most of the check.
__global__ void __launch_bounds__(kThreads) row_kernel(sankhya_pdhg_problem p, const double* row_dual,
                                                       double* base, int col_blocks, double* out) {
  const View v = carve(base);
  __shared__ double sh[kThreads / 32][5];
  __shared__ bool last;
  const double sense = p.maximize ? -1.0 : 1.0;
  double acc[5] = {0, 0, 0, 0, 0};
  const int stride = gridDim.x * blockDim.x;
  cudaGridDependencySynchronize();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < p.num_rows; i += stride)
    row_terms(p, i, v.activity[i], -sense * row_dual[i], acc);
  block_total<5, kThreads>(acc, kRowMax, sh);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int s = 0; s < 5; ++s) v.row_partials[(size_t)blockIdx.x * kSlots + s] = acc[s];
    __threadfence();
    last = atomicAdd(v.arrived, 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (!last) return;
  const auto total = [&](const double* partials, int blocks, unsigned max_mask, double (&t)[5]) {
#pragma unroll
    for (int s = 0; s < 5; ++s) t[s] = 0.0;
    for (int b = threadIdx.x; b < blocks; b += kThreads)
#pragma unroll
      for (int s = 0; s < 5; ++s) {
        const double o = __ldcg(partials + (size_t)b * kSlots + s);
        t[s] = ((max_mask >> s) & 1u) ? dmax(t[s], o) : t[s] + o;
      }
    __syncthreads();  // sh is free
    block_total<5, kThreads>(t, max_mask, sh);
  };
  double c[5], r[5];
  total(v.col_partials, col_blocks, kColumnMax, c);
  total(v.row_partials, gridDim.x, kRowMax, r);
  if (threadIdx.x == 0) write_residuals(c, r, __ldcg(v.error) != 0u, out);
}

// Device address of g_noalloc_scratch on the current device. In host code the array's name is
// only a stand-in for the symbol; kernels must be handed this address. It is resolved on every
// call with the caller's device current: the lookup allocates nothing and queues no work, and
// a cached address would go stale when the module is loaded again (after cudaDeviceReset, or
// under another context the caller makes current). The first call on a device is the one that
// loads this library's device code there (CUDA loads modules lazily), so make it before any
// stream capture.
int scratch_for_current_device(double** out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    sih26::g_last_error = "no current CUDA device";
    return SANKHYA_GPU_NO_COMPATIBLE_DEVICE;
  }
  void* p = nullptr;
  const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
  if (e != cudaSuccess || p == nullptr) {
    sih26::g_last_error = std::string("cudaGetSymbolAddress(g_noalloc_scratch) on device ") +
                          std::to_string(dev) + ": " + cudaGetErrorString(e);
    return SANKHYA_GPU_INIT_FAILED;
  }
  *out = static_cast<double*>(p);
  return SANKHYA_GPU_SUCCESS;
}

}  // namespace

extern "C" int sankhya_pdhg_gpu_residuals_noalloc(const sankhya_pdhg_problem* problem,
                                                  const double* x, const double* row_dual,
                                                  double* residuals_out, void* stream) {
  using sih26::g_last_error;
  if (!problem || !x || !residuals_out || (problem->num_rows > 0 && !row_dual)) {
    g_last_error = "problem, x, row_dual and residuals_out must be device pointers, not NULL";
    return SANKHYA_GPU_INVALID_ARGUMENT;
  }
  const sankhya_pdhg_problem& p = *problem;
  if (p.num_rows < 0 || p.num_cols < 0 || p.num_nonzeros < 0 || !p.col_starts ||
      (p.num_nonzeros > 0 && (!p.row_indices || !p.values)) ||
      (p.num_cols > 0 && (!p.cost || !p.col_lower || !p.col_upper)) ||
      (p.num_rows > 0 && (!p.row_lower || !p.row_upper))) {
    g_last_error = "malformed problem: negative size or NULL array";
    return SANKHYA_GPU_INVALID_ARGUMENT;
  }
  if ((size_t)p.num_rows > kMaxRows) {
    char buf[160];
    std::snprintf(buf, sizeof buf,
                  "%d rows exceed the %zu this entry point's fixed scratch can hold; use "
                  "sankhya_pdhg_gpu_solve, which allocates",
                  p.num_rows, kMaxRows);
    g_last_error = buf;
    return SANKHYA_GPU_INVALID_ARGUMENT;
  }
  double* base = nullptr;
  const int rc = scratch_for_current_device(&base);
  if (rc != SANKHYA_GPU_SUCCESS) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const auto blocks_for = [](int count) {
    int b = (count + kThreads - 1) / kThreads;
    return b < 1 ? 1 : (b > kGridBlocks ? kGridBlocks : b);
  };
  const long long work = (long long)p.num_nonzeros + p.num_cols + p.num_rows;
  if (p.num_rows <= kSmallRows && work <= kSmallWork) {
    small_kernel<<<1, kSmallThreads, 0, s>>>(p, x, row_dual, residuals_out);
  } else {
    const int cb = blocks_for(p.num_cols), rb = blocks_for(p.num_rows);
    clear_kernel<<<rb, kThreads, 0, s>>>(base, p.num_rows);
    cudaLaunchAttribute overlap{};
    overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    overlap.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t lc{};
    lc.blockDim = dim3(kThreads);
    lc.stream = s;
    lc.attrs = &overlap;
    lc.numAttrs = 1;
    lc.gridDim = dim3(cb);
    (void)cudaLaunchKernelEx(&lc, column_kernel, p, x, row_dual, base);
    lc.gridDim = dim3(rb);
    (void)cudaLaunchKernelEx(&lc, row_kernel, p, row_dual, base, cb, residuals_out);
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    g_last_error = std::string("launch failed: ") + cudaGetErrorString(e);
    return SANKHYA_GPU_KERNEL_LAUNCH_FAILED;
  }
  return SANKHYA_GPU_SUCCESS;
}
