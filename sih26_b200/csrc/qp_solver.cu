// Convex QP on the GPU behind sankhya_qp_gpu_solve (include/sankhya_pdhg_gpu.h): the reference's
// Condat-Vu method (src/qp/qp_condat_vu.cpp:150-323) on the LP engine's fused SpMV phases.
//
//   x'   = proj_box(x - tau (c_s + Q_s x + A'y))        c_s = sense c, Q_s = sense Q
//   xbar = 2 x' - x
//   y'   = v - sigma proj_C(v / sigma),  v = y + sigma A xbar
//
// Phase P runs over the rows of C = [A' | Q_s] (one row per column of the LP), gathering y for
// the A' part and x for the Q part, so the gradient is one fused row sum; phase D runs over the
// rows of A gathering xbar. Every 50 iterations (the reference's cadence, counted the same way)
// two more passes measure the termination residuals: max_i |Ax - proj(Ax)| and
// max_j |x - proj(x - gradient)|. Steps come from the reference's own power iterations for
// ||A|| and ||Q||, in its order of operations on the device or the host, so tau and sigma are the
// reference's to the bit. Everything is FP64, as in the reference.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "arena.cuh"
#include "convexity.cuh"
#include "packed_host.cuh"
#include "qp_norms.cuh"
#include "pdhg_host.cuh"
#include "pdhg_kernels.cuh"
#include "sankhya_pdhg_gpu.h"

namespace sih26 {

extern thread_local std::string g_last_error;

namespace {

// ---- device -----------------------------------------------------------------------------

struct QpDev {
  int m, n;
  Csr<double> A, C;  // A in permuted rows; C = [A' | Q_s] in permuted columns
  Part pa, pc;
  const double* c;   // sense c, permuted
  const double* cl;
  const double* cu;
  const double* rl;
  const double* ru;
  double* x[2];
  double* xbar;
  double* y[2];
  double* partials;  // [G][kPartSlots]
  Ctrl* ctrl;        // iteration, state, the two residuals in best.absolute_primal / _dual
  GridBarrier bar;
  double tau, sigma, tolerance;
  long long iteration_limit;
};

// sum_k C_jk z_k with z = [y; x]
struct CombinedGather {
  const double* y;
  const double* x;
  int m;
  __device__ __forceinline__ double at(int k) const { return k < m ? ld(y + k) : ld(x + (k - m)); }
  __device__ __forceinline__ void add(double (&s)[1], double a, int k) const { s[0] += a * at(k); }
  __device__ __forceinline__ double product(int, double a, int k) const { return a * at(k); }
  __device__ __forceinline__ double raw(int, int k) const { return k < m ? y[k] : x[k - m]; }
};

struct QpPrimal {
  const double* x;
  double* xn;
  double* xbar;
  const double* c;
  const double* cl;
  const double* cu;
  double tau;
  struct In {
    double xo, c, lo, hi;
  };
  __device__ __forceinline__ In load(int j) const {
    return In{ld(x + j), __ldg(c + j), __ldg(cl + j), __ldg(cu + j)};
  }
  __device__ __forceinline__ void apply(int j, const double (&s)[1], const In& v, double (&)[1]) const {
    const double xp = project(v.xo - tau * (v.c + s[0]), v.lo, v.hi);
    xn[j] = xp;
    xbar[j] = 2.0 * xp - v.xo;
  }
};

struct QpDual {
  const double* y;
  double* yn;
  const double* rl;
  const double* ru;
  double sigma;
  struct In {
    double yo, lo, hi;
  };
  __device__ __forceinline__ In load(int i) const { return In{ld(y + i), __ldg(rl + i), __ldg(ru + i)}; }
  __device__ __forceinline__ void apply(int i, const double (&s)[1], const In& v, double (&)[1]) const {
    const double u = v.yo + sigma * s[0];
    yn[i] = u - sigma * project(u / sigma, v.lo, v.hi);
  }
};

// termination measures (qp_condat_vu.cpp:263-289)
struct QpPrimalResidual {
  const double* rl;
  const double* ru;
  struct In {
    double lo, hi;
  };
  __device__ __forceinline__ In load(int i) const { return In{__ldg(rl + i), __ldg(ru + i)}; }
  __device__ __forceinline__ void apply(int, const double (&s)[1], const In& v, double (&acc)[2]) const {
    acc[0] = dmax(acc[0], fabs(s[0] - project(s[0], v.lo, v.hi)));
  }
};
struct QpDualResidual {
  const double* x;
  const double* c;
  const double* cl;
  const double* cu;
  struct In {
    double xo, c, lo, hi;
  };
  __device__ __forceinline__ In load(int j) const {
    return In{ld(x + j), __ldg(c + j), __ldg(cl + j), __ldg(cu + j)};
  }
  __device__ __forceinline__ void apply(int, const double (&s)[1], const In& v, double (&acc)[2]) const {
    const double g = v.c + s[0];
    acc[1] = dmax(acc[1], fabs(v.xo - project(v.xo - g, v.lo, v.hi)));
  }
};

// Cooperative: runs iterations until the limit, the chunk end or convergence. Ctrl fields
// used: iteration (the reference's loop counter), state, cur, best.absolute_primal/_dual.
//
// kPack: the blocks' parts of C and A are in shared memory for the launch (packed.cuh), for problems whose
// parts fit with their values; the same bits. B200, a solve without
// and with: 800 x 2,000 750 steps 12.6 and 6.8 ms, 10,007 x 25,001 1,000 steps 36.6 and 28.7.
template <bool kPack>
__global__ void __launch_bounds__(kThreads, 2) qp_kernel(QpDev Q, Packed<double> pk, long long max_steps) {
  __shared__ Ctrl c;
  __shared__ double sh[kWarps * 2];
  double* stream = warp_stream();
  if (threadIdx.x == 0) {
    c = *Q.ctrl;
    // read once per launch, before the first barrier, so every block sees the same flag
    c.time_up |= *((volatile int*)Q.bar.time_up);
  }
  __syncthreads();
  if (c.state != kRunning) return;
  __shared__ PackedView<double> side[2];  // rows of C, rows of A
  if constexpr (kPack) {
    const PackedView<double> rows_c = packed_load(pk.at, pk.plan.side[0], Q.C.ptr);
    const PackedView<double> rows_a = packed_load(pk.a, pk.plan.side[1], Q.A.ptr);
    packed_fetch(rows_c);
    packed_fetch(rows_a);
    if (threadIdx.x == 0) {
      side[0] = rows_c;
      side[1] = rows_a;
    }
    copy_wait();
    __syncthreads();
  }
  const auto phase = [&](auto of_c, const auto& gather, const auto& step, auto& acc) {
    constexpr int kSlots = std::extent_v<std::remove_reference_t<decltype(acc)>>;
    constexpr bool kC = decltype(of_c)::value;
    if constexpr (kPack) {
      unsigned char* mem = packed_smem();
      packed_phase<true>(side[kC ? 0 : 1], reinterpret_cast<double*>(mem + pk.plan.gat),
                         reinterpret_cast<double*>(mem + pk.plan.seg_sum), gather, step, acc);
    } else if constexpr (kC) {
      run_phase<1, kSlots>(Q.C.ptr, Q.C.idx, Q.C.val, Q.pc, gather, step, acc, stream);
    } else {
      run_phase<1, kSlots>(Q.A.ptr, Q.A.idx, Q.A.val, Q.pa, gather, step, acc, stream);
    }
  };
  constexpr std::true_type over_c{};
  constexpr std::false_type over_a{};
  const int G = gridDim.x;
  for (long long step = 0; step < max_steps; ++step) {
    if (c.iteration >= Q.iteration_limit) {
      if (threadIdx.x == 0) c.state = kIterationLimit;
      break;
    }
    if (c.time_up) {
      if (threadIdx.x == 0) c.state = kTimeLimit;
      break;
    }
    const int cur = c.cur, nxt = cur ^ 1;
    double dummy[1] = {0.0};
    phase(over_c, CombinedGather{Q.y[cur], Q.x[cur], Q.m},
          QpPrimal{Q.x[cur], Q.x[nxt], Q.xbar, Q.c, Q.cl, Q.cu, Q.tau}, dummy);
    if (!grid_barrier(Q.bar)) goto device_error;
    phase(over_a, Gather1<double>{Q.xbar}, QpDual{Q.y[cur], Q.y[nxt], Q.rl, Q.ru, Q.sigma}, dummy);
    if (!grid_barrier(Q.bar)) goto device_error;
    // the reference checks after the step when its counter is a multiple of 50, then counts
    if (c.iteration % 50 == 0) {
      double acc[2] = {0.0, 0.0};
      phase(over_a, Gather1<double>{Q.x[nxt]}, QpPrimalResidual{Q.rl, Q.ru}, acc);
      if constexpr (kPack) __syncthreads();  // both gather into one buffer
      phase(over_c, CombinedGather{Q.y[nxt], Q.x[nxt], Q.m}, QpDualResidual{Q.x[nxt], Q.c, Q.cl, Q.cu}, acc);
      block_reduce<2, 3u>(acc, sh);
      write_partials(Q.partials, 0, acc, 2);
      if (!grid_barrier(Q.bar)) goto device_error;
      double tot[2];
      reduce_partials<2, 3u>(Q.partials, 0, tot, sh);
      if (threadIdx.x == 0) {
        c.best.absolute_primal = tot[0];
        c.best.absolute_dual = tot[1];
        if (tot[0] <= Q.tolerance && tot[1] <= Q.tolerance) {
          c.state = kConverged;
          c.converged = 1;
        }
      }
    }
    if (threadIdx.x == 0) {
      c.cur = nxt;
      if (c.state != kConverged) ++c.iteration;
    }
    __syncthreads();
    if (c.state != kRunning) break;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *Q.ctrl = c;
  return;
device_error:
  if (blockIdx.x == 0 && threadIdx.x == 0) Q.ctrl->state = kDeviceError;
}

// ---- host --------------------------------------------------------------------------------

// Nonzeros of A and Q_s together from which the norms are estimated on the device (qp_norms.cuh), beside the
// layout. A solve on this side and the other, in ms: 13,000 entries 1.67 and 1.70, 26,000 6.3 and 6.7, 44,000
// 2.8 and 3.7, 320,000 18.8 and 27.1, 520,000 26 and 42; two entries 0.47 and 0.31.
constexpr long long kDeviceNorms = 20000;

// Unless a row or column holds most of it: its ordered sum is one warp's chain of loads and additions, 18 ns an
// entry (a vector's 4), against the host's 1.3 an operation. A solve on the device and here, in ms: one row of 20,000
// with a diagonal Q 10.3 and 6.0, of 200,000 104 and 65; 10 rows of 200,000 128 and 124, 100 of some 1,000 21 and 53.
bool norms_on_device(int n, long long nnz_a, long long nnz_q, int longest) {
  const double device_ns = 18.0 * longest + 4.0 * n;
  const double host_ns = 1.3 * (2.0 * static_cast<double>(nnz_a) + static_cast<double>(nnz_q) + 2.0 * n);
  return nnz_a + nnz_q >= kDeviceNorms && device_ns < host_ns;
}

// The reference's spectral_norm (qp_condat_vu.cpp:64-97): 20 power iterations on A'A from
// mt19937(26119) uniform(-1, 1), multiply_add / transpose_multiply_add in their order.
double qp_norm_a(const sankhya_pdhg_problem& p) {
  const int m = p.num_rows, n = p.num_cols;
  if (m == 0 || n == 0 || p.num_nonzeros == 0) return 0.0;
  std::vector<double> v(n), av(m);
  uniform_draws(26119u, -1.0, 1.0, n, v.data());
  double estimate = 0.0;
  for (int it = 0; it < 20; ++it) {
    double norm = 0.0;
    for (double t : v) norm += t * t;
    norm = std::sqrt(norm);
    if (norm <= 0.0) return 0.0;
    for (double& t : v) t /= norm;
    std::fill(av.begin(), av.end(), 0.0);
    for (int j = 0; j < n; ++j) {
      const double xj = 1.0 * v[j];
      if (xj == 0.0) continue;
      for (int k = p.col_starts[j]; k < p.col_starts[j + 1]; ++k) av[p.row_indices[k]] += p.values[k] * xj;
    }
    std::fill(v.begin(), v.end(), 0.0);
    for (int j = 0; j < n; ++j) {
      double dot = 0.0;
      for (int k = p.col_starts[j]; k < p.col_starts[j + 1]; ++k) dot += p.values[k] * av[p.row_indices[k]];
      v[j] += 1.0 * dot;
    }
    double next = 0.0;
    for (double t : v) next += t * t;
    estimate = std::sqrt(std::sqrt(next));
  }
  return estimate;
}

// Q v from the stored lower triangle (qp_condat_vu.cpp:137-150)
void qp_hessian_multiply(int n, const sankhya_qp_hessian& h, const std::vector<double>& v,
                         std::vector<double>& out) {
  std::fill(out.begin(), out.end(), 0.0);
  for (int j = 0; j < n; ++j) {
    for (int k = h.col_starts[j]; k < h.col_starts[j + 1]; ++k) {
      const int i = h.row_indices[k];
      const double value = h.values[k];
      out[i] += value * v[j];
      if (i != j) out[j] += value * v[i];
    }
  }
}

// The reference's hessian_norm (qp_condat_vu.cpp:101-134): 20 power iterations on Q from
// mt19937(20260826) uniform(-1, 1); the estimate is |v'Qv| with v normalised.
double qp_norm_q(int n, const sankhya_qp_hessian& h) {
  if (h.num_nonzeros == 0 || n == 0) return 0.0;
  std::vector<double> v(n), qv(n);
  uniform_draws(20260826u, -1.0, 1.0, n, v.data());
  double estimate = 0.0;
  for (int it = 0; it < 20; ++it) {
    double norm = 0.0;
    for (double t : v) norm += t * t;
    norm = std::sqrt(norm);
    if (norm <= 0.0) return 0.0;
    for (double& t : v) t /= norm;
    qp_hessian_multiply(n, h, v, qv);
    double next = 0.0;
    for (int i = 0; i < n; ++i) next += qv[i] * v[i];
    estimate = std::fabs(next);
    v = qv;
  }
  return estimate;
}

// check_convexity (src/qp/convexity.cpp:30-134): LDL' of sense * Q without interchanges, up to 2,000
// columns. Returns "" when convex, else the reason (the reference's wording). The factorisation runs
// on the device (convexity.cuh) from kDeviceConvexity columns on; below, the host is through before a
// launch would be, and it serves a machine without a GPU, where a refusal needs none.
constexpr int kDeviceConvexity = 96;

std::string not_convex_pivot(double pivot, int column) {
  char buf[256];
  std::snprintf(buf, sizeof buf,
                "the quadratic objective is not convex: LDL^T reached a pivot of %.6g at "
                "column %d",
                pivot, column);
  return buf;
}

std::string factor_on_host(int n, const sankhya_qp_hessian& h, double sense, double slack) {
  const size_t un = static_cast<size_t>(n);
  std::vector<double> q(un * un, 0.0);
  for (int j = 0; j < n; ++j)
    for (int k = h.col_starts[j]; k < h.col_starts[j + 1]; ++k) q[h.row_indices[k] * un + j] = sense * h.values[k];
  std::vector<double> l(un * un, 0.0), d(un, 0.0);
  for (int j = 0; j < n; ++j) {
    double pivot = q[static_cast<size_t>(j) * un + j];
    for (int k = 0; k < j; ++k) pivot -= l[j * un + k] * l[j * un + k] * d[k];
    if (pivot < -slack) return not_convex_pivot(pivot, j);
    if (pivot <= slack) continue;
    d[j] = pivot;
    for (int i = j + 1; i < n; ++i) {
      double sum = q[i * un + j];
      for (int k = 0; k < j; ++k) sum -= l[i * un + k] * l[j * un + k] * d[k];
      l[i * un + j] = sum / pivot;
    }
  }
  return "";
}

std::string factor_on_device(int n, const sankhya_qp_hessian& h, double sense, double slack, int device, int sms) {
  cudaStream_t stream;
  SIH26_CUDA(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking), SANKHYA_GPU_INIT_FAILED);
  struct StreamGuard {
    cudaStream_t s;
    ~StreamGuard() { cudaStreamDestroy(s); }
  } sg{stream};
  Arena a;
  a.set_device(device);
  a.set_stream(stream);
  const int* cs = a.upload_raw(h.col_starts, n + 1);
  const int* ri = a.upload_raw(h.row_indices, h.num_nonzeros);
  const double* val = a.upload_raw(h.values, h.num_nonzeros);
  ConvexityRun R{};
  R.n = n;
  R.slack = slack;
  R.w = a.zeros<double>(static_cast<size_t>(n) * n);
  R.l = a.alloc<double>(static_cast<size_t>(n) * kPanel);
  struct Verdict {
    int column;
    int pad;
    double pivot;
  };
  Verdict verdict{-2, 0, 0.0};
  Verdict* out = a.upload_raw(&verdict, 1);
  R.column = &out->column;
  R.pivot = &out->pivot;
  R.bar = GridBarrier{a.zeros<unsigned>(2), a.zeros<int>(2), 4000000000ull, a.zeros<int>(1), 0ull, -1};
  hessian_scatter<<<(n + 255) / 256, 256, 0, stream>>>(cs, ri, val, n, sense, R.w);
  SIH26_CUDA(cudaGetLastError(), SANKHYA_GPU_KERNEL_LAUNCH_FAILED);
  // a block per tile of the first panel's update, at most one per SM
  const int tiles = (n + kTile - 1) / kTile;
  const int G = std::max(1, std::min(sms, tiles * (tiles + 1) / 2));
  void* args[] = {&R};
  SIH26_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(convexity_kernel), dim3(G), dim3(kThreads),
                                         args, 0, stream), SANKHYA_GPU_KERNEL_LAUNCH_FAILED);
  SIH26_CUDA(cudaMemcpyAsync(&verdict, out, sizeof verdict, cudaMemcpyDeviceToHost, stream), SANKHYA_GPU_COPY_FAILED);
  SIH26_CUDA(cudaStreamSynchronize(stream), SANKHYA_GPU_SYNC_FAILED);
  if (verdict.column == -2) throw Failure{SANKHYA_GPU_DEVICE_TIMEOUT, "a grid barrier timed out in the convexity test"};
  return verdict.column < 0 ? std::string() : not_convex_pivot(verdict.pivot, verdict.column);
}

std::string qp_convexity(int n, const sankhya_qp_hessian& h, double sense, int device) {
  if (h.num_nonzeros == 0) return "";
  constexpr int kDenseLimit = 2000;
  constexpr double kPivotSlackFactor = 1e-10;
  char buf[256];
  if (n > kDenseLimit) {
    std::snprintf(buf, sizeof buf,
                  "convexity could not be established: %d columns exceeds the %d the dense "
                  "convexity test can decide",
                  n, kDenseLimit);
    return buf;
  }
  std::vector<double> diagonal(n, 0.0);
  double largest_diagonal = 0.0;
  for (int j = 0; j < n; ++j)
    for (int k = h.col_starts[j]; k < h.col_starts[j + 1]; ++k)
      if (h.row_indices[k] == j) {
        diagonal[j] = sense * h.values[k];
        largest_diagonal = std::max(largest_diagonal, std::fabs(diagonal[j]));
      }
  const double slack = kPivotSlackFactor * std::max(1.0, largest_diagonal);
  for (int i = 0; i < n; ++i) {
    if (diagonal[i] < -slack) {
      std::snprintf(buf, sizeof buf,
                    "the quadratic objective is not convex: the Hessian diagonal for column %d "
                    "is %.6g in minimization sense",
                    i, diagonal[i]);
      return buf;
    }
  }
  if (n >= kDeviceConvexity) {
    int devices = 0, sms = 0, major = 0;
    if (cudaGetDeviceCount(&devices) == cudaSuccess && device >= 0 && device < devices &&
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) == cudaSuccess &&
        cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device) == cudaSuccess && major >= 10) {
      SIH26_CUDA(cudaSetDevice(device), SANKHYA_GPU_INIT_FAILED);
      return factor_on_device(n, h, sense, slack, device, sms);
    }
    cudaGetLastError();
  }
  return factor_on_host(n, h, sense, slack);
}

void check_hessian(const sankhya_pdhg_problem& p, const sankhya_qp_hessian& h) {
  const auto bad = [](const std::string& why) { throw Failure{SANKHYA_GPU_INVALID_ARGUMENT, why}; };
  const int n = p.num_cols;
  if (h.num_nonzeros < 0) bad("negative Hessian size");
  if (!h.col_starts) bad("Hessian col_starts is NULL");
  if (h.num_nonzeros > 0 && (!h.row_indices || !h.values)) bad("Hessian arrays are NULL");
  if (h.col_starts[0] != 0 || h.col_starts[n] != h.num_nonzeros) bad("Hessian col_starts inconsistent");
  for (int j = 0; j < n; ++j) {
    if (h.col_starts[j + 1] < h.col_starts[j]) bad("Hessian col_starts decreases");
    for (int k = h.col_starts[j]; k < h.col_starts[j + 1]; ++k) {
      const int i = h.row_indices[k];
      if (i < j || i >= n) bad("the Hessian must be a lower triangle (row >= column < n)");
      if (k > h.col_starts[j] && i <= h.row_indices[k - 1]) bad("Hessian rows not ascending");
      if (!std::isfinite(h.values[k])) bad("non-finite Hessian entry");
    }
  }
}

Part upload_part(Arena& a, const HostPart& hp) {
  Part p;
  p.blk_seg_begin = a.upload_same(hp.blk_seg_begin);
  p.segs = a.upload_same(hp.segs);
  p.blk_long_begin = a.upload_same(hp.blk_long_begin);
  p.longs = a.upload_same(hp.longs);
  p.blk_item_begin = a.upload_same(hp.blk_item_begin);
  p.items = a.upload_same(hp.items);
  p.seg_sum = a.zeros<double>(hp.segs.size() * 2 + 1);
  return p;
}

std::vector<int> order_desc(const std::vector<int>& len) {
  std::vector<int> order(len.size());
  for (size_t i = 0; i < order.size(); ++i) order[i] = static_cast<int>(i);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return len[a] > len[b]; });
  return order;
}

int qp_solve_impl(const sankhya_pdhg_problem& prob, const sankhya_qp_hessian& hes,
                  const sankhya_pdhg_params& prm, sankhya_pdhg_result* res) {
  using Clock = std::chrono::steady_clock;
  const Clock::time_point t0 = Clock::now();
  const auto since = [&]() { return std::chrono::duration<double>(Clock::now() - t0).count(); };
  check_structure(prob);
  check_hessian(prob, hes);
  const int m = prob.num_rows, n = prob.num_cols;
  res->status = SANKHYA_PDHG_NOT_SOLVED;
  res->converged = 0;
  res->iterations = res->attempts = res->restarts = res->evaluations = res->fp32_iterations = 0;
  res->message[0] = '\0';
  const std::string why = validate_model(prob);
  const double sense = prob.maximize ? -1.0 : 1.0;
  std::string convex = prm.qp_assume_convex ? std::string() : qp_convexity(n, hes, sense, prm.device);
  if (!why.empty() || !convex.empty()) {
    res->status = SANKHYA_PDHG_MODEL_ERROR;
    std::snprintf(res->message, sizeof res->message, "%s", (why.empty() ? convex : why).c_str());
    return SANKHYA_GPU_SUCCESS;
  }
  int devices = 0;
  if (cudaGetDeviceCount(&devices) != cudaSuccess || devices == 0)
    throw Failure{SANKHYA_GPU_NO_COMPATIBLE_DEVICE, "no CUDA device is visible"};
  if (prm.device < 0 || prm.device >= devices)
    throw Failure{SANKHYA_GPU_INVALID_ARGUMENT, "device ordinal out of range"};
  SIH26_CUDA(cudaSetDevice(prm.device), SANKHYA_GPU_INIT_FAILED);
  int sms = 0, major = 0;
  SIH26_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, prm.device), SANKHYA_GPU_INIT_FAILED);
  SIH26_CUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, prm.device), SANKHYA_GPU_INIT_FAILED);
  if (major < 10)
    throw Failure{SANKHYA_GPU_NO_COMPATIBLE_DEVICE, "this library is built for sm_100a (B200)"};

  cudaStream_t stream;
  SIH26_CUDA(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking), SANKHYA_GPU_INIT_FAILED);
  struct StreamGuard {
    cudaStream_t s;
    ~StreamGuard() { cudaStreamDestroy(s); }
  } sg{stream};
  Arena a;  // destroyed before the stream (declared after it)
  a.set_device(prm.device);
  a.set_stream(stream);
  long long launches = 0;

  // ---- rows of A and of the full symmetric Q_s, each in the order in which the reference's products add
  // to it (a column's entries reach their rows, then the column's own row) ----
  std::vector<int> rlen(m, 0), clen(n, 0), q_ptr(n + 1, 0);
  for (int j = 0; j < n; ++j) {
    for (int k = prob.col_starts[j]; k < prob.col_starts[j + 1]; ++k) ++rlen[prob.row_indices[k]];
    for (int k = hes.col_starts[j]; k < hes.col_starts[j + 1]; ++k) {
      const int i = hes.row_indices[k];
      ++q_ptr[i + 1];
      if (i != j) ++q_ptr[j + 1];
    }
  }
  for (int j = 0; j < n; ++j) {
    clen[j] = prob.col_starts[j + 1] - prob.col_starts[j] + q_ptr[j + 1];
    q_ptr[j + 1] += q_ptr[j];
  }
  std::vector<int> q_idx(q_ptr[n]);
  std::vector<double> q_val(q_ptr[n]);
  {
    std::vector<int> next(q_ptr.begin(), q_ptr.end() - 1);
    const auto put = [&](int row, int col, double v) {
      q_idx[next[row]] = col;
      q_val[next[row]++] = v;
    };
    for (int j = 0; j < n; ++j)
      for (int k = hes.col_starts[j]; k < hes.col_starts[j + 1]; ++k) {
        const int i = hes.row_indices[k];
        const double v = sense * hes.values[k];
        put(i, j, v);
        if (i != j) put(j, i, v);
      }
  }

  // ---- norm estimates: on the device beside the layout, or here. The sign of Q_s cancels. ----
  double norms[2] = {0.0, 0.0};
  int longest = 0;
  for (int i = 0; i < m; ++i) longest = std::max(longest, rlen[i]);
  for (int j = 0; j < n; ++j)
    longest = std::max({longest, prob.col_starts[j + 1] - prob.col_starts[j], q_ptr[j + 1] - q_ptr[j]});
  const bool device_norms = norms_on_device(n, prob.num_nonzeros, q_ptr[n], longest);
  double* d_scalars = nullptr;
  if (device_norms) {
    const bool has_a = m > 0 && n > 0 && prob.num_nonzeros > 0, has_q = hes.num_nonzeros > 0 && n > 0;
    d_scalars = a.zeros<double>(4);
    NormRun ra{}, rq{};
    std::vector<double> va(has_a ? n : 0), vq(has_q ? n : 0);
    if (has_a) {
      std::vector<int> r_ptr(m + 1, 0), r_idx(prob.num_nonzeros);
      std::vector<double> r_val(prob.num_nonzeros);
      for (int i = 0; i < m; ++i) r_ptr[i + 1] = r_ptr[i] + rlen[i];
      std::vector<int> next(r_ptr.begin(), r_ptr.end() - 1);
      for (int j = 0; j < n; ++j)
        for (int k = prob.col_starts[j]; k < prob.col_starts[j + 1]; ++k) {
          const int slot = next[prob.row_indices[k]]++;
          r_idx[slot] = j;
          r_val[slot] = prob.values[k];
        }
      uniform_draws(26119u, -1.0, 1.0, n, va.data());
      ra.first = NormMatrix{m, a.upload_same(r_ptr), a.upload_same(r_idx), a.upload_same(r_val)};
      ra.second = NormMatrix{n, a.upload_raw(prob.col_starts, n + 1), a.upload_raw(prob.row_indices, prob.num_nonzeros),
                             a.upload_raw(prob.values, prob.num_nonzeros)};
      ra.n = n;
      ra.square = 1;
      ra.v = const_cast<double*>(a.upload_same(va));
      ra.w = a.alloc<double>(m);
      ra.scalar = d_scalars;
    }
    if (has_q) {
      uniform_draws(20260826u, -1.0, 1.0, n, vq.data());
      rq.first = NormMatrix{n, a.upload_same(q_ptr), a.upload_same(q_idx), a.upload_same(q_val)};
      rq.n = n;
      rq.v = const_cast<double*>(a.upload_same(vq));
      rq.w = a.alloc<double>(n);
      rq.scalar = d_scalars + 2;
    }
    qp_norm_kernel<<<2 * kNormTeam, kThreads, 0, stream>>>(ra, rq);
    SIH26_CUDA(cudaGetLastError(), SANKHYA_GPU_KERNEL_LAUNCH_FAILED);
    ++launches;
  } else {
    norms[0] = qp_norm_a(prob);
    norms[1] = qp_norm_q(n, hes);
  }

  // ---- layout: rows of A by length; columns by the length of their row of C = [A' | Q_s] ----
  const std::vector<int> row_perm = order_desc(rlen), col_perm = order_desc(clen);
  std::vector<int> row_pos(m), col_pos(n);
  for (int t = 0; t < m; ++t) row_pos[row_perm[t]] = t;
  for (int t = 0; t < n; ++t) col_pos[col_perm[t]] = t;
  // A in permuted rows, entries in ascending permuted column
  std::vector<int> a_ptr(m + 1, 0);
  for (int t = 0; t < m; ++t) a_ptr[t + 1] = a_ptr[t] + rlen[row_perm[t]];
  std::vector<int> a_idx(prob.num_nonzeros);
  std::vector<double> a_val(prob.num_nonzeros);
  {
    std::vector<int> next(a_ptr.begin(), a_ptr.end() - 1);
    for (int t = 0; t < n; ++t) {
      const int j = col_perm[t];
      for (int k = prob.col_starts[j]; k < prob.col_starts[j + 1]; ++k) {
        const int slot = next[row_pos[prob.row_indices[k]]]++;
        a_idx[slot] = t;
        a_val[slot] = prob.values[k];
      }
    }
  }
  // C in permuted columns: A' entries (permuted row positions, ascending), then Q_s entries
  // (m + permuted column positions, ascending)
  std::vector<int> c_ptr(n + 1, 0);
  for (int t = 0; t < n; ++t) c_ptr[t + 1] = c_ptr[t] + clen[col_perm[t]];
  std::vector<int> c_idx(c_ptr[n]);
  std::vector<double> c_val(c_ptr[n]);
  for (int t = 0; t < n; ++t) {
    const int j = col_perm[t];
    std::vector<std::pair<int, double>> a_part, q_part;
    for (int k = prob.col_starts[j]; k < prob.col_starts[j + 1]; ++k)
      a_part.push_back({row_pos[prob.row_indices[k]], prob.values[k]});
    for (int k = q_ptr[j]; k < q_ptr[j + 1]; ++k) q_part.push_back({m + col_pos[q_idx[k]], q_val[k]});
    std::sort(a_part.begin(), a_part.end());
    std::sort(q_part.begin(), q_part.end());
    int at = c_ptr[t];
    for (const auto& e : a_part) { c_idx[at] = e.first; c_val[at++] = e.second; }
    for (const auto& e : q_part) { c_idx[at] = e.first; c_val[at++] = e.second; }
  }
  std::vector<double> cs(n), cl(n), cu(n), rl(m), ru(m);
  for (int t = 0; t < n; ++t) {
    const int j = col_perm[t];
    cs[t] = sense * prob.cost[j];
    cl[t] = prob.col_lower[j];
    cu[t] = prob.col_upper[j];
  }
  for (int t = 0; t < m; ++t) {
    rl[t] = prob.row_lower[row_perm[t]];
    ru[t] = prob.row_upper[row_perm[t]];
  }
  std::vector<double> x0(n);
  for (int t = 0; t < n; ++t) {
    double v = 0.0;
    if (host_finite_bound(cl[t]) && v < cl[t]) v = cl[t];
    else if (host_finite_bound(cu[t]) && v > cu[t]) v = cu[t];
    x0[t] = v;
  }

  // ---- device ----
  int bpsm = 0;
  SIH26_CUDA(cudaFuncSetAttribute(qp_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)stream_smem_bytes()), SANKHYA_GPU_INIT_FAILED);
  SIH26_CUDA(cudaFuncSetAttribute(qp_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPackedBytes),
              SANKHYA_GPU_INIT_FAILED);
  SIH26_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bpsm, qp_kernel<false>, kThreads, stream_smem_bytes()),
              SANKHYA_GPU_INIT_FAILED);
  if (bpsm < 1) throw Failure{SANKHYA_GPU_INIT_FAILED, "kernel does not fit on an SM"};
  int G = sms * std::min(bpsm, 2);
  const long long work = static_cast<long long>(c_ptr[n]) + prob.num_nonzeros + m + n;
  G = static_cast<int>(std::max<long long>(1, std::min<long long>(G, (work + 4095) / 4096)));

  const HostPart hpa = partition(a_ptr, G, kWarps, 0), hpc = partition(c_ptr, G, kWarps, 0);
  const size_t stage = 13 * (a_idx.size() + c_idx.size()) + 100 * static_cast<size_t>(m + n) + (size_t(256) << 10);
  if (stage <= (size_t(8) << 20)) a.begin_staging(stage);
  QpDev Q{};
  Q.m = m;
  Q.n = n;
  Q.A.ptr = a.upload_same(a_ptr);
  Q.A.idx = a.upload_same(a_idx);
  Q.A.val = Q.A.val64 = a.upload_same(a_val);
  Q.C.ptr = a.upload_same(c_ptr);
  Q.C.idx = a.upload_same(c_idx);
  Q.C.val = Q.C.val64 = a.upload_same(c_val);
  Q.pa = upload_part(a, hpa);
  Q.pc = upload_part(a, hpc);
  Q.c = a.upload_same(cs);
  Q.cl = a.upload_same(cl);
  Q.cu = a.upload_same(cu);
  Q.rl = a.upload_same(rl);
  Q.ru = a.upload_same(ru);
  Q.x[0] = a.upload_same(x0);
  Q.x[1] = a.upload_same(x0);
  Ctrl c0{};
  c0.state = kRunning;
  c0.iteration_limit = prm.iteration_limit < 0 ? 1000000ll : prm.iteration_limit;
  Q.ctrl = a.upload_raw(&c0, 1);
  a.end_staging();
  a.begin_zeros();
  Q.xbar = a.zeros<double>(n);
  Q.y[0] = a.zeros<double>(m);
  Q.y[1] = a.zeros<double>(m);
  Q.partials = a.zeros<double>(static_cast<size_t>(G) * kPartSlots);
  unsigned* bar_words = a.zeros<unsigned>(2);
  int* flags = a.zeros<int>(2);
  a.end_zeros();
  const HostPacked kc = pack(hpc, c_ptr, G), ka = pack(hpa, a_ptr, G);
  Packed<double> pk{};
  pk.plan = plan_packed<double>(kc, ka, G, sms, reinterpret_cast<const void*>(qp_kernel<true>), true);
  const bool packed = pk.plan.bytes > 0;
  if (packed) {
    pk.at = upload_packed<double>(a, kc, Q.pc, Q.C.ptr, Q.C.idx, Q.C.val, G, stream);
    pk.a = upload_packed<double>(a, ka, Q.pa, Q.A.ptr, Q.A.idx, Q.A.val, G, stream);
  }
  // ---- step sizes, as the reference (qp_condat_vu.cpp:183-196) ----
  if (device_norms) {
    double scalars[4];
    SIH26_CUDA(cudaMemcpyAsync(scalars, d_scalars, sizeof scalars, cudaMemcpyDeviceToHost, stream),
                SANKHYA_GPU_COPY_FAILED);
    SIH26_CUDA(cudaStreamSynchronize(stream), SANKHYA_GPU_SYNC_FAILED);
    norms[0] = scalars[1];
    norms[1] = scalars[3];
  }
  const double norm_a = norms[0];
  const double margin = 1.05;
  const double lq = margin * norms[1];
  const double a2 = margin * margin * std::max(norm_a * norm_a, 1e-12);
  const double tau = 1.0 / (lq / 2.0 + std::sqrt(a2) + 1e-12);
  const double sigma = (m > 0) ? (1.0 / tau - lq / 2.0) / (2.0 * a2) : 0.0;
  const double tolerance = prm.tolerance > 0.0 ? prm.tolerance : 1e-8;
  Q.bar = GridBarrier{bar_words, flags, 4000000000ull, flags + 1, 0ull, -1};
  Q.tau = tau;
  Q.sigma = sigma;
  Q.tolerance = tolerance;
  Q.iteration_limit = c0.iteration_limit;
  const bool timed = std::isfinite(prm.time_limit) && prm.time_limit > 0.0;

  Ctrl host{};
  long long steps = 256;
  if (packed) launches += 2;
  for (;;) {
    void* args[] = {&Q, &pk, &steps};
    SIH26_CUDA(cudaLaunchCooperativeKernel(packed ? reinterpret_cast<const void*>(qp_kernel<true>)
                                                  : reinterpret_cast<const void*>(qp_kernel<false>),
                                            dim3(G), dim3(kThreads), args,
                                            packed ? pk.plan.bytes : stream_smem_bytes(), stream),
                SANKHYA_GPU_KERNEL_LAUNCH_FAILED);
    ++launches;
    SIH26_CUDA(cudaMemcpyAsync(&host, Q.ctrl, sizeof(Ctrl), cudaMemcpyDeviceToHost, stream),
                SANKHYA_GPU_COPY_FAILED);
    SIH26_CUDA(cudaStreamSynchronize(stream), SANKHYA_GPU_SYNC_FAILED);
    if (host.state == kDeviceError) throw Failure{SANKHYA_GPU_DEVICE_TIMEOUT, "a grid barrier timed out"};
    if (host.state != kRunning) break;
    if (timed && since() > prm.time_limit) {
      host.state = kTimeLimit;
      break;
    }
    if (steps < 4096) steps *= 2;
  }
  // ---- outputs, un-permuted; the reference's Solution fields (qp_condat_vu.cpp:296-321) ----
  std::vector<double> hx(n), hy(m);
  const int cur = host.cur;
  SIH26_CUDA(cudaMemcpy(hx.data(), Q.x[cur], n * sizeof(double), cudaMemcpyDeviceToHost), SANKHYA_GPU_COPY_FAILED);
  if (m)
    SIH26_CUDA(cudaMemcpy(hy.data(), Q.y[cur], m * sizeof(double), cudaMemcpyDeviceToHost), SANKHYA_GPU_COPY_FAILED);
  std::vector<double> x(n), y(m);
  for (int t = 0; t < n; ++t) x[col_perm[t]] = hx[t];
  for (int t = 0; t < m; ++t) y[row_perm[t]] = hy[t];
  for (double v : x)
    if (!std::isfinite(v)) throw Failure{SANKHYA_GPU_NON_FINITE_OUTPUT, "the point is not finite"};
  std::vector<double> qx(n), aty(n, 0.0);
  qp_hessian_multiply(n, hes, x, qx);
  for (int j = 0; j < n; ++j) {
    double dot = 0.0;
    for (int k = prob.col_starts[j]; k < prob.col_starts[j + 1]; ++k) dot += prob.values[k] * y[prob.row_indices[k]];
    aty[j] = dot;
  }
  if (res->col_value) std::memcpy(res->col_value, x.data(), n * sizeof(double));
  if (res->row_dual) for (int i = 0; i < m; ++i) res->row_dual[i] = -sense * y[i];
  if (res->col_dual) for (int j = 0; j < n; ++j) res->col_dual[j] = prob.cost[j] + qx[j] + sense * aty[j];
  // Model::evaluate_objective (src/core/model.cpp:99-125): offset + c'x + 0.5 x'Qx, Q from its
  // lower triangle (an off-diagonal entry counts twice)
  double obj = prob.objective_offset;
  for (int j = 0; j < n; ++j) obj += prob.cost[j] * x[j];
  double quad = 0.0;
  for (int j = 0; j < n; ++j) {
    for (int k = hes.col_starts[j]; k < hes.col_starts[j + 1]; ++k) {
      const int i = hes.row_indices[k];
      quad += (i == j ? 0.5 : 1.0) * hes.values[k] * x[i] * x[j];
    }
  }
  obj += quad;
  res->objective = obj;
  res->converged = host.converged;
  res->iterations = host.iteration;
  res->attempts = host.iteration;
  res->spectral_norm = norm_a;
  std::memset(&res->residuals, 0, sizeof res->residuals);
  res->residuals.absolute_primal = host.best.absolute_primal;
  res->residuals.absolute_dual = host.best.absolute_dual;
  res->residuals.primal_objective = obj;
  // primal_infeasibility: the largest bound violation (Solution::recompute_quality)
  {
    std::vector<double> act(m, 0.0);
    for (int j = 0; j < n; ++j)
      for (int k = prob.col_starts[j]; k < prob.col_starts[j + 1]; ++k) act[prob.row_indices[k]] += prob.values[k] * x[j];
    double worst = 0.0;
    for (int j = 0; j < n; ++j) {
      if (host_finite_bound(prob.col_lower[j])) worst = std::max(worst, prob.col_lower[j] - x[j]);
      if (host_finite_bound(prob.col_upper[j])) worst = std::max(worst, x[j] - prob.col_upper[j]);
    }
    for (int i = 0; i < m; ++i) {
      if (host_finite_bound(prob.row_lower[i])) worst = std::max(worst, prob.row_lower[i] - act[i]);
      if (host_finite_bound(prob.row_upper[i])) worst = std::max(worst, act[i] - prob.row_upper[i]);
    }
    res->primal_infeasibility = worst;
    // the dual measures are the LP engines' (the QP's gradient is c + Qx): not measured here
    res->quality = sankhya_pdhg_quality{worst, NAN, NAN, NAN, NAN, NAN, NAN};
  }
  if (host.state == kConverged) {
    res->status = SANKHYA_PDHG_OPTIMAL;
    std::snprintf(res->message, sizeof res->message,
                  "converged after %lld iterations: primal residual %.3e, dual residual %.3e "
                  "(tolerance %.1e)",
                  host.iteration, host.best.absolute_primal, host.best.absolute_dual, tolerance);
  } else if (host.state == kTimeLimit) {
    res->status = SANKHYA_PDHG_TIME_LIMIT;
    std::snprintf(res->message, sizeof res->message, "time limit %.3gs reached", prm.time_limit);
  } else {
    res->status = SANKHYA_PDHG_ITERATION_LIMIT;
    std::snprintf(res->message, sizeof res->message, "iteration limit %lld reached", c0.iteration_limit);
  }
  res->dual_bound = res->status == SANKHYA_PDHG_OPTIMAL ? obj : (prob.maximize ? INFINITY : -INFINITY);
  res->kernel_launches = launches;
  res->total_seconds = since();
  res->solve_seconds = res->total_seconds;
  return SANKHYA_GPU_SUCCESS;
}

}  // namespace
}  // namespace sih26

extern "C" int sankhya_qp_gpu_solve(const sankhya_pdhg_problem* problem,
                                    const sankhya_qp_hessian* hessian,
                                    const sankhya_pdhg_params* params,
                                    sankhya_pdhg_result* result) {
  using namespace sih26;
  if (!problem || !hessian || !result) {
    g_last_error = "problem, hessian and result must not be NULL";
    return SANKHYA_GPU_INVALID_ARGUMENT;
  }
  sankhya_pdhg_params defaults;
  sankhya_pdhg_gpu_default_params(&defaults);
  if (!params) {
    defaults.tolerance = 1e-8;  // qp_tolerance (src/util/options.cpp:335-341)
    params = &defaults;
  }
  DeviceGuard guard;
  try {
    return qp_solve_impl(*problem, *hessian, *params, result);
  } catch (const Failure& f) {
    g_last_error = f.message;
    std::snprintf(result->message, sizeof result->message, "%s", f.message.c_str());
    result->status = SANKHYA_PDHG_NUMERICAL_ERROR;
    return f.code;
  } catch (const std::bad_alloc&) {
    g_last_error = "host allocation failed";
    return SANKHYA_GPU_OUT_OF_MEMORY;
  }
}
