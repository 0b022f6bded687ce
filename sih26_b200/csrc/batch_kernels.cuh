// Batched restarted PDHG: many independent LPs in one persistent launch.
//
// A team of thread blocks (resident.cuh) -- one block, or a thread-block cluster for the larger LPs --
// takes LPs from a device work queue (largest first) and runs the whole restarted PDHG of
// src/pdhg/pdhg.cpp:267-726 on one LP: the norm estimate, the attempts, the evaluations every 40
// accepted iterations with per-LP restarts and termination, and the final report. The gathered
// vectors are in shared memory where they fit (some 20,000 rows and columns together), the matrix too
// where it fits beside them, else streamed from L2; of larger LPs the gathered vector alone (up to 27,136
// entries), and beyond that its entries are gathered out of L2, by clusters in a launch of their own
// that leaves the shared memory to L1. An LP runs for at most `chunk_attempts` attempts per launch and keeps
// its state in device memory between launches, so a host loop can admit and retire LPs between launches.
//
// An LP's work partition is built for its group size alone, so its row sums follow the same
// code and summation order whatever else is in the batch: a result is the same alone and in
// the mix.
//
// Infeasibility and unboundedness: at every fourth evaluation the dual movement since the last
// restart is tested as a Farkas certificate and the last primal step as a primal ray (see
// certificate_test in pdhg_kernels.cuh); the host re-checks every candidate exactly with the
// reference's rules (src/core/certificate.cpp) before reporting it.
//
// One block per SM: a block's shared memory is the LP's, and an iteration bound by the latency of its own
// chain gains more from that than the SM from a second LP. FP64, us per Halpern iteration of one LP alone,
// gathering from L2 with two blocks a SM before and as here (300 at once, per LP): 2,252 nonzeros 10.2
// and 3.2 (0.07, 0.03), 15,752: 34 and 13 (0.32, 0.24), 16,561 on a cluster: 15.3 and 4.3 (0.55, 0.32),
// 112,727: 33 and 17 (2.1, 2.0). From L2, alone and of 36 at once: 450,000: 152 and 74 (10.7, 8.1), 1 million
// (100,000 x 250,000): 367 and 230, 10 million (1,000,000 x 2,500,000): 4,415 and 2,834.
#pragma once

#include "team_prep.cuh"

namespace sih26 {

constexpr int kClusterSize = 8;
constexpr long long kChunkNnz = 16384;  // nonzeros per block an attempt of chunk_attempts covers

struct BatchSlot {
  Prob<double> P;   // partitions built for the LP's group size (pai == pae, pati == pate)
  State<double> S;  // partials and barrier unused; cert_row, cert_col: the certificate's outputs
  ResidentPlan plan;
  RawLp raw;            // what the setup launch prepares the LP from
  const double* start;   // the norm estimate's random start, for S.xc
  const double* x_start;  // the starting point of an LP the host has prepared (raw.v null)
  double* zero;         // arrays that start at zero
  size_t zeros;
  double* x_out;    // report: unscaled x, permuted
  double* red_out;  // report: min-space reduced costs, permuted
  double* y_out;    // report: unscaled y (PDHG sign), permuted
};

// A new LP for the setup launch: its slot and what goes there.
struct NewSlot {
  BatchSlot slot;
  Ctrl ctrl;
  int index;
};

// One team per admitted LP (`group` blocks each): places its slot and control block, clears its
// state, and scales and lays out its matrix.
__global__ void __launch_bounds__(kThreads) batch_setup_kernel(const NewSlot* fresh, int group, BatchSlot* slots,
                                                               Ctrl* ctrls) {
  __shared__ BatchSlot b;
  const NewSlot& f = fresh[blockIdx.x / group];
  const auto copy = [](void* dst, const void* src, size_t bytes) {
    for (int w = threadIdx.x; w < (int)(bytes / 4); w += kThreads)
      static_cast<int*>(dst)[w] = static_cast<const int*>(src)[w];
  };
  copy(&b, &f.slot, sizeof b);
  const Team tm{group, group > 1 ? (int)cooperative_groups::this_cluster().block_rank() : 0};
  if (tm.rank == 0) {
    copy(slots + f.index, &f.slot, sizeof b);
    copy(ctrls + f.index, &f.ctrl, sizeof(Ctrl));
  }
  __syncthreads();
  const int base = tm.rank * kThreads + threadIdx.x, stride = tm.cs * kThreads;
  for (size_t k = base; k < b.zeros; k += stride) b.zero[k] = 0.0;
  double* start = reinterpret_cast<double*>(b.S.xc);
  for (int j = base; j < b.P.n; j += stride) start[j] = b.start[j];
  if (tm.cs > 1) tm.sync();  // the starting point goes over the zeros
  else __syncthreads();
  if (!b.raw.v)
    for (int j = base; j < b.P.n; j += stride)
      for (int k = 0; k < 3; ++k) b.raw.x0[k][j] = b.x_start[j];
  team_setup(b.P, b.raw, tm);
}

template <bool kOnlyL2 = false>
__device__ __forceinline__ void run_slot(const BatchSlot* from, BatchSlot& b, TeamShared& ts, SideView<double>& sp,
                                         SideView<double>& sd, const Team& tm, long long chunk_attempts) {
  for (int w = threadIdx.x; w < (int)(sizeof(BatchSlot) / 4); w += kThreads)
    reinterpret_cast<int*>(&b)[w] = reinterpret_cast<const int*>(from)[w];
  __syncthreads();
  // The chunk is a budget of work, not of attempts: chunk_attempts for an LP with at most
  // kChunkNnz nonzeros per block, proportionally fewer attempts (at least 8) for larger ones,
  // so a launch lasts about as long for every LP and no slot idles behind one large LP.
  const long long per_block = (long long)__ldg(b.P.A.ptr + b.P.m) / tm.cs;
  if (per_block > kChunkNnz && chunk_attempts < (1ll << 40)) {
    const long long scaled = chunk_attempts * kChunkNnz / per_block;
    chunk_attempts = scaled < 8 ? 8 : scaled;
  }
  team_solve<double, -1, kOnlyL2>(b.P, b.S, b.plan, b.plan, b.x_out, b.red_out, b.y_out, ts, sp, sd, sp, sd, tm,
                         chunk_attempts, 1 << 30);
}

// The persistent batch kernels: blocks (or clusters) take LPs from the active list through a
// device counter (the list is ordered largest first) until it is exhausted.
__global__ void __launch_bounds__(kThreads, 1) batch_kernel(const BatchSlot* slots, const int* active,
                                                            const int* active_count, int* queue_head,
                                                            long long chunk_attempts) {
  __shared__ TeamShared ts;
  __shared__ SideView<double> sp, sd;
  __shared__ BatchSlot b;
  __shared__ int s_take;
  const int count = *active_count;
  for (;;) {
    if (threadIdx.x == 0) s_take = atomicAdd(queue_head, 1);
    __syncthreads();
    const int q = s_take;
    __syncthreads();
    if (q >= count) break;
    run_slot(slots + active[q], b, ts, sp, sd, Team{1, 0}, chunk_attempts);
  }
}

// kOnlyL2: for LPs gathered out of L2, launched without dynamic shared memory.
template <bool kOnlyL2>
__global__ void __cluster_dims__(kClusterSize, 1, 1) __launch_bounds__(kThreads, 1)
    cluster_batch_kernel(const BatchSlot* slots, const int* active, const int* active_count,
                         int* queue_head, long long chunk_attempts) {
  __shared__ TeamShared ts;
  __shared__ SideView<double> sp, sd;
  __shared__ BatchSlot b;
  __shared__ int s_take;
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  const Team tm{kClusterSize, (int)cl.block_rank()};
  const int count = *active_count;
  for (;;) {
    if (tm.rank == 0 && threadIdx.x == 0) s_take = atomicAdd(queue_head, 1);
    cl.sync();
    const int q = *cl.map_shared_rank(&s_take, 0);
    cl.sync();
    if (q >= count) break;
    run_slot<kOnlyL2>(slots + active[q], b, ts, sp, sd, tm, chunk_attempts);
  }
}

// Copies the control blocks of the active LPs into one compact array for the host.
__global__ void gather_ctrl_kernel(const Ctrl* ctrls, const int* active, const int* active_count,
                                   Ctrl* out) {
  const int count = *active_count;
  for (int q = blockIdx.x; q < count; q += gridDim.x) {
    const int* src = reinterpret_cast<const int*>(ctrls + active[q]);
    int* dst = reinterpret_cast<int*>(out + q);
    for (int w = threadIdx.x; w < (int)(sizeof(Ctrl) / sizeof(int)); w += blockDim.x) dst[w] = src[w];
  }
}

}  // namespace sih26
