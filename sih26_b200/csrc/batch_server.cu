// Batched and served restarted PDHG behind the C ABI (sankhya_pdhg_server_* and
// sankhya_pdhg_gpu_batch_solve in include/sankhya_pdhg_gpu.h).
//
// A server owns one device memory pool (a fraction of free HBM, taken once at creation),
// a table of LP slots and one CUDA graph. submit() checks an LP and builds what needs no arithmetic
// on its values (permutations, row pointers, the work partition for one block -- or for an 8-block
// cluster when the LP has at least cluster_min_nnz nonzeros); step() admits waiting LPs that fit the
// pool -- one copy each, then one launch in which a block or cluster per LP scales and lays it out
// (team_prep.cuh) -- replays the graph (the single-block and the cluster
// persistent kernels side by side on forked streams, over every active LP of their
// class, each LP for at most chunk_attempts attempts),
// reads the compact control blocks back, re-checks every Farkas certificate on the host, and
// retires finished LPs with their answers. LPs admitted while others run simply join the
// next launch: that is continuous batching.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "batch_kernels.cuh"
#include "device_cache.cuh"
#include "pdhg_host.cuh"
#include "sankhya_pdhg_gpu.h"

namespace sih26 {

extern thread_local std::string g_last_error;

#define SIH26_SCUDA(expr, code)                                                          \
  do {                                                                                   \
    const cudaError_t e_ = (expr);                                                       \
    if (e_ != cudaSuccess)                                                               \
      throw Failure{code, std::string(#expr) + ": " + cudaGetErrorString(e_)};           \
  } while (0)

namespace {

using Clock = std::chrono::steady_clock;

// Offsets of one LP's arrays inside its device image (bytes, 256-byte aligned).
struct Layout {
  size_t bytes = 0;
  size_t put(size_t n) {
    const size_t at = bytes;
    bytes += (n + 255) & ~size_t(255);
    return at;
  }
};

struct PartOff {
  size_t blk_seg_begin, segs, blk_long_begin, longs, blk_item_begin, items, seg_sum, sell_idx, sell_val;
};

// The classes of LPs, each with a queue and a launch of its own: a block an LP, a cluster, and a cluster for
// LPs whose entries are gathered out of L2, which leave the shared memory to L1: in one launch with the others
// (212 KB a block, some 16 KB of L1) such an LP took 2 to 2.5 times as long an iteration (1 million nonzeros,
// 100,000 x 250,000, 8 blocks: 497 us, 230 in a launch of its own).
enum { kOneBlock = 0, kCluster = 1, kClusterL2 = 2, kKinds = 3 };

// One submitted LP.
struct Job {
  int64_t ticket = 0;
  int m = 0, n = 0;
  long long nnz = 0;
  // what goes to the device, in its layout: the lists, then the problem as given (the objective, the
  // certificate check and the outputs read it here), then the prepared arrays of an LP the host
  // prepares
  std::vector<unsigned char> up;
  size_t send = 0;  // bytes of it that are sent
  size_t bytes = 0, legacy_bytes = 0;  // of the device region; without slices and scratch
  sankhya_pdhg_problem view{};
  sankhya_pdhg_params prm{};
  std::vector<int> row_perm, col_perm;
  bool device_prep = false;
  ResidentPlan plan{};
  struct {
    size_t cs, ri, val, cost, cl, cu, rl, ru;  // the problem as given
    size_t a_ptr, a_idx, a_val, at_ptr, at_idx, at_val, rptr, row_perm, col_perm, start, x_start;
    PartOff pa, pat;
    size_t c, scl, scu, srl, sru, dr, dc, c0, cl0, cu0, rl0, ru0;
    size_t row_pos, col_pos, next, ecol, ev, rp, cp;
    size_t zero, zeros;
    size_t x0, x1, y0, y1, ax0, ax1, xsum, ysum, xr, yr, best_x, best_y;
    size_t xt, yt, axr;  // the Halpern operator's T(z) and A x_0
    size_t xc, yc;       // both candidates of an evaluation; then the report's x, reduced costs and y
    size_t farkas_out, ray_out;
  } off{};
  Ctrl ctrl0{};
  // lifecycle
  int group = 1;  // blocks working on this LP: 1, or kClusterSize
  int kind() const { return group == 1 ? kOneBlock : plan.outside == kFromL2 ? kClusterL2 : kCluster; }
  int slot = -1;
  unsigned char* base = nullptr;  // its device region: in the pool at pool_offset, or
  size_t pool_offset = 0;
  Chunk own_chunk;                // a chunk of its own
  bool finished = false;
  bool model_error = false;
  std::string message;
  double submit_time = 0.0, admit_time = 0.0, finish_time = 0.0;
  // solved alone on the whole GPU by the single-LP engine; its result as that engine filled it
  bool solo = false;
  sankhya_pdhg_result solo_result{};
  // result
  int status = SANKHYA_PDHG_NOT_SOLVED;
  Ctrl last{};
  std::vector<double> x, row_dual, col_dual, farkas, ray;
};

template <class T>
void write(std::vector<unsigned char>& img, size_t at, const std::vector<T>& v) {
  if (!v.empty()) std::memcpy(img.data() + at, v.data(), v.size() * sizeof(T));
}
void write(std::vector<unsigned char>& img, size_t at, const void* from, size_t bytes) {
  if (bytes) std::memcpy(img.data() + at, from, bytes);
}

template <class T>
std::vector<T> gathered(const std::vector<T>& v, const std::vector<int>& perm) {
  std::vector<T> out(perm.size());
  for (size_t t = 0; t < perm.size(); ++t) out[t] = v[perm[t]];
  return out;
}
std::vector<double> gathered(const double* v, const std::vector<int>& perm) {
  std::vector<double> out(perm.size());
  for (size_t t = 0; t < perm.size(); ++t) out[t] = v[perm[t]];
  return out;
}

// Host work of one LP: the checks, the lists, and the problem as given; for an LP with a row or column
// of more than kTeamPrepRow entries also its scaling and layout.
void prepare(Job& J, const sankhya_pdhg_problem& p, const sankhya_pdhg_params& prm,
             long long cluster_min_nnz, long long solo_min_nnz) {
  check_structure(p);
  const int m = p.num_rows, n = p.num_cols;
  const size_t um = m, un = n, nnz = p.num_nonzeros;
  J.m = m;
  J.n = n;
  J.nnz = p.num_nonzeros;
  J.prm = prm;
  J.view = p;
  const std::string why = validate_model(p);
  if (!why.empty()) {
    J.model_error = true;
    J.message = why;
    return;
  }
  auto& o = J.off;
  Layout L;
  const bool solo = solo_min_nnz > 0 && J.nnz >= solo_min_nnz;
  PermutedLp q;
  HostPart pa, pat;
  std::vector<int> row_ptr;
  std::vector<double> v0;
  if (!solo) {
    int longest = 0;
    q = outline(p, row_ptr, longest);
    J.device_prep = longest <= kTeamPrepRow;
    J.group = (cluster_min_nnz > 0 && q.nnz >= cluster_min_nnz) ? kClusterSize : 1;
    pa = partition(q.a_ptr, J.group, kWarps, prm.group_size_rows, Schedule{}, true);
    pat = partition(q.at_ptr, J.group, kWarps, prm.group_size_cols, Schedule{}, true);
    J.plan = plan_resident(m, n, q.at_ptr, q.a_ptr, pat, pa, J.group, 8,
                           prm.algorithm == SANKHYA_PDHG_ALGORITHM_HALPERN, true);
    if (J.plan.cs == 0) J.plan = plan_outside(m, n, J.group);
    o.a_ptr = L.put((um + 1) * 4);
    o.at_ptr = L.put((un + 1) * 4);
    o.rptr = L.put((um + 1) * 4);
    o.row_perm = L.put(um * 4);
    o.col_perm = L.put(un * 4);
    o.start = L.put(un * 8);
    const auto lists = [&](const HostPart& hp, PartOff& po) {
      po.blk_seg_begin = L.put(hp.blk_seg_begin.size() * 4);
      po.segs = L.put(hp.segs.size() * 16);
      po.blk_long_begin = L.put(hp.blk_long_begin.size() * 4);
      po.longs = L.put(hp.longs.size() * 16);
      po.blk_item_begin = L.put(hp.blk_item_begin.size() * 4);
      po.items = L.put(hp.items.size() * 16);
    };
    lists(pa, o.pa);
    lists(pat, o.pat);
  }
  // the problem as given; once it is prepared, the slices of A' go over it
  const size_t raw = L.bytes;
  o.ri = L.put(nnz * 4);
  o.val = L.put(nnz * 8);
  o.cs = L.put((un + 1) * 4);
  for (size_t* f : {&o.cost, &o.cl, &o.cu}) *f = L.put(un * 8);
  for (size_t* f : {&o.rl, &o.ru}) *f = L.put(um * 8);
  const size_t raw_end = L.bytes;
  if (!solo) {
    L.bytes = raw;
    o.pat.sell_idx = L.put(pat.sell_entries * 4);
    o.pat.sell_val = L.put(pat.sell_entries * 8);
    L.bytes = std::max(L.bytes, raw_end);
    // scaled and laid out
    o.a_idx = L.put(nnz * 4);
    o.a_val = L.put(nnz * 8);
    o.at_idx = L.put(nnz * 4);
    o.at_val = L.put(nnz * 8);
    for (size_t* f : {&o.c, &o.scl, &o.scu, &o.dc, &o.c0, &o.cl0, &o.cu0, &o.x_start}) *f = L.put(un * 8);
    for (size_t* f : {&o.srl, &o.sru, &o.dr, &o.rl0, &o.ru0}) *f = L.put(um * 8);
  }
  const size_t host_end = solo ? raw_end : (J.device_prep ? raw_end : L.bytes);
  if (!solo) {
    // the row-major copy that the preparation works on, and after it the slices of A
    const size_t at = L.bytes;
    o.ecol = L.put(nnz * 4);
    o.ev = L.put(nnz * 8);
    const size_t end = L.bytes;
    L.bytes = at;
    o.pa.sell_idx = L.put(pa.sell_entries * 4);
    o.pa.sell_val = L.put(pa.sell_entries * 8);
    L.bytes = std::max(L.bytes, end);
    o.row_pos = L.put(um * 4);
    o.col_pos = L.put(un * 4);
    o.next = L.put(um * 4);
    o.rp = L.put(um * 16);
    o.cp = L.put(un * 16);
    o.xc = L.put(un * 16);
    o.yc = L.put(um * 16);
    o.zero = L.bytes;
    for (size_t* f : {&o.x0, &o.x1, &o.xsum, &o.xr, &o.best_x, &o.ray_out, &o.xt}) *f = L.put(un * 8);
    for (size_t* f : {&o.y0, &o.y1, &o.ax0, &o.ax1, &o.ysum, &o.yr, &o.best_y, &o.farkas_out, &o.yt, &o.axr})
      *f = L.put(um * 8);
    o.pa.seg_sum = L.put(pa.segs.size() * 16);
    o.pat.seg_sum = L.put(pat.segs.size() * 16);
    o.zeros = (L.bytes - o.zero) / 8;
    J.bytes = L.bytes;
    J.legacy_bytes = 24 * nnz + 136 * (um + un) + (raw - o.row_perm);
  }
  J.up.resize(host_end);
  auto& up = J.up;
  write(up, o.cs, p.col_starts, (un + 1) * 4);
  write(up, o.ri, p.row_indices, nnz * 4);
  write(up, o.val, p.values, nnz * 8);
  write(up, o.cost, p.cost, un * 8);
  write(up, o.cl, p.col_lower, un * 8);
  write(up, o.cu, p.col_upper, un * 8);
  write(up, o.rl, p.row_lower, um * 8);
  write(up, o.ru, p.row_upper, um * 8);
  const auto I = [&](size_t at) { return reinterpret_cast<const int32_t*>(up.data() + at); };
  const auto D = [&](size_t at) { return reinterpret_cast<const double*>(up.data() + at); };
  J.view = sankhya_pdhg_problem{m, n, p.num_nonzeros, I(o.cs), I(o.ri), D(o.val), D(o.cost), D(o.cl), D(o.cu),
                                D(o.rl), D(o.ru), p.maximize, p.objective_offset};
  if (solo) {
    J.solo = true;  // the single-LP engine prepares it itself
    return;
  }
  J.send = host_end;
  const double sense = p.maximize ? -1.0 : 1.0;
  double cs2 = 0.0, bs2 = 0.0;
  for (int j = 0; j < n; ++j) cs2 += (sense * p.cost[j]) * (sense * p.cost[j]);
  for (int i = 0; i < m; ++i) {
    const double b = host_finite_bound(p.row_lower[i])
                         ? p.row_lower[i]
                         : (host_finite_bound(p.row_upper[i]) ? p.row_upper[i] : 0.0);
    bs2 += b * b;
  }
  write(up, o.a_ptr, q.a_ptr);
  write(up, o.at_ptr, q.at_ptr);
  write(up, o.rptr, row_ptr);
  write(up, o.row_perm, q.row_perm);
  write(up, o.col_perm, q.col_perm);
  const auto part_write = [&](const HostPart& hp, const PartOff& po) {
    write(up, po.blk_seg_begin, hp.blk_seg_begin);
    write(up, po.segs, hp.segs);
    write(up, po.blk_long_begin, hp.blk_long_begin);
    write(up, po.longs, hp.longs);
    write(up, po.blk_item_begin, hp.blk_item_begin);
    write(up, po.items, hp.items);
  };
  part_write(pa, o.pa);
  part_write(pat, o.pat);
  // random start of the norm estimate (seed + 1)
  v0.resize(n);
  uniform_draws(static_cast<uint32_t>(prm.random_seed) + 1u, -1.0, 1.0, n, v0.data());
  write(up, o.start, gathered(v0, q.col_perm));
  if (!J.device_prep) {
    std::vector<double> cmin(n);
    for (int j = 0; j < n; ++j) cmin[j] = sense * p.cost[j];
    const Scaling sc = build_scaling(J.view, cmin, 10);
    const PermutedLp f = permute(J.view, sc.values);
    write(up, o.a_idx, f.a_idx);
    write(up, o.a_val, f.a_val);
    write(up, o.at_idx, f.at_idx);
    write(up, o.at_val, f.at_val);
    write(up, o.c, gathered(sc.cost, q.col_perm));
    write(up, o.scl, gathered(sc.cl, q.col_perm));
    write(up, o.scu, gathered(sc.cu, q.col_perm));
    write(up, o.srl, gathered(sc.rl, q.row_perm));
    write(up, o.sru, gathered(sc.ru, q.row_perm));
    write(up, o.dr, gathered(sc.dr, q.row_perm));
    write(up, o.dc, gathered(sc.dc, q.col_perm));
    write(up, o.c0, gathered(cmin, q.col_perm));
    write(up, o.cl0, gathered(p.col_lower, q.col_perm));
    write(up, o.cu0, gathered(p.col_upper, q.col_perm));
    write(up, o.rl0, gathered(p.row_lower, q.row_perm));
    write(up, o.ru0, gathered(p.row_upper, q.row_perm));
    // start: the projection of zero (pdhg.cpp:329-334), also the restart anchor and best point
    std::vector<double> x0(n);
    for (int t = 0; t < n; ++t) {
      const int j = q.col_perm[t];
      double v = 0.0;
      if (host_finite_bound(sc.cl[j]) && v < sc.cl[j]) v = sc.cl[j];
      else if (host_finite_bound(sc.cu[j]) && v > sc.cu[j]) v = sc.cu[j];
      x0[t] = v;
    }
    write(up, o.x_start, x0);
  }
  J.row_perm = std::move(q.row_perm);
  J.col_perm = std::move(q.col_perm);

  Ctrl& c = J.ctrl0;
  c = Ctrl{};
  c.omega = 1.0;
  c.restart_kkt = INFINITY;
  c.best_worst = INFINITY;
  c.best.primal = c.best.dual = c.best.gap = INFINITY;
  c.state = kSetup;
  c.tolerance = prm.tolerance;
  c.bound_norm = std::sqrt(bs2);
  c.cost_norm = std::sqrt(cs2);
  c.iteration_limit = prm.iteration_limit < 0 ? 1000000ll : prm.iteration_limit;
  c.use_restarts = prm.restart ? 1 : 0;
  c.stop_at_request = prm.stop_at_request ? 1 : 0;
  c.stop_rule = prm.stop_rule;
  c.farkas_cooldown = prm.detect_infeasibility ? 0 : (1 << 30);
  c.halpern = prm.algorithm == SANKHYA_PDHG_ALGORITHM_HALPERN ? 1 : 0;
}

// First-fit allocator over the pool, coalescing on free.
class PoolAllocator {
 public:
  explicit PoolAllocator(size_t bytes) { free_[0] = bytes; }
  bool alloc(size_t bytes, size_t* at) {
    for (auto it = free_.begin(); it != free_.end(); ++it) {
      if (it->second >= bytes) {
        *at = it->first;
        const size_t rest = it->second - bytes, start = it->first + bytes;
        free_.erase(it);
        if (rest) free_[start] = rest;
        used_ += bytes;
        return true;
      }
    }
    return false;
  }
  void release(size_t at, size_t bytes) {
    used_ -= bytes;
    auto it = free_.emplace(at, bytes).first;
    auto next = std::next(it);
    if (next != free_.end() && it->first + it->second == next->first) {
      it->second += next->second;
      free_.erase(next);
    }
    if (it != free_.begin()) {
      auto prev = std::prev(it);
      if (prev->first + prev->second == it->first) {
        prev->second += it->second;
        free_.erase(it);
      }
    }
  }

 private:
  std::map<size_t, size_t> free_;
  size_t used_ = 0;
};

}  // namespace

struct Server {
  sankhya_pdhg_server_config cfg{};
  cudaStream_t stream = nullptr;
  unsigned char* pool = nullptr;
  size_t pool_bytes = 0;  // what the LPs may take
  // the chunks of the memory cache that everything below sits in
  Chunk device_chunk, pinned_chunk, table_chunk;
  std::unique_ptr<PoolAllocator> alloc;
  int own_chunks = 0;     // running LPs with a chunk of their own, beside the pool: at most one
  BatchSlot* d_slots = nullptr;
  NewSlot* d_fresh = nullptr;  // the LPs being admitted
  Ctrl* d_ctrls = nullptr;
  struct Class {
    std::vector<int> active;  // slot indices, largest LP first
    // on the device: active list, count, queue head, and the active LPs' control blocks
    int *d_active = nullptr, *d_count = nullptr, *d_head = nullptr;
    Ctrl* d_compact = nullptr;
    // pinned mirrors
    Ctrl* h_compact = nullptr;
    int *h_active = nullptr, *h_count = nullptr;
  } cls[kKinds];
  size_t running() const {
    size_t n = 0;
    for (const Class& c : cls) n += c.active.size();
    return n;
  }
  cudaGraphExec_t graph = nullptr;
  // the split of the GPU between the classes: clusters for the large LPs, single blocks
  // for the others; chosen per round from the active work, the graph rebuilt when it changes
  int slots_total = 0;     // co-resident blocks of the batch kernels
  int max_clusters = 0;    // co-resident 8-block clusters
  int clusters = 0;        // clusters of the current graph, of both kinds
  int l2_clusters = 0;     // of them, for the LPs gathered out of L2
  int small_grid = 0;      // single blocks of the current graph
  std::vector<int> free_slots;
  std::vector<std::shared_ptr<Job>> slot_job;
  std::deque<std::shared_ptr<Job>> waiting;
  std::deque<std::shared_ptr<Job>> solo_waiting;  // LPs the single-LP engine solves alone
  std::map<int64_t, std::shared_ptr<Job>> jobs;
  int64_t next_ticket = 1;
  std::mutex mu;
  Clock::time_point t0 = Clock::now();
  long long launches = 0;
  unsigned long long device_clock0 = 0;
  double last_round_seconds = 0.0;  // wall time of the last batched launch
  long long rounds = 0;             // batched launches so far
  // attempts per LP per launch (LPs of at most 16,384 nonzeros per block; larger ones get
  // proportionally fewer): the configured value, or the autotuner's (chunk_attempts = -1)
  long long chunk = 0;
  long long graph_chunk = -1;  // the chunk the current graph was built with
  bool auto_chunk = false;
  int chunk_source = 0;        // 0 configured, 1 tuned here, 2 read from the cache
  std::string chunk_family;    // cache key, once enough LPs have been admitted
  std::vector<long long> family_nnz;
  std::vector<double> family_per_row;
  // the chunk search: LPs finished per second over windows of at least kChunkWindow launches
  // and kChunkWindowSeconds, for every chunk tried
  double round_work = 0.0;     // LPs the last launch finished
  double window_work = 0.0, window_time = 0.0;
  int window_rounds = 0;
  std::map<long long, double> chunk_rate;
  long long best_chunk = 0;
  double best_rate = 0.0;
  int direction = 1;           // 1 doubling, -1 halving
  bool chunk_settled = false;

  double now() const { return std::chrono::duration<double>(Clock::now() - t0).count(); }
};

namespace {

__global__ void read_clock(unsigned long long* out) { *out = global_ns(); }

BatchSlot relocate(const Job& J, unsigned char* base, Ctrl* ctrl) {
  const auto& o = J.off;
  const auto D = [&](size_t off) { return reinterpret_cast<double*>(base + off); };
  const auto I = [&](size_t off) { return reinterpret_cast<int*>(base + off); };
  const auto I4 = [&](size_t off) { return reinterpret_cast<int4*>(base + off); };
  BatchSlot b{};
  Prob<double>& P = b.P;
  P.m = J.m;
  P.n = J.n;
  P.A = Csr<double>{I(o.a_ptr), I(o.a_idx), D(o.a_val), D(o.a_val)};
  P.AT = Csr<double>{I(o.at_ptr), I(o.at_idx), D(o.at_val), D(o.at_val)};
  const auto part = [&](const PartOff& po) {
    return Part{I(po.blk_seg_begin), I4(po.segs), I(po.blk_long_begin), I4(po.longs),
                I(po.blk_item_begin), I4(po.items), D(po.seg_sum), I(po.sell_idx), base + po.sell_val};
  };
  P.pai = P.pae = part(o.pa);
  P.pati = P.pate = part(o.pat);
  P.c = P.c64 = D(o.c);
  P.cl = P.cl64 = D(o.scl);
  P.cu = P.cu64 = D(o.scu);
  P.rl = P.rl64 = D(o.srl);
  P.ru = P.ru64 = D(o.sru);
  P.dr = D(o.dr);
  P.dc = D(o.dc);
  P.c0 = D(o.c0);
  P.cl0 = D(o.cl0);
  P.cu0 = D(o.cu0);
  P.rl0 = D(o.rl0);
  P.ru0 = D(o.ru0);
  State<double>& S = b.S;
  S.x[0] = D(o.x0);
  S.x[1] = D(o.x1);
  S.y[0] = D(o.y0);
  S.y[1] = D(o.y1);
  S.ax[0] = D(o.ax0);
  S.ax[1] = D(o.ax1);
  S.xsum = D(o.xsum);
  S.ysum = D(o.ysum);
  S.xr = D(o.xr);
  S.yr = D(o.yr);
  S.xc = reinterpret_cast<double2*>(base + o.xc);
  S.yc = reinterpret_cast<double2*>(base + o.yc);
  S.best_x = D(o.best_x);
  S.best_y = D(o.best_y);
  S.cert_row = D(o.farkas_out);
  S.cert_col = D(o.ray_out);
  S.xt = D(o.xt);
  S.yt = D(o.yt);
  S.axr = D(o.axr);
  S.partials = nullptr;
  S.ctrl = ctrl;
  b.plan = J.plan;
  RawLp& R = b.raw;
  R.v = J.device_prep ? D(o.val) : nullptr;
  R.cs = I(o.cs);
  R.ri = I(o.ri);
  R.cost = D(o.cost);
  R.cl = D(o.cl);
  R.cu = D(o.cu);
  R.rl = D(o.rl);
  R.ru = D(o.ru);
  R.sense = J.view.maximize ? -1.0 : 1.0;
  R.rptr = I(o.rptr);
  R.row_perm = I(o.row_perm);
  R.col_perm = I(o.col_perm);
  R.row_pos = I(o.row_pos);
  R.col_pos = I(o.col_pos);
  R.next = I(o.next);
  R.ecol = I(o.ecol);
  R.ev = D(o.ev);
  R.rp = D(o.rp);
  R.cp = D(o.cp);
  R.x0[0] = S.x[0];
  R.x0[1] = S.xr;
  R.x0[2] = S.best_x;
  b.start = D(o.start);
  b.x_start = D(o.x_start);
  b.zero = D(o.zero);
  b.zeros = o.zeros;
  // the report's outputs go where the evaluations kept their candidates
  b.x_out = D(o.xc);
  b.red_out = D(o.xc) + J.n;
  b.y_out = D(o.yc);
  return b;
}

// Occupancy of the batch kernels: how many blocks, and how many 8-block clusters, fit at once.
void query_capacity(Server& s) {
  int bpsm = 0;
  SIH26_SCUDA(cudaFuncSetAttribute(batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   kResidentBytes), SANKHYA_GPU_INIT_FAILED);
  SIH26_SCUDA(cudaFuncSetAttribute(cluster_batch_kernel<false>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   kResidentBytes), SANKHYA_GPU_INIT_FAILED);
  // asked for: an SM otherwise keeps the split of the launch before (a round of such LPs 14.2 ms, 13.0 with it)
  SIH26_SCUDA(cudaFuncSetAttribute(cluster_batch_kernel<true>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                   (int)cudaSharedmemCarveoutMaxL1), SANKHYA_GPU_INIT_FAILED);
  SIH26_SCUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bpsm, batch_kernel, kThreads,
                                                            kResidentBytes),
              SANKHYA_GPU_INIT_FAILED);
  int sms = 0;
  SIH26_SCUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s.cfg.device),
              SANKHYA_GPU_INIT_FAILED);
  s.slots_total = sms * std::max(1, bpsm);
  cudaLaunchConfig_t lc{};
  lc.gridDim = dim3(kClusterSize);
  lc.blockDim = dim3(kThreads);
  lc.dynamicSmemBytes = kResidentBytes;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = kClusterSize;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  lc.attrs = &attr;
  lc.numAttrs = 1;
  int max_clusters = 0;
  SIH26_SCUDA(cudaOccupancyMaxActiveClusters(&max_clusters, cluster_batch_kernel<false>, &lc),
              SANKHYA_GPU_INIT_FAILED);
  // keep at least one cluster's worth of blocks for the single-block class
  s.max_clusters = std::max(1, std::min(max_clusters, (s.slots_total - kClusterSize) / kClusterSize));
}

// The round's graph for `clusters` 8-block clusters, as many again as `l2` for the LPs gathered out of L2, and
// the remaining blocks as single blocks: the persistent kernels side by side on forked streams, then the control
// blocks of each class compacted for the host. A class of clusters without any has no launch.
void build_graph(Server& s, int clusters, int l2) {
  const int small_grid = std::max(1, s.slots_total - (clusters + l2) * kClusterSize);
  if (s.graph && clusters == s.clusters - s.l2_clusters && l2 == s.l2_clusters && small_grid == s.small_grid &&
      s.chunk == s.graph_chunk)
    return;
  if (s.graph) {
    cudaGraphExecDestroy(s.graph);
    s.graph = nullptr;
  }
  cudaStream_t cap, side[kKinds];  // side[0] unused
  cudaEvent_t fork, join[kKinds];
  SIH26_SCUDA(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking), SANKHYA_GPU_INIT_FAILED);
  SIH26_SCUDA(cudaEventCreateWithFlags(&fork, cudaEventDisableTiming), SANKHYA_GPU_INIT_FAILED);
  for (int k = kCluster; k < kKinds; ++k) {
    SIH26_SCUDA(cudaStreamCreateWithFlags(&side[k], cudaStreamNonBlocking), SANKHYA_GPU_INIT_FAILED);
    SIH26_SCUDA(cudaEventCreateWithFlags(&join[k], cudaEventDisableTiming), SANKHYA_GPU_INIT_FAILED);
  }
  const long long chunk = s.chunk;
  cudaGraph_t g;
  SIH26_SCUDA(cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal), SANKHYA_GPU_INIT_FAILED);
  for (const Server::Class& c : s.cls) cudaMemsetAsync(c.d_head, 0, sizeof(int), cap);
  cudaEventRecord(fork, cap);
  const int grids[kKinds] = {small_grid, clusters * kClusterSize, l2 * kClusterSize};
  for (int k = kCluster; k < kKinds; ++k) {
    if (grids[k] == 0) continue;
    const Server::Class& c = s.cls[k];
    cudaStreamWaitEvent(side[k], fork, 0);
    if (k == kCluster)
      cluster_batch_kernel<false><<<grids[k], kThreads, kResidentBytes, side[k]>>>(s.d_slots, c.d_active, c.d_count,
                                                                                  c.d_head, chunk);
    else
      cluster_batch_kernel<true><<<grids[k], kThreads, 0, side[k]>>>(s.d_slots, c.d_active, c.d_count, c.d_head, chunk);
    gather_ctrl_kernel<<<64, 128, 0, side[k]>>>(s.d_ctrls, c.d_active, c.d_count, c.d_compact);
    cudaEventRecord(join[k], side[k]);
  }
  const Server::Class& one = s.cls[kOneBlock];
  batch_kernel<<<grids[0], kThreads, kResidentBytes, cap>>>(s.d_slots, one.d_active, one.d_count, one.d_head, chunk);
  gather_ctrl_kernel<<<128, 128, 0, cap>>>(s.d_ctrls, one.d_active, one.d_count, one.d_compact);
  for (int k = kCluster; k < kKinds; ++k)
    if (grids[k] > 0) cudaStreamWaitEvent(cap, join[k], 0);
  SIH26_SCUDA(cudaStreamEndCapture(cap, &g), SANKHYA_GPU_INIT_FAILED);
  SIH26_SCUDA(cudaGraphInstantiate(&s.graph, g, 0), SANKHYA_GPU_INIT_FAILED);
  cudaGraphDestroy(g);
  cudaEventDestroy(fork);
  for (int k = kCluster; k < kKinds; ++k) {
    cudaEventDestroy(join[k]);
    cudaStreamDestroy(side[k]);
  }
  cudaStreamDestroy(cap);
  s.l2_clusters = l2;
  s.clusters = clusters + l2;
  s.small_grid = small_grid;
  s.graph_chunk = chunk;
}

// The chunk autotuner (chunk_attempts = -1). Chunking only decides where an LP pauses between
// launches, never what it computes, so the chunk is free to follow measurement. A launch has
// a fixed cost (control blocks, the LPs' start-up, the host round trip) besides its attempts,
// so longer chunks cost less per attempt; but an LP that finishes early in a launch leaves its
// slot idle until the launch ends, so longer chunks also refill the slots of the small LPs
// later. The search measures the served stream's own figure of merit, LPs finished per
// second, over windows of at least kChunkWindow launches and kChunkWindowSeconds, starting at
// kChunkStart and moving by factors of two from the best chunk so far while a step gains more
// than 3 %; when neither neighbour of the best is untried, the best is kept and stored in the
// autotune cache under the family of the first kChunkFamilySample admitted LPs. A chunk cached
// for the family is used as it is.
constexpr long long kChunkMin = 16, kChunkMax = 8192, kChunkStart = 512;
constexpr int kChunkFamilySample = 32, kChunkWindow = 8;
constexpr double kChunkWindowSeconds = 1.0;

void note_family(Server& s, const Job& J) {
  if (!s.auto_chunk || !s.chunk_family.empty()) return;
  s.family_nnz.push_back(J.nnz);
  s.family_per_row.push_back(J.m > 0 ? static_cast<double>(J.nnz) / J.m : 0.0);
  if (static_cast<int>(s.family_nnz.size()) < kChunkFamilySample) return;
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s.cfg.device);
  s.chunk_family = chunk_key(sms, s.slots_total, s.family_nnz, s.family_per_row);
  long long cached = 0;
  if (chunk_lookup(autotune_cache_path(), s.chunk_family, &cached)) {
    s.chunk = std::max(kChunkMin, std::min(kChunkMax, cached));
    s.chunk_source = 2;
    s.chunk_settled = true;
  }
}

void tune_chunk(Server& s) {
  if (!s.auto_chunk || s.chunk_settled || s.last_round_seconds <= 0.0) return;
  s.window_work += s.round_work;
  s.window_time += s.last_round_seconds;
  if (++s.window_rounds < kChunkWindow || s.window_time < kChunkWindowSeconds) return;
  const double rate = s.window_work / s.window_time;
  s.window_work = s.window_time = 0.0;
  s.window_rounds = 0;
  s.chunk_rate[s.chunk] = rate;
  if (s.best_chunk == 0 || rate > 1.03 * s.best_rate) {
    s.best_chunk = s.chunk;
    s.best_rate = rate;
  }
  for (int turn = 0; turn < 2; ++turn) {
    const long long next = s.direction > 0 ? s.best_chunk * 2 : s.best_chunk / 2;
    if (next >= kChunkMin && next <= kChunkMax && !s.chunk_rate.count(next)) {
      s.chunk = next;
      return;
    }
    s.direction = -s.direction;
  }
  s.chunk = s.best_chunk;
  s.chunk_settled = true;
  if (!s.chunk_family.empty())
    chunk_store(autotune_cache_path(), s.chunk_family, s.chunk, s.best_rate);  // LPs/s
}

// Clusters for this round: the large class's share of the active nonzeros (its work per
// attempt) of the GPU's blocks, no more than it has LPs, and the configured number when the
// split is fixed (config.clusters > 0 and no adaptation).
int clusters_for_round(const Server& s, long long small_nnz, long long big_nnz, int big_count) {
  if (s.cfg.clusters > 0) return s.cfg.clusters;
  if (big_count == 0) return 1;
  const double share = static_cast<double>(big_nnz) / static_cast<double>(std::max(1ll, small_nnz + big_nnz));
  int want = static_cast<int>(std::lround(share * s.slots_total / kClusterSize));
  want = std::min(want, big_count);
  if (small_nnz > 0) want = std::min(want, s.max_clusters);
  return std::max(1, want);
}

// Of them, those for the LPs gathered out of L2: the split with the shortest round. An LP's share of a round goes
// with its nonzeros up to the chunk's budget (run_slot), which all larger ones take in full; a class lasts as
// long as its LPs take side by side, and as its largest take in turns. (Split by nonzeros alone, a queue of the
// served family left the smaller clusters' LPs a third of the clusters that they needed.)
int l2_clusters_for_round(const Server& s, int clusters) {
  const double budget = s.chunk > 0 ? static_cast<double>(kChunkNnz) * kClusterSize : INFINITY;
  double total[kKinds] = {0, 0, 0}, top[kKinds] = {0, 0, 0};
  int count_top[kKinds] = {0, 0, 0};
  for (int k = kCluster; k < kKinds; ++k)
    for (int slot : s.cls[k].active) {
      const double w = std::min(budget, static_cast<double>(s.slot_job[slot]->nnz));
      total[k] += w;
      if (w > top[k]) count_top[k] = 0;
      top[k] = std::max(top[k], w);
      count_top[k] += w == top[k];
    }
  if (s.cls[kClusterL2].active.empty()) return 0;
  if (s.cls[kCluster].active.empty()) return clusters;
  const auto lasts = [&](int k, int c) { return std::max(total[k] / c, top[k] * ((count_top[k] + c - 1) / c)); };
  int best = 1;
  double best_time = INFINITY;
  for (int l2 = 1; l2 < clusters; ++l2) {
    const double time = std::max(lasts(kClusterL2, l2), lasts(kCluster, clusters - l2));
    // of equal ones the present split, which needs no new graph
    if (time < best_time || (time == best_time && l2 == s.l2_clusters)) {
      best = l2;
      best_time = time;
    }
  }
  return best;
}

// Bytes of the report's outputs, from off.xc on.
size_t output_bytes(const Job& J) { return J.off.yc - J.off.xc + static_cast<size_t>(J.m) * 8; }

// The answer of an LP whose outputs have come back to `out`.
void finish_job(Server& s, Job& J, const Ctrl& c, const unsigned char* out) {
  const int m = J.m, n = J.n;
  const double sense = J.view.maximize ? -1.0 : 1.0;
  const double* hx = reinterpret_cast<const double*>(out);
  const double* hred = hx + n;
  const double* hy = reinterpret_cast<const double*>(out + (J.off.yc - J.off.xc));
  J.x.assign(n, 0.0);
  J.col_dual.assign(n, 0.0);
  J.row_dual.assign(m, 0.0);
  for (int t = 0; t < n; ++t) {
    J.x[J.col_perm[t]] = hx[t];
    J.col_dual[J.col_perm[t]] = sense * hred[t];
  }
  for (int t = 0; t < m; ++t) J.row_dual[J.row_perm[t]] = sense * (-hy[t]);
  J.last = c;
  const Residuals& f = c.best;
  const bool standard = f.absolute_primal <= 1e-7 && f.absolute_dual <= 1e-7 &&
                        f.gap_as_verified <= 1e-9 && f.complementarity <= 1e-6;
  if (c.state == kInfeasible) {
    J.status = SANKHYA_PDHG_INFEASIBLE;
  } else if (c.state == kUnbounded) {
    // a ray is certified; unboundedness also claims a feasible point for it to start from,
    // which the batched engine does not search for: claimed only when the reported point is
    // feasible to the project's standard (its largest bound violation, measured on the device)
    J.status = c.primal_violation <= 1e-7 ? SANKHYA_PDHG_UNBOUNDED
                                          : SANKHYA_PDHG_INFEASIBLE_OR_UNBOUNDED;
  } else if (c.converged) {
    J.status = standard ? SANKHYA_PDHG_OPTIMAL : SANKHYA_PDHG_FEASIBLE;
  } else {
    J.status = c.state == kTimeLimit ? SANKHYA_PDHG_TIME_LIMIT : SANKHYA_PDHG_ITERATION_LIMIT;
  }
  char msg[256];
  if (J.status == SANKHYA_PDHG_INFEASIBLE) {
    std::snprintf(msg, sizeof msg,
                  "primal infeasible: Farkas certificate from the dual movement after %lld "
                  "iterations (normalised margin %.3e), checked on the original model",
                  c.iteration, c.farkas_margin);
  } else if (J.status == SANKHYA_PDHG_UNBOUNDED) {
    std::snprintf(msg, sizeof msg,
                  "unbounded: primal ray from the last step after %lld iterations, checked on "
                  "the original model",
                  c.iteration);
  } else if (J.status == SANKHYA_PDHG_INFEASIBLE_OR_UNBOUNDED) {
    std::snprintf(msg, sizeof msg,
                  "primal ray from the last step after %lld iterations, checked on the original "
                  "model; the point is not feasible (largest violation %.3e), so unboundedness "
                  "is not claimed",
                  c.iteration, c.primal_violation);
  } else {
    std::snprintf(msg, sizeof msg,
                  "%lld iterations and %lld restarts; relative primal %.3e, dual %.3e, gap %.3e",
                  c.iteration, c.restarts, f.primal, f.dual, f.gap);
  }
  J.message = msg;
  J.finished = true;
  J.finish_time = s.now();
}

}  // namespace

// ---- server operations (called under the server mutex) -----------------------------------

// LPs routed to the single-LP engine, oldest first, each on the whole GPU with its own params,
// between two batched launches (in stream order with the batched work, so the two never share
// the GPU at once): at least one per step and then as many as fit in the time the last batched
// launch took, so either class gets about half of the GPU while both have work; with no
// batched work, up to 16 per step.
static void solve_one_solo(Server& s);

static void run_solo(Server& s) {
  const bool batch_idle = s.running() == 0 && s.waiting.empty();
  const double budget = batch_idle ? 1e30 : s.last_round_seconds;
  const double start = s.now();
  for (int k = 0; k < 16 && !s.solo_waiting.empty(); ++k) {
    if (k > 0 && s.now() - start >= budget) break;
    solve_one_solo(s);
  }
}

static void solve_one_solo(Server& s) {
  std::shared_ptr<Job> J = s.solo_waiting.front();
  s.solo_waiting.pop_front();
  SIH26_SCUDA(cudaStreamSynchronize(s.stream), SANKHYA_GPU_SYNC_FAILED);
  J->admit_time = s.now();
  J->x.assign(J->n, 0.0);
  J->col_dual.assign(J->n, 0.0);
  J->row_dual.assign(J->m, 0.0);
  J->farkas.assign(J->m, 0.0);
  J->ray.assign(J->n, 0.0);
  sankhya_pdhg_result& r = J->solo_result;
  r = sankhya_pdhg_result{};
  r.col_value = J->x.data();
  r.row_dual = J->row_dual.data();
  r.col_dual = J->col_dual.data();
  r.farkas_dual = J->farkas.data();
  r.primal_ray = J->ray.data();
  sankhya_pdhg_params prm = J->prm;
  prm.device = s.cfg.device;
  const int rc = sankhya_pdhg_gpu_solve(&J->view, &prm, &r);
  if (rc != SANKHYA_GPU_SUCCESS) {
    r.status = SANKHYA_PDHG_NUMERICAL_ERROR;
    std::snprintf(r.message, sizeof r.message, "single-LP engine failed: %s",
                  sankhya_pdhg_gpu_last_error());
  }
  if (r.status != SANKHYA_PDHG_INFEASIBLE) J->farkas.clear();
  if (r.status != SANKHYA_PDHG_UNBOUNDED && r.status != SANKHYA_PDHG_INFEASIBLE_OR_UNBOUNDED)
    J->ray.clear();
  J->status = r.status;
  J->message = r.message;
  J->finished = true;
  J->finish_time = s.now();
  s.launches += r.kernel_launches;
}

static void release(Server& s, Job& J) {
  if (J.own_chunk) {
    MemoryCache::get().give_device(J.own_chunk);
    J.own_chunk = Chunk{};
    --s.own_chunks;
  } else if (J.base) {
    s.alloc->release(J.pool_offset, J.bytes);
  }
  J.base = nullptr;
}

// Admits the waiting LPs that fit, oldest first: a copy each, and per class one launch that places and
// prepares them all. Everything is ordered on the server's stream.
static void admit(Server& s) {
  std::vector<NewSlot> fresh[2];
  while (!s.waiting.empty() && !s.free_slots.empty()) {
    std::shared_ptr<Job> J = s.waiting.front();
    size_t at = 0;
    if (J->bytes > s.pool_bytes) {
      // larger than the whole pool by its slices and scratch only: a chunk of its own, one such LP at a time
      if (s.own_chunks > 0) break;
      J->own_chunk = MemoryCache::get().take_device(s.cfg.device, J->bytes);
      J->base = static_cast<unsigned char*>(J->own_chunk.p);
      if (J->base) {
        ++s.own_chunks;
      } else {
        if (s.running() > 0) break;  // what runs may give memory back
        s.waiting.pop_front();
        J->status = SANKHYA_PDHG_NUMERICAL_ERROR;
        J->message = "the LP does not fit the device's memory";
        J->finished = true;
        J->finish_time = s.now();
        continue;
      }
    } else {
      if (!s.alloc->alloc(J->bytes, &at)) break;  // no room: wait for retirements
      J->pool_offset = at;
      J->base = s.pool + at;
    }
    s.waiting.pop_front();
    const int slot = s.free_slots.back();
    s.free_slots.pop_back();
    J->slot = slot;
    J->admit_time = s.now();
    SIH26_SCUDA(cudaMemcpyAsync(J->base, J->up.data(), J->send, cudaMemcpyHostToDevice, s.stream),
                SANKHYA_GPU_COPY_FAILED);
    NewSlot f{};
    f.ctrl = J->ctrl0;
    if (std::isfinite(J->prm.time_limit) && J->prm.time_limit > 0.0) {
      const double since = s.now();
      f.ctrl.deadline_ns = s.device_clock0 +
                           static_cast<unsigned long long>((since + J->prm.time_limit) * 1e9);
    }
    f.slot = relocate(*J, J->base, s.d_ctrls + slot);
    f.index = slot;
    fresh[J->group > 1].push_back(f);
    s.slot_job[slot] = J;
    s.cls[J->kind()].active.push_back(slot);
    note_family(s, *J);
  }
  if (fresh[0].empty() && fresh[1].empty()) return;
  NewSlot* to = s.d_fresh;
  for (int k = 0; k < 2; ++k) {
    const int count = static_cast<int>(fresh[k].size());
    if (count == 0) continue;
    SIH26_SCUDA(cudaMemcpyAsync(to, fresh[k].data(), count * sizeof(NewSlot), cudaMemcpyHostToDevice, s.stream),
                SANKHYA_GPU_COPY_FAILED);
    const int group = k ? kClusterSize : 1;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = group;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t lc{};
    lc.gridDim = dim3(count * group);
    lc.blockDim = dim3(kThreads);
    lc.stream = s.stream;
    lc.attrs = &attr;
    lc.numAttrs = 1;
    SIH26_SCUDA(cudaLaunchKernelEx(&lc, batch_setup_kernel, static_cast<const NewSlot*>(to), group, s.d_slots,
                                   s.d_ctrls), SANKHYA_GPU_KERNEL_LAUNCH_FAILED);
    ++s.launches;
    to += count;
  }
  // the copies above read `fresh`: staged by the runtime, as pageable memory is, before they return
  const auto larger = [&](int a, int b) { return s.slot_job[a]->nnz > s.slot_job[b]->nnz; };
  for (Server::Class& c : s.cls) std::stable_sort(c.active.begin(), c.active.end(), larger);
}

// Handles the LPs of one class whose control blocks came back in `compact`; returns those
// still running.
static std::vector<int> settle(Server& s, const std::vector<int>& list, const Ctrl* compact) {
  std::vector<int> still, done;
  std::vector<size_t> at;  // where each finished LP's outputs land
  size_t landing_bytes = 0;
  for (size_t q = 0; q < list.size(); ++q) {
    const int slot = list[q];
    const Ctrl& c = compact[q];
    Job& J = *s.slot_job[slot];
    if (c.state == kDeviceError) throw Failure{SANKHYA_GPU_DEVICE_TIMEOUT, "batch kernel error"};
    bool over = c.state == kConverged || c.state == kIterationLimit || c.state == kTimeLimit;
    if (c.state == kInfeasible || c.state == kUnbounded) {
      const bool rows = c.state == kInfeasible;
      const int len = rows ? J.m : J.n;
      std::vector<double> h(len), v(len);
      if (len)
        SIH26_SCUDA(cudaMemcpy(h.data(), J.base + (rows ? J.off.farkas_out : J.off.ray_out),
                               len * 8, cudaMemcpyDeviceToHost), SANKHYA_GPU_COPY_FAILED);
      const std::vector<int>& perm = rows ? J.row_perm : J.col_perm;
      for (int t = 0; t < len; ++t) v[perm[t]] = h[t];
      bool ok = rows ? farkas_holds(J.view, v) : ray_holds(J.view, v);
      if (!ok && !rows && repair_ray(J.view, v)) ok = ray_holds(J.view, v);
      if (ok) {
        (rows ? J.farkas : J.ray) = v;
        over = true;
      } else {
        // not a proof after all: carry on, and give the test a rest
        Ctrl r = c;
        r.state = kRunning;
        r.farkas_cooldown = kCertCooldown;
        SIH26_SCUDA(cudaMemcpyAsync(s.d_ctrls + slot, &r, sizeof(Ctrl), cudaMemcpyHostToDevice,
                                    s.stream), SANKHYA_GPU_COPY_FAILED);
        SIH26_SCUDA(cudaStreamSynchronize(s.stream), SANKHYA_GPU_SYNC_FAILED);
      }
    }
    if (!over) {
      still.push_back(slot);
      continue;
    }
    done.push_back(static_cast<int>(q));
    at.push_back(landing_bytes);
    landing_bytes += (output_bytes(J) + 255) & ~size_t(255);
  }
  if (done.empty()) return still;
  // all the answers, then one wait
  PinnedBuffer landing(landing_bytes);
  std::vector<unsigned char> pageable;
  unsigned char* out = landing.data();
  if (!out) {
    pageable.resize(landing_bytes);
    out = pageable.data();
  }
  for (size_t k = 0; k < done.size(); ++k) {
    const Job& J = *s.slot_job[list[done[k]]];
    if (output_bytes(J))
      SIH26_SCUDA(cudaMemcpyAsync(out + at[k], J.base + J.off.xc, output_bytes(J), cudaMemcpyDeviceToHost,
                                  s.stream), SANKHYA_GPU_COPY_FAILED);
  }
  SIH26_SCUDA(cudaStreamSynchronize(s.stream), SANKHYA_GPU_SYNC_FAILED);
  for (size_t k = 0; k < done.size(); ++k) {
    const int slot = list[done[k]];
    Job& J = *s.slot_job[slot];
    s.round_work += 1.0;
    finish_job(s, J, compact[done[k]], out + at[k]);
    release(s, J);
    s.slot_job[slot].reset();
    s.free_slots.push_back(slot);
  }
  return still;
}

static void run_round(Server& s) {
  if (s.running() == 0) return;
  long long nnz[kKinds] = {0, 0, 0};
  for (int k = 0; k < kKinds; ++k)
    for (int slot : s.cls[k].active) nnz[k] += s.slot_job[slot]->nnz;
  const long long big_nnz = nnz[kCluster] + nnz[kClusterL2];
  int want = clusters_for_round(s, nnz[kOneBlock], big_nnz, static_cast<int>(s.running() - s.cls[kOneBlock].active.size()));
  // hysteresis, as above
  if (s.graph && std::abs(want - s.clusters) <= std::max(1, s.clusters / 4)) want = s.clusters;
  want = std::max(1, std::min(want, s.max_clusters));
  const int l2 = l2_clusters_for_round(s, want);
  // a class with LPs always gets a cluster (one that does not fit beside the others waits for them)
  build_graph(s, std::max(want - l2, s.cls[kCluster].active.empty() ? 0 : 1), l2);
  for (Server::Class& c : s.cls) {
    const size_t count = c.active.size();
    *c.h_count = static_cast<int>(count);
    SIH26_SCUDA(cudaMemcpyAsync(c.d_count, c.h_count, sizeof(int), cudaMemcpyHostToDevice, s.stream),
                SANKHYA_GPU_COPY_FAILED);
    if (count == 0) continue;
    std::memcpy(c.h_active, c.active.data(), count * sizeof(int));
    SIH26_SCUDA(cudaMemcpyAsync(c.d_active, c.h_active, count * sizeof(int), cudaMemcpyHostToDevice, s.stream),
                SANKHYA_GPU_COPY_FAILED);
  }
  const double started = s.now();
  SIH26_SCUDA(cudaGraphLaunch(s.graph, s.stream), SANKHYA_GPU_KERNEL_LAUNCH_FAILED);
  ++s.launches;
  ++s.rounds;
  for (Server::Class& c : s.cls)
    if (!c.active.empty())
      SIH26_SCUDA(cudaMemcpyAsync(c.h_compact, c.d_compact, c.active.size() * sizeof(Ctrl), cudaMemcpyDeviceToHost,
                                  s.stream), SANKHYA_GPU_COPY_FAILED);
  SIH26_SCUDA(cudaStreamSynchronize(s.stream), SANKHYA_GPU_SYNC_FAILED);
  s.last_round_seconds = s.now() - started;
  s.round_work = 0.0;
  for (Server::Class& c : s.cls) c.active = settle(s, c.active, c.h_compact);
  tune_chunk(s);
}

}  // namespace sih26

// ---- C ABI ----------------------------------------------------------------------------------

using sih26::Failure;
using sih26::Server;

extern "C" {

void sankhya_pdhg_server_default_config(sankhya_pdhg_server_config* c) {
  std::memset(c, 0, sizeof *c);
  c->device = 0;
  c->memory_fraction = 0.8;
  c->pool_bytes = 0;
  c->max_active = 4096;
  c->chunk_attempts = -1;  // the autotuner's (measured against fixed lengths on the served family)
  c->cluster_min_nnz = 16384;
  c->clusters = 0;  // adaptive: the large class's share of the active nonzeros
  c->solo_min_nnz = 0;  // never: routing gains nothing on the served family
}

int sankhya_pdhg_server_create(const sankhya_pdhg_server_config* config,
                               sankhya_pdhg_server** out) {
  if (!out) {
    sih26::g_last_error = "out must not be NULL";
    return SANKHYA_GPU_INVALID_ARGUMENT;
  }
  *out = nullptr;
  auto s = std::make_unique<Server>();
  if (config) s->cfg = *config; else sankhya_pdhg_server_default_config(&s->cfg);
  s->auto_chunk = s->cfg.chunk_attempts < 0;
  s->chunk = s->auto_chunk ? sih26::kChunkStart
                           : (s->cfg.chunk_attempts > 0 ? s->cfg.chunk_attempts : (1ll << 40));
  s->chunk_source = s->auto_chunk ? 1 : 0;
  sih26::DeviceGuard guard;
  try {
    int devices = 0;
    if (cudaGetDeviceCount(&devices) != cudaSuccess || devices == 0)
      throw Failure{SANKHYA_GPU_NO_COMPATIBLE_DEVICE, "no CUDA device is visible"};
    SIH26_SCUDA(cudaSetDevice(s->cfg.device), SANKHYA_GPU_INIT_FAILED);
    SIH26_SCUDA(cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking), SANKHYA_GPU_INIT_FAILED);
    size_t free_b = 0, total_b = 0;
    SIH26_SCUDA(cudaMemGetInfo(&free_b, &total_b), SANKHYA_GPU_INIT_FAILED);
    sih26::MemoryCache& cache = sih26::MemoryCache::get();
    free_b += cache.kept(s->cfg.device);  // given back when an allocation needs it
    const int cap = s->cfg.max_active > 0 ? s->cfg.max_active : 4096;
    const size_t share =
        static_cast<size_t>(free_b * std::min(0.95, std::max(0.01, s->cfg.memory_fraction)));
    s->pool_bytes = s->cfg.pool_bytes > 0 ? std::min(static_cast<size_t>(s->cfg.pool_bytes), share)
                                          : share;
    s->pool_bytes &= ~size_t(255);
    // one chunk each for the LPs, the device tables and the pinned mirrors
    const auto chunk = [&](size_t bytes) {
      const sih26::Chunk c = cache.take_device(s->cfg.device, std::max<size_t>(bytes, 256));
      if (!c) throw Failure{SANKHYA_GPU_OUT_OF_MEMORY, "cudaMalloc: out of memory"};
      return c;
    };
    s->device_chunk = chunk(s->pool_bytes);
    s->pool = static_cast<unsigned char*>(s->device_chunk.p);
    s->alloc = std::make_unique<sih26::PoolAllocator>(s->pool_bytes);
    const size_t slots_b = (cap * sizeof(sih26::BatchSlot) + 255) & ~size_t(255);
    const size_t ctrls_b = (cap * sizeof(sih26::Ctrl) + 255) & ~size_t(255);
    const size_t list_b = (cap * sizeof(int) + 255) & ~size_t(255);
    const size_t fresh_b = (cap * sizeof(sih26::NewSlot) + 255) & ~size_t(255);
    s->table_chunk = chunk(slots_b + fresh_b + (1 + sih26::kKinds) * ctrls_b + sih26::kKinds * (list_b + 512) + 256);
    unsigned char* at = static_cast<unsigned char*>(s->table_chunk.p);
    const auto carve = [&](size_t bytes) {
      unsigned char* p = at;
      at += bytes;
      return p;
    };
    s->d_slots = reinterpret_cast<sih26::BatchSlot*>(carve(slots_b));
    s->d_fresh = reinterpret_cast<sih26::NewSlot*>(carve(fresh_b));
    s->d_ctrls = reinterpret_cast<sih26::Ctrl*>(carve(ctrls_b));
    for (Server::Class& c : s->cls) {
      c.d_compact = reinterpret_cast<sih26::Ctrl*>(carve(ctrls_b));
      c.d_active = reinterpret_cast<int*>(carve(list_b));
      c.d_count = reinterpret_cast<int*>(carve(256));
      c.d_head = reinterpret_cast<int*>(carve(256));
      SIH26_SCUDA(cudaMemsetAsync(c.d_count, 0, sizeof(int), s->stream), SANKHYA_GPU_INIT_FAILED);
    }
    unsigned long long* d_clock = reinterpret_cast<unsigned long long*>(carve(256));
    s->pinned_chunk = cache.take_pinned(sih26::kKinds * (ctrls_b + list_b + 256));
    if (!s->pinned_chunk) throw Failure{SANKHYA_GPU_OUT_OF_MEMORY, "cudaMallocHost: out of memory"};
    at = static_cast<unsigned char*>(s->pinned_chunk.p);
    for (Server::Class& c : s->cls) {
      c.h_compact = reinterpret_cast<sih26::Ctrl*>(carve(ctrls_b));
      c.h_active = reinterpret_cast<int*>(carve(list_b));
      c.h_count = reinterpret_cast<int*>(carve(256));
    }
    s->slot_job.resize(cap);
    for (int k = cap - 1; k >= 0; --k) s->free_slots.push_back(k);
    sih26::query_capacity(*s);
    sih26::build_graph(*s, std::min(s->cfg.clusters > 0 ? s->cfg.clusters : 16, s->max_clusters), 0);
    sih26::read_clock<<<1, 1, 0, s->stream>>>(d_clock);
    SIH26_SCUDA(cudaMemcpyAsync(&s->device_clock0, d_clock, sizeof *d_clock,
                                cudaMemcpyDeviceToHost, s->stream), SANKHYA_GPU_COPY_FAILED);
    SIH26_SCUDA(cudaStreamSynchronize(s->stream), SANKHYA_GPU_SYNC_FAILED);
    s->t0 = sih26::Clock::now();
  } catch (const Failure& f) {
    sih26::g_last_error = f.message;
    sankhya_pdhg_server_free(reinterpret_cast<sankhya_pdhg_server*>(s.release()));
    return f.code;
  }
  *out = reinterpret_cast<sankhya_pdhg_server*>(s.release());
  return SANKHYA_GPU_SUCCESS;
}

void sankhya_pdhg_server_free(sankhya_pdhg_server* server) {
  Server* s = reinterpret_cast<Server*>(server);
  if (!s) return;
  sih26::DeviceGuard guard;
  cudaSetDevice(s->cfg.device);
  const bool idle = !s->stream || cudaStreamSynchronize(s->stream) == cudaSuccess;
  if (s->graph) cudaGraphExecDestroy(s->graph);
  sih26::MemoryCache& cache = sih26::MemoryCache::get();
  const auto back = [&](const sih26::Chunk& c) {
    if (idle) cache.give_device(c);
    else if (c) cudaFree(c.p);
  };
  back(s->device_chunk);
  back(s->table_chunk);
  if (idle) cache.give_pinned(s->pinned_chunk);
  else if (s->pinned_chunk) cudaFreeHost(s->pinned_chunk.p);
  for (auto& J : s->slot_job)
    if (J) back(J->own_chunk);
  if (s->stream) cudaStreamDestroy(s->stream);
  delete s;
}

int sankhya_pdhg_server_submit(sankhya_pdhg_server* server, const sankhya_pdhg_problem* problem,
                               const sankhya_pdhg_params* params, int64_t* ticket) {
  Server* s = reinterpret_cast<Server*>(server);
  if (!s || !problem || !ticket) {
    sih26::g_last_error = "server, problem and ticket must not be NULL";
    return SANKHYA_GPU_INVALID_ARGUMENT;
  }
  sankhya_pdhg_params defaults;
  sankhya_pdhg_gpu_default_params(&defaults);
  auto J = std::make_shared<sih26::Job>();
  try {
    J->submit_time = s->now();
    sih26::prepare(*J, *problem, params ? *params : defaults, s->cfg.cluster_min_nnz,
                   s->cfg.solo_min_nnz);  // host work, outside the lock
  } catch (const Failure& f) {
    sih26::g_last_error = f.message;
    return f.code;
  } catch (const std::bad_alloc&) {
    sih26::g_last_error = "host allocation failed";
    return SANKHYA_GPU_OUT_OF_MEMORY;
  }
  std::lock_guard<std::mutex> lock(s->mu);
  J->ticket = s->next_ticket++;
  *ticket = J->ticket;
  s->jobs[J->ticket] = J;
  if (J->model_error) {
    J->status = SANKHYA_PDHG_MODEL_ERROR;
    J->finished = true;
    J->finish_time = J->submit_time;
  } else if (J->solo) {
    s->solo_waiting.push_back(J);
  } else if (J->bytes > s->pool_bytes && J->legacy_bytes > s->pool_bytes) {
    J->status = SANKHYA_PDHG_NUMERICAL_ERROR;
    J->message = "the LP does not fit the server's device pool";
    J->finished = true;
    J->finish_time = J->submit_time;
  } else {
    s->waiting.push_back(J);
  }
  return SANKHYA_GPU_SUCCESS;
}

int sankhya_pdhg_server_step(sankhya_pdhg_server* server, int32_t* active, int32_t* waiting,
                             int32_t* finished) {
  Server* s = reinterpret_cast<Server*>(server);
  if (!s) {
    sih26::g_last_error = "server must not be NULL";
    return SANKHYA_GPU_INVALID_ARGUMENT;
  }
  std::lock_guard<std::mutex> lock(s->mu);
  sih26::DeviceGuard guard;
  try {
    SIH26_SCUDA(cudaSetDevice(s->cfg.device), SANKHYA_GPU_INIT_FAILED);
    sih26::admit(*s);
    sih26::run_round(*s);
    sih26::admit(*s);
    sih26::run_solo(*s);
  } catch (const Failure& f) {
    sih26::g_last_error = f.message;
    return f.code;
  }
  if (active) *active = static_cast<int32_t>(s->running());
  if (waiting) *waiting = static_cast<int32_t>(s->waiting.size() + s->solo_waiting.size());
  if (finished) {
    int32_t k = 0;
    for (auto& kv : s->jobs) k += kv.second->finished ? 1 : 0;
    *finished = k;
  }
  return SANKHYA_GPU_SUCCESS;
}

int sankhya_pdhg_server_get_stats(sankhya_pdhg_server* server, sankhya_pdhg_server_stats* st) {
  Server* s = reinterpret_cast<Server*>(server);
  if (!s || !st) {
    sih26::g_last_error = "server and stats must not be NULL";
    return SANKHYA_GPU_INVALID_ARGUMENT;
  }
  std::lock_guard<std::mutex> lock(s->mu);
  std::memset(st, 0, sizeof *st);
  st->chunk_attempts = s->chunk >= (1ll << 40) ? 0 : s->chunk;
  st->chunk_source = s->chunk_source;
  st->clusters = s->clusters;
  st->rounds = s->rounds;
  st->last_round_ms = s->last_round_seconds * 1e3;
  std::snprintf(st->family, sizeof st->family, "%s", s->chunk_family.c_str());
  return SANKHYA_GPU_SUCCESS;
}

int sankhya_pdhg_server_result(sankhya_pdhg_server* server, int64_t ticket,
                               sankhya_pdhg_result* r) {
  Server* s = reinterpret_cast<Server*>(server);
  if (!s || !r) {
    sih26::g_last_error = "server and result must not be NULL";
    return SANKHYA_GPU_INVALID_ARGUMENT;
  }
  std::lock_guard<std::mutex> lock(s->mu);
  auto it = s->jobs.find(ticket);
  if (it == s->jobs.end()) {
    sih26::g_last_error = "unknown ticket";
    return SANKHYA_GPU_INVALID_ARGUMENT;
  }
  sih26::Job& J = *it->second;
  if (!J.finished) return SANKHYA_GPU_NOT_READY;
  if (J.solo) {
    // the single-LP engine's own result, with the caller's arrays and the served times
    sankhya_pdhg_result out = J.solo_result;
    out.col_value = r->col_value;
    out.row_dual = r->row_dual;
    out.col_dual = r->col_dual;
    out.farkas_dual = r->farkas_dual;
    out.primal_ray = r->primal_ray;
    if (out.col_value && !J.x.empty()) std::memcpy(out.col_value, J.x.data(), J.n * 8);
    if (out.col_dual && !J.col_dual.empty()) std::memcpy(out.col_dual, J.col_dual.data(), J.n * 8);
    if (out.row_dual && !J.row_dual.empty()) std::memcpy(out.row_dual, J.row_dual.data(), J.m * 8);
    if (out.farkas_dual && !J.farkas.empty()) std::memcpy(out.farkas_dual, J.farkas.data(), J.m * 8);
    if (out.primal_ray && !J.ray.empty()) std::memcpy(out.primal_ray, J.ray.data(), J.n * 8);
    out.setup_seconds = std::max(0.0, J.admit_time - J.submit_time);
    out.solve_seconds = std::max(0.0, J.finish_time - J.admit_time);
    out.total_seconds = std::max(0.0, J.finish_time - J.submit_time);
    *r = out;
    s->jobs.erase(it);
    return SANKHYA_GPU_SUCCESS;
  }
  r->status = J.status;
  const sih26::Ctrl& c = J.last;
  r->converged = c.converged;
  r->iterations = c.iteration;
  r->attempts = c.attempts;
  r->restarts = c.restarts;
  r->evaluations = c.evaluations;
  r->fp32_iterations = 0;
  r->spectral_norm = c.spectral_norm;
  double obj = J.view.objective_offset;
  for (int j = 0; j < J.n && !J.x.empty(); ++j) obj += J.view.cost[j] * J.x[j];
  r->objective = obj;
  const sih26::Residuals& f = c.best;
  r->primal_infeasibility = c.primal_violation;
  r->residuals = sankhya_pdhg_residuals{f.primal, f.dual, f.gap, f.primal_objective,
                                        f.dual_objective, f.absolute_primal, f.absolute_dual,
                                        f.gap_as_verified, f.complementarity};
  const double sense = J.view.maximize ? -1.0 : 1.0;
  r->dual_bound = (J.status == SANKHYA_PDHG_OPTIMAL)
                      ? sense * f.dual_objective + J.view.objective_offset
                      : (J.view.maximize ? INFINITY : -INFINITY);
  r->quality = sih26::quality_from_slots(c.quality, r->objective, r->dual_bound);
  r->quality.primal_infeasibility = r->primal_infeasibility;  // one figure for both fields
  if (r->col_value && !J.x.empty()) std::memcpy(r->col_value, J.x.data(), J.n * 8);
  if (r->col_dual && !J.col_dual.empty()) std::memcpy(r->col_dual, J.col_dual.data(), J.n * 8);
  if (r->row_dual && !J.row_dual.empty()) std::memcpy(r->row_dual, J.row_dual.data(), J.m * 8);
  if (r->farkas_dual && !J.farkas.empty()) std::memcpy(r->farkas_dual, J.farkas.data(), J.m * 8);
  if (r->primal_ray && !J.ray.empty()) std::memcpy(r->primal_ray, J.ray.data(), J.n * 8);
  r->setup_seconds = std::max(0.0, J.admit_time - J.submit_time);
  r->solve_seconds = std::max(0.0, J.finish_time - J.admit_time);
  r->total_seconds = std::max(0.0, J.finish_time - J.submit_time);
  r->h2d_bytes = r->d2h_bytes = 0;
  r->iterate_kernel_seconds = 0.0;
  r->iterate_launches = 0;
  r->kernel_launches = s->launches;
  std::snprintf(r->message, sizeof r->message, "%s", J.message.c_str());
  s->jobs.erase(it);
  return SANKHYA_GPU_SUCCESS;
}

int sankhya_pdhg_gpu_batch_solve(const sankhya_pdhg_problem* problems, int32_t count,
                                 const sankhya_pdhg_params* params, sankhya_pdhg_result* results) {
  if (count < 0 || (count > 0 && (!problems || !results))) {
    sih26::g_last_error = "problems and results must hold count entries";
    return SANKHYA_GPU_INVALID_ARGUMENT;
  }
  sankhya_pdhg_server_config cfg;
  sankhya_pdhg_server_default_config(&cfg);
  if (params) cfg.device = params->device;
  cfg.chunk_attempts = 0;  // run every LP to its end in one launch
  cfg.max_active = std::max(1, std::min(cfg.max_active, count));
  // a pool just large enough for every LP at once (an upper bound of the layout of prepare(): both
  // matrix copies, their slices over the problem as given and the scratch, some 20 FP64 vectors per row
  // and per column, the lists and alignment), instead of a share of all free memory
  {
    size_t bound = size_t(16) << 20;
    for (int k = 0; k < count; ++k) {
      const sankhya_pdhg_problem& q = problems[k];
      if (q.num_rows < 0 || q.num_cols < 0 || q.num_nonzeros < 0) continue;
      bound += 49 * static_cast<size_t>(q.num_nonzeros) +
               300 * (static_cast<size_t>(q.num_rows) + static_cast<size_t>(q.num_cols)) +
               (size_t(64) << 10);
    }
    cfg.pool_bytes = static_cast<int64_t>(bound);
  }
  sankhya_pdhg_server* server = nullptr;
  int rc = sankhya_pdhg_server_create(&cfg, &server);
  if (rc != SANKHYA_GPU_SUCCESS) return rc;
  // host preparation (validation, scaling, layout) of the LPs on several threads; submit is
  // thread-safe and the results do not depend on the order of admission
  std::vector<int64_t> tickets(count);
  std::vector<int> codes(count, SANKHYA_GPU_SUCCESS);
  std::vector<std::string> errors(count);
  {
    const int workers = std::max(1, std::min<int>(count, std::min(16u, std::max(1u, std::thread::hardware_concurrency()))));
    std::atomic<int> next{0};
    std::vector<std::thread> pool;
    for (int w = 0; w < workers; ++w) {
      pool.emplace_back([&] {
        for (int k = next++; k < count; k = next++) {
          codes[k] = sankhya_pdhg_server_submit(server, &problems[k], params, &tickets[k]);
          if (codes[k] != SANKHYA_GPU_SUCCESS) errors[k] = sih26::g_last_error;
        }
      });
    }
    for (auto& t : pool) t.join();
  }
  for (int k = 0; k < count; ++k) {
    if (codes[k] != SANKHYA_GPU_SUCCESS) {
      rc = codes[k];
      sih26::g_last_error = errors[k];
      break;
    }
  }
  int32_t active = 0, waiting = 0, finished = 0;
  while (rc == SANKHYA_GPU_SUCCESS) {
    rc = sankhya_pdhg_server_step(server, &active, &waiting, &finished);
    if (active == 0 && waiting == 0) break;
  }
  for (int k = 0; k < count && rc == SANKHYA_GPU_SUCCESS; ++k)
    rc = sankhya_pdhg_server_result(server, tickets[k], &results[k]);
  sankhya_pdhg_server_free(server);
  return rc;
}

}  // extern "C"
