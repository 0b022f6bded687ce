// Restarted PDHG of one LP on one thread-block cluster with everything an iteration touches in
// shared memory.
//
// The grid-wide iteration kernel (pdhg_kernels.cuh) spends some 10 us per iteration on an LP
// of any size up to a few 100,000 nonzeros: two grid barriers and, per phase, a chain of dependent
// L2 accesses (item, row pointers, column index, gathered entry). An LP of some 10,000 nonzeros
// has microseconds of L2 latency and nanoseconds of work in that. Here
//
//   * each block of a cluster of 1 to 16 owns the rows of A and of A' that the work partition
//     gives it, and keeps their entries (16-bit column indices, values in the level's type), row
//     lengths and step constants in its shared memory;
//   * each block keeps a whole copy of the gathered vectors x and y; a row's owner writes its new
//     entry into every block's copy through distributed shared memory;
//   * phases are separated by the hardware cluster barrier, and the whole solve -- norm estimate,
//     iterations, evaluations, restarts, report -- runs in one launch.
//
// A row is summed in the order of the sliced layout (one lane per short row in stored order, lane
// groups for rows of 33-512 nonzeros, segments beyond) and reductions fold warps, then blocks, as
// the grid-wide kernels do, so on the same partition every bit is theirs.
//
// What bounds it (2,000 x 5,000, 50,000 nonzeros, 14 blocks, FP64, cycles of an iteration's ~9,000):
// the vector exchange (all-to-all stores of 40 + 16 KB through distributed shared memory run at
// some 11 B per cycle and SM), two cluster barriers (450-530 each with release and acquire), and
// chains of dependent shared-memory loads and FP64 divisions; shared-memory bandwidth alone would
// take ~1,500. Loop of that LP, evaluations included: 8.4 ms grid-wide, 4.6 here for 720 iterations
// (FP32 level 8.1 and 4.2); 60 x 150 on one block, 240 iterations: 1.9 and 0.7 ms.
//
// Evaluations run every 40 iterations over the FP64 slices in global memory, as in
// evaluate_kernel; the step that precedes one writes the iterates there.
#pragma once

#include <cooperative_groups.h>

#include <algorithm>
#include <vector>

#include "pdhg_host.cuh"
#include "pdhg_kernels.cuh"
#include "quotient.cuh"
#include "resident_plan.cuh"

namespace sih26 {

constexpr int kTeamSlots = 31;  // reduction slots of an evaluation

#ifdef SIH26_PHASE_TIMING
// Instrumented builds only: cycles of rank 0 per section, read back with sih26_team_clocks.
__device__ unsigned long long g_team_clocks[16];
#define SIH26_TEAM_MARK(k)                                                          \
  do {                                                                              \
    if (threadIdx.x == 0 && tm.rank == 0) {                                         \
      const unsigned long long now_ = clock64();                                    \
      if ((k) >= 0) g_team_clocks[(k) < 0 ? 0 : (k)] += now_ - g_team_clocks[15];   \
      g_team_clocks[15] = clock64();                                                \
    }                                                                               \
  } while (0)
#else
#define SIH26_TEAM_MARK(k) \
  do {                     \
  } while (0)
#endif

// ---- the team of blocks ----------------------------------------------------------------------

struct Team {
  int cs, rank;
  __device__ __forceinline__ void sync() const {
    if (cs == 1) {
      __syncthreads();
    } else {
      asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
    }
  }
};

__device__ __forceinline__ unsigned shared_address(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ unsigned block_address(unsigned a, int rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_block(unsigned a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void st_block(unsigned a, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
// *p = v in every block's copy of the shared array p points into
template <class T>
__device__ __forceinline__ void put_all(const Team& tm, T* p, T v) {
  if (tm.cs == 1) {
    *p = v;
    return;
  }
  const unsigned a = shared_address(p);
  for (int r = 0; r < tm.cs; ++r) st_block(block_address(a, r), v);
}

// Static shared memory of a team kernel.
struct TeamShared {
  Ctrl c;
  Ctrl before;
  double warp[kWarps][kTeamSlots];       // warp totals of the reduction slots
  double block[kMaxTeam][kTeamSlots];    // every block's totals
  double total[kTeamSlots];
  double step[kMaxTeam][3];              // every block's step totals (reference operator)
  double growth[2];                      // the attempt's shrink and grow factors
  double weight[40], rweight[40];        // Halpern weights up to the next evaluation
  unsigned long long section_start;
  int flags[4];                          // best updated, restart, chosen average, certificate kind
};

// The slots first..first+NS-1 of this warp's threads.
template <int NS, unsigned MAXMASK>
__device__ __forceinline__ void team_part(TeamShared& ts, int first, double (&v)[NS]) {
  warp_reduce<NS, MAXMASK>(v);
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int s = 0; s < NS; ++s) ts.warp[threadIdx.x >> 5][first + s] = v[s];
  }
}
// The total over the team of one slot, from every block's: the xor tree of reduce_partials over
// lanes that hold the blocks' totals, so the grid-wide kernels' on the same partition.
__device__ __forceinline__ double fold_blocks(double v, bool have, bool mx) {
  double t = have ? (mx ? dmax(0.0, v) : 0.0 + v) : 0.0;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const double o = __shfl_xor_sync(0xffffffffu, t, off);
    t = mx ? dmax(t, o) : t + o;
  }
  return t;
}
// Totals of slots 0..ns-1 over the team in ts.total: warps in order, then the blocks. A barrier of
// the team has to lie between two calls.
__device__ __forceinline__ void team_total(TeamShared& ts, const Team& tm, int ns, unsigned max_mask) {
  __syncthreads();
  const int s = threadIdx.x;
  if (s < ns) {
    const bool mx = (max_mask >> s) & 1u;
    double t = ts.warp[0][s];
    for (int w = 1; w < kWarps; ++w) t = mx ? dmax(t, ts.warp[w][s]) : t + ts.warp[w][s];
    put_all(tm, &ts.block[tm.rank][s], t);
  }
  tm.sync();
  const int lane = threadIdx.x & 31;
  for (int k = threadIdx.x >> 5; k < ns; k += kWarps) {
    const double t = fold_blocks(ts.block[lane < tm.cs ? lane : 0][k], lane < tm.cs, (max_mask >> k) & 1u);
    if (lane == 0) ts.total[k] = t;
  }
  __syncthreads();
}

// ---- one block's rows of one matrix --------------------------------------------------------------

__device__ __forceinline__ unsigned char* team_memory() {
  extern __shared__ double dyn_smem[];
  return reinterpret_cast<unsigned char*>(dyn_smem);
}

// The lists and entries of one side in this block's shared memory (offsets from team_memory(), so
// the compiler sees shared-memory accesses) and, for a side that is not resident, the CSR and slice
// arrays in global memory.
template <class V>
struct SideView {
  ResidentPlan::Side at;
  int ni, ns, nl;
  const int* gidx;
  const V* gval;
  const int* sidx;
  const V* sval;
  template <class U>
  __device__ __forceinline__ U* in(int offset) const { return reinterpret_cast<U*>(team_memory() + offset); }
  // {first row, rows | lanes << 8 | longest << 16, entry offset, first slot}
  __device__ __forceinline__ int4* items() const { return in<int4>(at.items); }
  // {entry offset, entries, position in the CSR arrays, 0}
  __device__ __forceinline__ int4* segs() const { return in<int4>(at.segs); }
  // {row, first segment, segments, slot}
  __device__ __forceinline__ int4* longs() const { return in<int4>(at.longs); }
  __device__ __forceinline__ double* seg_sum() const { return in<double>(at.seg_sum); }
  // by slot: entries of the row, and where it starts in the CSR arrays
  __device__ __forceinline__ unsigned short* len() const { return in<unsigned short>(at.len); }
  __device__ __forceinline__ int* gptr() const { return in<int>(at.gptr); }
  // epilogue arrays, at.stride slots each
  __device__ __forceinline__ double* epi() const { return in<double>(at.epi); }
  __device__ __forceinline__ unsigned short* idx() const { return in<unsigned short>(at.idx); }
  __device__ __forceinline__ V* val() const { return in<V>(at.val); }
};

// fn(slot, row) for every row of the side, each by one thread.
template <class V, class F>
__device__ __forceinline__ void for_rows(const SideView<V>& sd, F fn) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int q = threadIdx.x; q < sd.nl; q += kThreads) fn(q, sd.longs()[q].x);
  for (int it = warp; it < sd.ni; it += kWarps) {
    const int4 item = sd.items()[it];
    if (lane < (item.y & 255)) fn(item.w + lane, item.x + lane);
  }
}

// The FP64 slice arrays of this block's items, in global memory (once per LP, in a launch before the
// one that reads them through the read-only path).
__device__ inline void fill_slices(const Csr<double>& M, const Part& p, int rank) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int* sidx = const_cast<int*>(p.sell_idx);
  double* sval = static_cast<double*>(const_cast<void*>(p.sell_val));
  const int ib = __ldg(p.blk_item_begin + rank), ie = __ldg(p.blk_item_begin + rank + 1);
  for (int it = ib + warp; it < ie; it += kWarps) {
    const int4 item = __ldg(p.items + it);
    const int rows = item.y - item.x, L = -item.z;
    if (item.z >= 0 || lane >= rows) continue;
    const int b = M.ptr[item.x + lane], len = M.ptr[item.x + lane + 1] - b;
#pragma unroll 4
    for (int k = 0; k < L; ++k) {
      const size_t o = (size_t)item.w + (size_t)k * rows + lane;
      sidx[o] = k < len ? M.idx[b + k] : 0;
      sval[o] = k < len ? M.val64[b + k] : 0.0;
    }
  }
  __syncthreads();
}

// Reads the block's share of a partition into shared memory: the lists always, the entries where
// the plan holds them (values rounded to V as the level's own copies are).
template <class V>
__device__ __noinline__ void load_side(SideView<V>& sd, const ResidentPlan::Side& pl, const Csr<V>& M,
                                       const Part& p, const Part& p64, int rank) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sb = __ldg(p64.blk_seg_begin + rank), lb = __ldg(p64.blk_long_begin + rank),
            ib = __ldg(p64.blk_item_begin + rank);
  const int ns = __ldg(p64.blk_seg_begin + rank + 1) - sb, nl = __ldg(p64.blk_long_begin + rank + 1) - lb,
            ni = __ldg(p64.blk_item_begin + rank + 1) - ib;
  SideView<V> v;
  v.at = pl;
  v.ni = ni;
  v.ns = ns;
  v.nl = nl;
  v.gidx = M.idx;
  v.gval = M.val;
  v.sidx = p.sell_idx;
  v.sval = static_cast<const V*>(p.sell_val);
  int4 *items = v.items(), *segs = v.segs(), *longs = v.longs();
  unsigned short *len = v.len(), *idx = v.idx();
  int* gptr = v.gptr();
  V* val = v.val();
  const int* sidx = p64.sell_idx;
  const double* sval = static_cast<const double*>(p64.sell_val);
  if (warp == 0) {
    // entry offsets and slots: the long rows' segments first, then the items, in order
    int off = 0, slot = nl;
    const auto scan = [&](int v, int& before) {
      int t = v;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, t, d);
        if (lane >= d) t += o;
      }
      before = t - v;
      return __shfl_sync(0xffffffffu, t, 31);
    };
    for (int q0 = 0; q0 < ns; q0 += 32) {
      const int q = q0 + lane;
      const int4 sg = q < ns ? __ldg(p64.segs + sb + q) : make_int4(0, 0, 0, 0);
      int at;
      const int sum = scan(sg.z - sg.y, at);
      if (q < ns) segs[q] = make_int4(off + at, sg.z - sg.y, sg.y, 0);
      off += sum;
    }
    for (int q = lane; q < nl; q += 32) {
      const int4 lr = __ldg(p64.longs + lb + q);
      longs[q] = make_int4(lr.x, lr.y - sb, lr.z, q);
    }
    for (int q0 = 0; q0 < ni; q0 += 32) {
      const int q = q0 + lane;
      int4 it = make_int4(0, 0, 0, 0);
      int rows = 0, size = 0;
      if (q < ni) {
        it = __ldg(p64.items + ib + q);
        rows = it.y - it.x;
        size = it.z < 0 ? 32 * -it.z : __ldg(M.ptr + it.y) - __ldg(M.ptr + it.x);
      }
      int at, sat;
      const int sum = scan(size, at), ssum = scan(rows, sat);
      if (q < ni)
        items[q] = make_int4(it.x, rows | (it.z < 0 ? 0 : it.z << 8) | (it.z < 0 ? -it.z << 16 : 0),
                             pl.resident ? off + at : it.w, slot + sat);
      off += sum;
      slot += ssum;
    }
  }
  if (threadIdx.x == 0) sd = v;
  __syncthreads();
  for (int it = warp; it < ni; it += kWarps) {
    const int4 item = items[it];
    const int rows = item.y & 255, L = item.y >> 16;
    int b = 0;
    if (lane < rows) {
      b = __ldg(M.ptr + item.x + lane);
      len[item.w + lane] = static_cast<unsigned short>(__ldg(M.ptr + item.x + lane + 1) - b);
      gptr[item.w + lane] = b;
    }
    if (!pl.resident) continue;
    if (L > 0) {
      // a slice: entry k of lane l at 32 k + l
      const size_t from = (size_t)__ldg(p64.items + ib + it).w + lane;
      if (lane < rows) {
#pragma unroll 4
        for (int k = 0; k < L; ++k) {
          idx[item.z + 32 * k + lane] = static_cast<unsigned short>(sidx[from + (size_t)k * rows]);
          val[item.z + 32 * k + lane] = static_cast<V>(sval[from + (size_t)k * rows]);
        }
      }
    } else {
      const int from = __shfl_sync(0xffffffffu, b, 0);
      const int count = __ldg(M.ptr + item.x + rows) - from;
#pragma unroll 4
      for (int e = lane; e < count; e += 32) {
        idx[item.z + e] = static_cast<unsigned short>(M.idx[from + e]);
        val[item.z + e] = static_cast<V>(M.val64[from + e]);
      }
    }
  }
  if (pl.resident) {
    for (int q = warp; q < ns; q += kWarps) {
      const int4 sg = segs[q];
#pragma unroll 4
      for (int e = lane; e < sg.y; e += 32) {
        idx[sg.x + e] = static_cast<unsigned short>(__ldg(M.idx + sg.z + e));
        val[sg.x + e] = static_cast<V>(__ldg(M.val64 + sg.z + e));
      }
    }
  }
  __syncthreads();
}

// s_r = sum_k val g(idx) over the side's rows, then epi.apply(slot, row, s_r, epi.load(slot, row)).
// g: the gathered vector in shared memory. Entries out of shared memory (kRes): bound by the latency of
// index, gathered entry and addition and by the instructions around them, so slices are stored 32
// lanes wide (constant strides) and only the entries past the shortest row's end are predicated.
// Entries out of global memory: bound by L2 latency, two batches of kStreamUnroll a short row.
//
// kRound: each product is rounded before it is added, and the gathered entry is scaled by `scale` first
// (the norm estimate's sums, as power_kernel forms them over stream items).
constexpr int kStreamUnroll = 8;
template <bool kRes, bool kRound = false, class V, class Epi>
__device__ __forceinline__ void team_phase(const SideView<V>& sd, const V* __restrict__ g, Epi& epi,
                                           double scale = 1.0) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // rows of slices; longer rows add fused in either mode, as there
  const auto add = [&](double s, V a, V x) {
    if constexpr (kRound)
      return __dadd_rn(s, __dmul_rn(static_cast<double>(a), static_cast<double>(x) * scale));
    else
      return s + static_cast<double>(a) * static_cast<double>(x);
  };
  const auto add_long = [&](double s, V a, V x) {
    if constexpr (kRound) return s + static_cast<double>(a) * (static_cast<double>(x) * scale);
    else return s + static_cast<double>(a) * static_cast<double>(x);
  };
  for (int q = warp; q < sd.ns; q += kWarps) {
    const int4 sg = sd.segs()[q];
    double s = 0.0;
#pragma unroll 4
    for (int k = lane; k < sg.y; k += 32) {
      const int j = kRes ? sd.idx()[sg.x + k] : ld_stream(sd.gidx + sg.z + k);
      const V a = kRes ? sd.val()[sg.x + k] : ld_stream(sd.gval + sg.z + k);
      s = add_long(s, a, g[j]);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) sd.seg_sum()[q] = s;
  }
  for (int it = warp; it < sd.ni; it += kWarps) {
    const int4 item = sd.items()[it];
    const int rows = item.y & 255, lanes = (item.y >> 8) & 255;
    if (lanes == 0) {
      const int L = item.y >> 16, slot = item.w + lane, row = item.x + lane;
      const bool mine = lane < rows;
      typename Epi::In in{};
      int len = 0;
      if (mine) {
        in = epi.load(slot, row);
        len = sd.len()[slot];
      }
      double s = 0.0;
      if constexpr (kRes) {
        // Rows are sorted by length: up to the last lane's every lane has an entry. FP32 keeps eight entries
        // in flight and takes the rest of a row four at a time: 2.86 -> 2.61 us an iteration at 600 entries,
        // 5.70 -> 5.45 at 50,000. FP64 gained 1 to 4 % alone and lost 1.5 % in a batch: four, then one by one.
        const int full = __shfl_sync(0xffffffffu, len, rows - 1);
        const unsigned short* __restrict__ pi = sd.idx() + item.z + lane;
        const V* __restrict__ pv = sd.val() + item.z + lane;
        if (mine) {
          int k = 0;
          if constexpr (sizeof(V) == 4) {
            for (; k + 8 <= full; k += 8, pi += 256, pv += 256) {
              int j[8];
              V a[8], x[8];
#pragma unroll
              for (int t = 0; t < 8; ++t) j[t] = pi[32 * t], a[t] = pv[32 * t];
#pragma unroll
              for (int t = 0; t < 8; ++t) x[t] = g[j[t]];
#pragma unroll
              for (int t = 0; t < 8; ++t) s = add(s, a[t], x[t]);
            }
            for (; k < len; k += 4, pi += 128, pv += 128) {
              const bool b1 = k + 1 < len, b2 = k + 2 < len, b3 = k + 3 < len;
              const int j0 = pi[0], j1 = b1 ? pi[32] : 0, j2 = b2 ? pi[64] : 0, j3 = b3 ? pi[96] : 0;
              const V a0 = pv[0], a1 = b1 ? pv[32] : V(0), a2 = b2 ? pv[64] : V(0), a3 = b3 ? pv[96] : V(0);
              const V x0 = g[j0], x1 = g[j1], x2 = g[j2], x3 = g[j3];
              s = add(s, a0, x0);
              if (b1) s = add(s, a1, x1);
              if (b2) s = add(s, a2, x2);
              if (b3) s = add(s, a3, x3);
            }
          } else {
            for (; k + 4 <= full; k += 4, pi += 128, pv += 128) {
              const int j0 = pi[0], j1 = pi[32], j2 = pi[64], j3 = pi[96];
              const V a0 = pv[0], a1 = pv[32], a2 = pv[64], a3 = pv[96];
              const V x0 = g[j0], x1 = g[j1], x2 = g[j2], x3 = g[j3];
              s = add(s, a0, x0);
              s = add(s, a1, x1);
              s = add(s, a2, x2);
              s = add(s, a3, x3);
            }
            for (; k < len; ++k, pi += 32, pv += 32) s = add(s, pv[0], g[pi[0]]);
          }
        }
      } else {
        constexpr int U = kStreamUnroll;
        const int* si = sd.sidx + item.z + lane;
        const V* sv = sd.sval + item.z + lane;
        for (int k0 = 0; k0 < L; k0 += U) {
          int j[U];
          V a[U];
#pragma unroll
          for (int t = 0; t < U; ++t) {
            const bool live = k0 + t < len;
            j[t] = live ? ld_stream(si + t * rows) : 0;
            a[t] = live ? ld_stream(sv + t * rows) : V(0);
          }
          si += U * rows;
          sv += U * rows;
#pragma unroll
          for (int t = 0; t < U; ++t)
            if (k0 + t < len) s = add(s, a[t], g[j[t]]);
        }
      }
      if (mine) epi.apply(slot, row, s, in);
    } else {
      const int gid = lane / lanes, gl = lane - gid * lanes;
      const int slot = item.w + gid, row = item.x + gid;
      const bool valid = gid < rows;
      typename Epi::In in{};
      double s = 0.0;
      if (valid) {
        if (gl == 0) in = epi.load(slot, row);
        const int len = sd.len()[slot];
        const int b = kRes ? item.z + (sd.gptr()[slot] - sd.gptr()[item.w]) : sd.gptr()[slot];
#pragma unroll 4
        for (int k = gl; k < len; k += lanes) {
          const int j = kRes ? sd.idx()[b + k] : ld_stream(sd.gidx + b + k);
          const V a = kRes ? sd.val()[b + k] : ld_stream(sd.gval + b + k);
          s = add_long(s, a, g[j]);
        }
      }
      for (int off = lanes >> 1; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
      if (valid && gl == 0) epi.apply(slot, row, s, in);
    }
  }
  if (sd.nl > 0) {
    __syncthreads();
    for (int q = warp; q < sd.nl; q += kWarps) {
      const int4 lr = sd.longs()[q];
      typename Epi::In in{};
      if (lane == 0) in = epi.load(lr.w, lr.x);
      double s = 0.0;
      for (int k = lane; k < lr.z; k += 32) s += sd.seg_sum()[lr.y + k];
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
      if (lane == 0) epi.apply(lr.w, lr.x, s, in);
    }
  }
}
// kStreams: the side's entries may be in global memory (the batched engine, and the norm estimate's FP64 view
// beside an FP32 level; a single LP's own plan has none such).
template <bool kStreams, class V, class Epi>
__device__ __forceinline__ void side_phase(const SideView<V>& sd, const V* g, Epi& epi) {
  if (!kStreams || sd.at.resident) team_phase<true>(sd, g, epi);
  else team_phase<false>(sd, g, epi);
}

// ---- the steps ----------------------------------------------------------------------------------
//
// Epilogue arrays by slot (e0 .. in the order of the loads). Columns: c (FP32 level: c + A'yr),
// lower and upper bound (FP32 level: relative to xr), then x_0 (Halpern, FP64) or the running sum
// (reference). Rows, FP64: both bounds, then y_0 and A x_0 (Halpern) or the running sum and two
// buffers of A x (reference); FP32 level: yr, A xr, both bounds, then the reference operator's.

// project() on bounds whose absent sides are infinite (effective_lower / _upper)
__device__ __forceinline__ double clamp(double v, double lo, double hi) {
  double t = v > hi ? hi : v;
  t = v < lo ? lo : t;
  return t;
}
__device__ __forceinline__ double effective_lower(double lo) { return finite_bound(lo) ? lo : -INFINITY; }
__device__ __forceinline__ double effective_upper(double hi) { return finite_bound(hi) ? hi : INFINITY; }

template <class T>
struct TeamPrimalHalpern {
  Team tm;
  T* x;
  const double* e;
  int es;
  double tau, w;
  T *gx, *gxn, *gxt;  // non-null: the step before an evaluation, whose iterates it reads
  struct In {
    double xo, c, lo, hi, x0;
  };
  __device__ __forceinline__ In load(int q, int j) const {
    return In{static_cast<double>(x[j]), e[q], e[es + q], e[2 * es + q], kDelta<T> ? 0.0 : e[3 * es + q]};
  }
  __device__ __forceinline__ void apply(int, int j, double s, const In& v) const {
    // halpern_primal
    const T xp = static_cast<T>(clamp(v.xo - tau * (v.c + s), v.lo, v.hi));
    T xn;
    if constexpr (kDelta<T>)
      xn = static_cast<T>(w * (2.0 * static_cast<double>(xp) - v.xo));
    else
      xn = static_cast<T>(w * (2.0 * static_cast<double>(xp) - v.xo) + (1.0 - w) * v.x0);
    put_all(tm, x + j, xn);
    if (gxn) {
      gx[j] = static_cast<T>(v.xo);
      gxn[j] = xn;
      gxt[j] = xp;
    }
  }
};

template <class T>
struct TeamDualHalpern {
  Team tm;
  T* y;
  const double* e;
  int es;
  double sigma, w, rsigma, rw;  // and their reciprocals
  T *gy, *gyn, *gyt;
  double* gax;
  struct In {
    double yo, lo, hi, y0, a0;
  };
  __device__ __forceinline__ In load(int q, int i) const {
    const double yo = static_cast<double>(y[i]);
    if constexpr (kDelta<T>) return In{yo, e[2 * es + q], e[3 * es + q], e[q], e[es + q]};
    else return In{yo, e[q], e[es + q], e[2 * es + q], e[3 * es + q]};
  }
  __device__ __forceinline__ void apply(int, int i, double s, const In& v) const {
    // halpern_dual
    T yp, yn;
    if constexpr (kDelta<T>) {
      const double u = (v.y0 + v.yo) + sigma * (v.a0 + quotient(s, w, rw));
      const double full = u - sigma * clamp(quotient(u, sigma, rsigma), v.lo, v.hi);
      yp = static_cast<T>(full - v.y0);
      yn = static_cast<T>(w * (2.0 * static_cast<double>(yp) - v.yo));
    } else {
      const double axbar = quotient(s - (1.0 - w) * v.a0, w, rw);
      const double u = v.yo + sigma * axbar;
      yp = static_cast<T>(u - sigma * clamp(quotient(u, sigma, rsigma), v.lo, v.hi));
      yn = static_cast<T>(w * (2.0 * static_cast<double>(yp) - v.yo) + (1.0 - w) * v.y0);
    }
    put_all(tm, y + i, yn);
    if (gyn) {
      gy[i] = static_cast<T>(v.yo);
      gyn[i] = yn;
      gyt[i] = yp;
      gax[i] = s;
    }
  }
};

template <class T>
struct TeamPrimal {
  Team tm;
  const T* x;
  T* xn;
  double* e;
  int es;
  double tau;
  int pending;
  double* acc;
  struct In {
    double xo, c, lo, hi, xs;
  };
  __device__ __forceinline__ In load(int q, int j) const {
    return In{static_cast<double>(x[j]), e[q], e[es + q], e[2 * es + q], e[3 * es + q]};
  }
  __device__ __forceinline__ void apply(int q, int j, double s, const In& v) const {
    if (pending) e[3 * es + q] = v.xs + v.xo;
    const T xs = static_cast<T>(clamp(v.xo - tau * (v.c + s), v.lo, v.hi));
    put_all(tm, xn + j, xs);
    const double d = static_cast<double>(xs) - v.xo;
    acc[0] += d * d;
  }
};

template <class T>
struct TeamDual {
  static constexpr int kBounds = kDelta<T> ? 2 : 0, kSum = kDelta<T> ? 4 : 2;
  Team tm;
  const T* y;
  T* yn;
  double* e;
  int es;
  int cur;  // which A x buffer is the stored iterate's
  double sigma, rsigma;
  int pending;
  double* acc;
  struct In {
    double yo, aold, lo, hi, ys, yr, axr;
  };
  __device__ __forceinline__ In load(int q, int i) const {
    In v;
    v.yo = static_cast<double>(y[i]);
    v.lo = e[kBounds * es + q];
    v.hi = e[(kBounds + 1) * es + q];
    v.ys = e[kSum * es + q];
    v.aold = e[(kSum + 1 + cur) * es + q];
    v.yr = kDelta<T> ? e[q] : 0.0;
    v.axr = kDelta<T> ? e[es + q] : 0.0;
    return v;
  }
  __device__ __forceinline__ void apply(int q, int i, double anew, const In& v) const {
    if (pending) e[kSum * es + q] = v.ys + v.yo;
    T ys;
    if constexpr (kDelta<T>) {
      const double w = (v.yr + v.yo) + sigma * (v.axr + 2.0 * anew - v.aold);
      ys = static_cast<T>(w - sigma * clamp(quotient(w, sigma, rsigma), v.lo, v.hi) - v.yr);
    } else {
      const double w = v.yo + sigma * (2.0 * anew - v.aold);
      ys = static_cast<T>(w - sigma * clamp(quotient(w, sigma, rsigma), v.lo, v.hi));
    }
    put_all(tm, yn + i, ys);
    e[(kSum + 1 + (cur ^ 1)) * es + q] = anew;
    const double d = static_cast<double>(ys) - v.yo;
    acc[1] += d * d;
    acc[2] += d * (anew - v.aold);
  }
};

// A x of the starting point, with the iteration's own sums (FP64 level).
struct TeamStoreAx {
  double* ax;
  double* axr;
  struct In {};
  __device__ __forceinline__ In load(int, int) const { return In{}; }
  __device__ __forceinline__ void apply(int, int i, double s, const In&) const {
    ax[i] = s;
    axr[i] = s;
  }
};

// The vector copies and the epilogue arrays from the LP's state in global memory.
template <class T>
__device__ __forceinline__ void load_vectors(const Prob<T>& P, const State<T>& S, const ResidentPlan& pl,
                                             int cur) {
  unsigned char* mem = team_memory();
  T* x = reinterpret_cast<T*>(mem + pl.x[cur]);
  T* y = reinterpret_cast<T*>(mem + pl.y[cur]);
  for (int j = threadIdx.x; j < P.n; j += kThreads) x[j] = S.x[cur][j];
  for (int i = threadIdx.x; i < P.m; i += kThreads) y[i] = S.y[cur][i];
}
template <class T>
__device__ __forceinline__ void load_epilogues(const Prob<T>& P, const State<T>& S, const SideView<T>& sp,
                                               const SideView<T>& sd, bool halpern, int cur) {
  for_rows(sp, [&](int q, int j) {
    double* e = sp.epi() + q;
    const int es = sp.at.stride;
    if constexpr (kDelta<T>) {
      e[0] = S.cg[j];
      e[es] = effective_lower(static_cast<double>(S.dl[j]));
      e[2 * es] = effective_upper(static_cast<double>(S.du[j]));
      if (!halpern) e[3 * es] = S.xsum[j];
    } else {
      e[0] = static_cast<double>(P.c[j]);
      e[es] = effective_lower(static_cast<double>(P.cl[j]));
      e[2 * es] = effective_upper(static_cast<double>(P.cu[j]));
      e[3 * es] = halpern ? S.xr[j] : S.xsum[j];
    }
  });
  for_rows(sd, [&](int q, int i) {
    double* e = sd.epi() + q;
    const int es = sd.at.stride;
    int k = 0;
    if constexpr (kDelta<T>) {
      e[0] = S.yr[i];
      e[es] = S.axr[i];
      e[2 * es] = effective_lower(P.rl64[i]);
      e[3 * es] = effective_upper(P.ru64[i]);
      k = 4;
    } else {
      e[0] = effective_lower(static_cast<double>(P.rl[i]));
      e[es] = effective_upper(static_cast<double>(P.ru[i]));
      k = 2;
      if (halpern) {
        e[2 * es] = S.yr[i];
        e[3 * es] = S.axr[i];
      }
    }
    if (!halpern) {
      e[k * es] = S.ysum[i];
      e[(k + 1 + cur) * es] = S.ax[cur][i];
    }
  });
}

// `steps` (at most 40) Halpern steps, the last of which writes the iterates to global memory. A function
// of its own, for its registers: the loop keeps both sides' offsets and the step constants in them.
template <class T, bool kStreams>
__device__ __noinline__ void team_halpern(const State<T>& S, const ResidentPlan& pl, const SideView<T>& sp_,
                                          const SideView<T>& sd_, TeamShared& ts, const Team& tm_, int steps) {
  const SideView<T> sp = sp_, sd = sd_;
  const Team tm = tm_;
  unsigned char* mem = team_memory();
  T* x = reinterpret_cast<T*>(mem + pl.x[0]);
  T* y = reinterpret_cast<T*>(mem + pl.y[0]);
  Ctrl& c = ts.c;
  // the steps' weights and their reciprocals
  if (threadIdx.x < steps) {
    const double w = (double)(c.averaged + 1 + threadIdx.x) / (double)(c.averaged + 2 + threadIdx.x);
    ts.weight[threadIdx.x] = w;
    ts.rweight[threadIdx.x] = quotient_reciprocal(w);
  }
  const double tau = c.eta / c.omega, sigma = c.eta * c.omega, rsigma = quotient_reciprocal(sigma);
  int cur = c.cur;
  __syncthreads();
  for (int t = 0; t < steps; ++t, cur ^= 1) {
    const bool dump = t + 1 == steps;
    const double w = ts.weight[t], rw = ts.rweight[t];
    TeamPrimalHalpern<T> ps{tm, x, sp.epi(), sp.at.stride, tau, w, dump ? S.x[cur] : nullptr,
                            dump ? S.x[cur ^ 1] : nullptr, dump ? S.xt : nullptr};
    side_phase<kStreams>(sp, y, ps);
    SIH26_TEAM_MARK(0);
    tm.sync();
    SIH26_TEAM_MARK(1);
    TeamDualHalpern<T> ds{tm, y, sd.epi(), sd.at.stride, sigma, w, rsigma, rw,
                          dump ? S.y[cur] : nullptr,
                          dump ? S.y[cur ^ 1] : nullptr, dump ? S.yt : nullptr, dump ? S.ax[cur ^ 1] : nullptr};
    side_phase<kStreams>(sd, x, ds);
    SIH26_TEAM_MARK(2);
    tm.sync();
    SIH26_TEAM_MARK(3);
  }
  if (threadIdx.x == 0) {
    c.cur = cur;
    c.averaged += steps;
    c.iteration += steps;
    c.attempts += steps;
    c.pending = 0;
    if (steps > 0 && c.iteration % 40 == 0) c.state = kNeedEval;
  }
  __syncthreads();
}

// The end of an attempt: its reductions over the team and the step control, in every block.
__device__ __forceinline__ void finish_attempt(TeamShared& ts, const Team& tm, double (&acc)[3]) {
  Ctrl& c = ts.c;
  team_part<3, 0u>(ts, 0, acc);
  __syncthreads();
  if (threadIdx.x < 3) {
    double t = ts.warp[0][threadIdx.x];
    for (int w = 1; w < kWarps; ++w) t += ts.warp[w][threadIdx.x];
    put_all(tm, &ts.step[tm.rank][threadIdx.x], t);
  }
  tm.sync();
  if (threadIdx.x < 32) {
    const int b = threadIdx.x < tm.cs ? threadIdx.x : 0;
    double tot[3];
#pragma unroll
    for (int s = 0; s < 3; ++s) tot[s] = fold_blocks(ts.step[b][s], threadIdx.x < tm.cs, false);
    if (threadIdx.x == 0) step_control(c, tot, ts.growth[0], ts.growth[1]);
  }
  __syncthreads();
}

// One attempt of the reference's adaptive step.
template <class T, bool kStreams>
__device__ __noinline__ void team_attempt(const ResidentPlan& pl,
                                          const SideView<T>& sp_, const SideView<T>& sd_, TeamShared& ts,
                                          const Team& tm_) {
  const SideView<T> sp = sp_, sd = sd_;
  const Team tm = tm_;
  unsigned char* mem = team_memory();
  Ctrl& c = ts.c;
  const int cur = c.cur, nxt = cur ^ 1;
  T *xc = reinterpret_cast<T*>(mem + pl.x[cur]), *xn = reinterpret_cast<T*>(mem + pl.x[nxt]);
  T *yc = reinterpret_cast<T*>(mem + pl.y[cur]), *yn = reinterpret_cast<T*>(mem + pl.y[nxt]);
  const double tau = c.eta / c.omega, sigma = c.eta * c.omega;
  double acc[3] = {0.0, 0.0, 0.0};
  TeamPrimal<T> ps{tm, xc, xn, sp.epi(), sp.at.stride, tau, c.pending, acc};
  side_phase<kStreams>(sp, yc, ps);
  // the step factors depend on the iteration alone: formed beside the phases, by a thread of the
  // last warp, which has the fewest rows
  if (threadIdx.x == kThreads - 1) step_growth(c.iteration, ts.growth[0], ts.growth[1]);
  tm.sync();
  TeamDual<T> ds{tm, yc, yn, sd.epi(), sd.at.stride, cur, sigma, quotient_reciprocal(sigma), c.pending, acc};
  side_phase<kStreams>(sd, xn, ds);
  finish_attempt(ts, tm, acc);
}

// ---- an LP whose vectors do not fit beside each other -------------------------------------------------
//
// s_r = sum_k val vec[idx] over this block's rows, then the epilogue (the grid-wide kernels', whose
// inputs are in global memory). The block copies the gathered vector into shared memory, coalesced, and
// passes over its rows. Bound by reading the matrix and the vector from L2 (12 bytes an entry and
// 8 bytes per column and row and block); gathering the vector's entries from L2 instead moves a 32-byte
// sector for each that L1 does not hold.
template <int NS, bool kRound, class Epi>
__device__ __forceinline__ void turn_phase(const Csr<double>& M, const Part& p, const double* vec, int size,
                                           double scale, const Epi& epi, double (&acc)[NS], int rank) {
  constexpr int U = 8;
  double* const g = reinterpret_cast<double*>(team_memory());
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ib = __ldg(p.blk_item_begin + rank), ie = __ldg(p.blk_item_begin + rank + 1);
  const int lb = __ldg(p.blk_long_begin + rank), le = __ldg(p.blk_long_begin + rank + 1);
  const int sb = __ldg(p.blk_seg_begin + rank), se = __ldg(p.blk_seg_begin + rank + 1);
  const int* __restrict__ sidx = p.sell_idx;
  const double* __restrict__ sval = static_cast<const double*>(p.sell_val);
  const auto add = [&](double s, double a, double x) {
    if constexpr (kRound) return __dadd_rn(s, __dmul_rn(a, x));
    else return s + a * x;
  };
  __syncthreads();  // the vector before is done with
  {
    // vectors start on 256 bytes: two entries a load
    const double2* src = reinterpret_cast<const double2*>(vec);
    double2* dst = reinterpret_cast<double2*>(g);
#pragma unroll 8
    for (int k = threadIdx.x; k < size / 2; k += kThreads) {
      double2 t = src[k];
      if constexpr (kRound) {
        t.x *= scale;
        t.y *= scale;
      }
      dst[k] = t;
    }
    if ((size & 1) && threadIdx.x == 0) g[size - 1] = kRound ? vec[size - 1] * scale : vec[size - 1];
  }
  __syncthreads();
  // long rows in segments, a warp each, folded at the end (a warp for a whole row of 20,000 took 46 us an
  // iteration where the segments take 23)
  for (int q = sb + warp; q < se; q += kWarps) {
    const int4 sg = __ldg(p.segs + q);
    double s = 0.0;
#pragma unroll
    for (int t = 0; t < kSegment / 32; ++t) {
      const int k = sg.y + lane + 32 * t;
      if (k < sg.z) s += __ldg(M.val64 + k) * g[__ldg(M.idx + k)];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) p.seg_sum[q] = s;
  }
  // the headers of the warp's next rows are on their way while these are summed: the item two
  // ahead, its rows' range one ahead
  struct Header {
    int b, len;
  };
  const auto lane_row = [&](const int4& item) { return item.z < 0 ? item.x + lane : item.x + lane / item.z; };
  const auto header = [&](const int4& item) {
    Header h{0, 0};
    const int r = lane_row(item);
    if (r < item.y) {
      h.b = __ldg(M.ptr + r);
      h.len = __ldg(M.ptr + r + 1) - h.b;
    }
    return h;
  };
  const int4 none = make_int4(0, 0, -1, 0);
  int it = ib + warp;
  int4 item = it < ie ? __ldg(p.items + it) : none;
  int4 next = it + kWarps < ie ? __ldg(p.items + it + kWarps) : none;
  Header h = header(item);
  for (; it < ie; it += kWarps) {
    const int4 after = it + 2 * kWarps < ie ? __ldg(p.items + it + 2 * kWarps) : none;
    const Header hn = header(next);
    const int rows = item.y - item.x, r = lane_row(item);
    const bool mine = r < item.y;
    typename Epi::In in{};
    double s[1] = {0.0};
    if (item.z < 0) {
      if (mine) in = epi.load(r);
      const int* si = sidx + item.w + lane;
      const double* sv = sval + item.w + lane;
      for (int k = 0; __any_sync(0xffffffffu, k < h.len); k += U) {
        int j[U];
        double a[U];
#pragma unroll
        for (int t = 0; t < U; ++t) {
          const bool live = k + t < h.len;
          j[t] = live ? __ldg(si + (k + t) * rows) : 0;
          a[t] = live ? __ldg(sv + (k + t) * rows) : 0.0;
        }
#pragma unroll
        for (int t = 0; t < U; ++t)
          if (k + t < h.len) s[0] = add(s[0], a[t], g[j[t]]);
      }
      if (mine) epi.apply(r, s, in, acc);
    } else {
      const int lanes = item.z, gl = lane & (lanes - 1);
      if (mine) {
        if (gl == 0) in = epi.load(r);
#pragma unroll 8
        for (int k = gl; k < h.len; k += lanes) s[0] += __ldg(M.val64 + h.b + k) * g[__ldg(M.idx + h.b + k)];
      }
      for (int off = lanes >> 1; off > 0; off >>= 1) s[0] += __shfl_xor_sync(0xffffffffu, s[0], off);
      if (mine && gl == 0) epi.apply(r, s, in, acc);
    }
    item = next;
    next = after;
    h = hn;
  }
  if (le > lb) {
    __syncthreads();
    for (int q = lb + warp; q < le; q += kWarps) {
      const int4 lr = __ldg(p.longs + q);
      typename Epi::In in{};
      if (lane == 0) in = epi.load(lr.x);
      double s[1] = {0.0};
      for (int k = lane; k < lr.z; k += 32) s[0] += p.seg_sum[lr.y + k];
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) s[0] += __shfl_xor_sync(0xffffffffu, s[0], off);
      if (lane == 0) epi.apply(lr.x, s, in, acc);
    }
  }
}

// One pass over the rows of a matrix, kTurns: the vector copied into shared memory, else its entries gathered out
// of L2 by the grid-wide kernels' code.
template <bool kTurns, int NS, bool kRound, class Epi>
__device__ __forceinline__ void vector_phase(const Csr<double>& M, const Part& p, const double* vec, int size,
                                             double scale, const Epi& epi, double (&acc)[NS], int rank) {
  if constexpr (kTurns) {
    turn_phase<NS, kRound>(M, p, vec, size, scale, epi, acc, rank);
  } else if constexpr (kRound) {
    run_phase<1, NS, false, true, kSliceUnroll, false, true>(M.ptr, M.idx, M.val64, p, ScaledGather{vec, scale}, epi,
                                                             acc, nullptr, rank);
  } else {
    run_phase<1, NS, false, true>(M.ptr, M.idx, M.val64, p, Gather1<double>{vec}, epi, acc, nullptr, rank);
  }
}

template <bool kTurns>
__device__ __noinline__ void vector_halpern(const Prob<double>& P, const State<double>& S, TeamShared& ts,
                                            const Team& tm_, int steps) {
  const Team tm = tm_;
  Ctrl& c = ts.c;
  const double tau = c.eta / c.omega, sigma = c.eta * c.omega;
  long long k = c.averaged;
  int cur = c.cur;
  double acc[3] = {0.0, 0.0, 0.0};
  for (int t = 0; t < steps; ++t, ++k, cur ^= 1) {
    const double w = (double)(k + 1) / (double)(k + 2);
    vector_phase<kTurns, 3, false>(
        P.AT, P.pate, S.y[cur], P.m, 1.0,
        PrimalStepHalpern<double>{S.x[cur], S.x[cur ^ 1], S.xt, P.c, P.cl, P.cu, S.xr, tau, w}, acc, tm.rank);
    tm.sync();
    vector_phase<kTurns, 3, false>(P.A, P.pae, S.x[cur ^ 1], P.n, 1.0,
                                   DualStepHalpern<double>{S.y[cur], S.y[cur ^ 1], S.yt, S.ax[cur ^ 1], P.rl, P.ru,
                                                           S.yr, S.axr, sigma, w},
                                   acc, tm.rank);
    tm.sync();
  }
  if (threadIdx.x == 0) {
    c.cur = cur;
    c.averaged = k;
    c.iteration += steps;
    c.attempts += steps;
    c.pending = 0;
    if (steps > 0 && c.iteration % 40 == 0) c.state = kNeedEval;
  }
  __syncthreads();
}

template <bool kTurns>
__device__ __noinline__ void vector_attempt(const Prob<double>& P, const State<double>& S, TeamShared& ts,
                                            const Team& tm_) {
  const Team tm = tm_;
  Ctrl& c = ts.c;
  const int cur = c.cur, nxt = cur ^ 1;
  const double tau = c.eta / c.omega, sigma = c.eta * c.omega;
  double acc[3] = {0.0, 0.0, 0.0};
  vector_phase<kTurns, 3, false>(P.AT, P.pate, S.y[cur], P.m, 1.0,
                                 PrimalStep<double>{S.x[cur], S.x[nxt], P.c, P.cl, P.cu, S.xsum, tau, c.pending},
                                 acc, tm.rank);
  if (threadIdx.x == kThreads - 1) step_growth(c.iteration, ts.growth[0], ts.growth[1]);
  tm.sync();
  vector_phase<kTurns, 3, false>(P.A, P.pae, S.x[nxt], P.n, 1.0,
                                 DualStep<double>{S.y[cur], S.y[nxt], S.ax[cur], S.ax[nxt], P.rl, P.ru, S.ysum,
                                                  sigma, c.pending},
                                 acc, tm.rank);
  finish_attempt(ts, tm, acc);
}

// The norm estimate (team_power) and A x_0 of such an LP. v sits in S.xt while the estimate runs and u in
// S.yt; neither is read before the first step writes it.
template <bool kTurns>
__device__ __noinline__ double vector_setup(const Prob<double>& P, const State<double>& S, int nnz, TeamShared& ts,
                                            const Team& tm_) {
  const Team tm = tm_;
  double norm = 1.0;
  if (P.m > 0 && P.n > 0 && nnz > 0) {
    double *v = S.xt, *u = S.yt;
    const double* start = reinterpret_cast<const double*>(S.xc);
    double len2[1] = {0.0};
    for (int j = tm.rank * kThreads + threadIdx.x; j < P.n; j += tm.cs * kThreads) {
      v[j] = start[j];
      len2[0] += v[j] * v[j];
    }
    team_part<1, 0u>(ts, 0, len2);
    team_total(ts, tm, 1, 0u);
    bool zero = false;
    for (int step = 0; step < 30; ++step) {
      const double length = sqrt(ts.total[0]);
      if (length == 0.0) {
        zero = true;
        break;
      }
      double dummy[1] = {0.0};
      vector_phase<kTurns, 1, true>(P.A, P.pae, v, P.n, 1.0 / length, StoreRow<1>{u, -1}, dummy, tm.rank);
      tm.sync();
      double nx[1] = {0.0};
      vector_phase<kTurns, 1, true>(P.AT, P.pate, u, P.m, 1.0, StoreRow<1>{v, 0}, nx, tm.rank);
      team_part<1, 0u>(ts, 0, nx);
      team_total(ts, tm, 1, 0u);
    }
    const double root = zero ? 0.0 : sqrt(sqrt(ts.total[0]));
    norm = root > 0.0 ? root * 1.01 : 1.0;
    tm.sync();
  }
  double dummy[1] = {0.0};
  const int cur = ts.c.cur;
  vector_phase<kTurns, 1, false>(P.A, P.pae, S.x[cur], P.n, 1.0, StoreRow<1>{S.ax[cur], -1}, dummy, tm.rank);
  tm.sync();
  for (int i = tm.rank * kThreads + threadIdx.x; i < P.m; i += tm.cs * kThreads) S.axr[i] = S.ax[cur][i];
  return norm;
}

// The reference operator's state to global memory, for an evaluation or the next launch.
template <class T>
__device__ __forceinline__ void spill(const State<T>& S, const ResidentPlan& pl, const SideView<T>& sp,
                                      const SideView<T>& sd, const Ctrl& c) {
  unsigned char* mem = team_memory();
  constexpr int kSum = TeamDual<T>::kSum;
  for_rows(sp, [&](int q, int j) {
    for (int k = 0; k < 2; ++k) S.x[k][j] = reinterpret_cast<const T*>(mem + pl.x[k])[j];
    S.xsum[j] = sp.epi()[3 * sp.at.stride + q];
  });
  for_rows(sd, [&](int q, int i) {
    for (int k = 0; k < 2; ++k) S.y[k][i] = reinterpret_cast<const T*>(mem + pl.y[k])[i];
    S.ysum[i] = sd.epi()[kSum * sd.at.stride + q];
    S.ax[c.cur][i] = sd.epi()[(kSum + 1 + c.cur) * sd.at.stride + q];
  });
}

// ---- norm estimate, evaluation and report over the state in global memory ---------------------------

// Stores a row sum in every block's copy of a vector; optionally its square.
struct TeamStoreRow {
  Team tm;
  double* out;
  double* square;
  struct In {};
  __device__ __forceinline__ In load(int, int) const { return In{}; }
  __device__ __forceinline__ void apply(int, int r, double s, const In&) const {
    put_all(tm, out + r, s);
    if (square) *square += s * s;
  }
};

// Norm estimate of the LP's scaled matrix (src/la/scaling.cpp:161-194); S.xc holds the random start in
// its first n doubles. With a plan in FP64 the sides are in shared memory (loaded by the caller) and v
// and u are exchanged like the iterates; without one both live in S.xc and S.yc. The 30 steps' 60
// phases took 330 us out of global memory on the 2,000 x 5,000 LP.
template <class T, bool kStreams>
__device__ __noinline__ double team_power(const Prob<T>& P, const State<T>& S, int nnz, const ResidentPlan& pl,
                                          const SideView<double>& sp_, const SideView<double>& sd_, TeamShared& ts,
                                          const Team& tm_) {
  if (P.m == 0 || P.n == 0 || nnz == 0) return 1.0;
  const Team tm = tm_;
  double* v = reinterpret_cast<double*>(S.xc);
  double* u = reinterpret_cast<double*>(S.yc);
  double len2[1] = {0.0};
  for (int j = tm.rank * kThreads + threadIdx.x; j < P.n; j += tm.cs * kThreads) len2[0] += v[j] * v[j];
  team_part<1, 0u>(ts, 0, len2);
  if (pl.cs > 0) {
    const SideView<double> sp = sp_, sd = sd_;
    double* x = reinterpret_cast<double*>(team_memory() + pl.x[0]);
    double* y = reinterpret_cast<double*>(team_memory() + pl.y[0]);
    for (int j = threadIdx.x; j < P.n; j += kThreads) x[j] = v[j];
    team_total(ts, tm, 1, 0u);
    for (int step = 0; step < 30; ++step) {
      const double length = sqrt(ts.total[0]);
      if (length == 0.0) return 1.0;
      TeamStoreRow to_u{tm, y, nullptr};
      if (!kStreams || sd.at.resident) team_phase<true, true>(sd, x, to_u, 1.0 / length);
      else team_phase<false, true>(sd, x, to_u, 1.0 / length);
      tm.sync();
      double nx[1] = {0.0};
      TeamStoreRow to_v{tm, x, nx};
      if (!kStreams || sp.at.resident) team_phase<true, true>(sp, y, to_v);
      else team_phase<false, true>(sp, y, to_v);
      team_part<1, 0u>(ts, 0, nx);
      team_total(ts, tm, 1, 0u);
    }
  } else {
    team_total(ts, tm, 1, 0u);
    for (int step = 0; step < 30; ++step) {
      const double length = sqrt(ts.total[0]);
      if (length == 0.0) return 1.0;
      double dummy[1] = {0.0};
      run_phase<1, 1, false, true, kSliceUnroll, false, true>(P.A.ptr, P.A.idx, P.A.val64, P.pae,
                                                              ScaledGather{v, 1.0 / length},
                                                              StoreRow<1>{u, -1}, dummy, nullptr, tm.rank);
      tm.sync();
      double nx[1] = {0.0};
      run_phase<1, 1, false, true, kSliceUnroll, false, true>(P.AT.ptr, P.AT.idx, P.AT.val64, P.pate,
                                                              ScaledGather{u, 1.0}, StoreRow<1>{v, 0}, nx,
                                                              nullptr, tm.rank);
      team_part<1, 0u>(ts, 0, nx);
      team_total(ts, tm, 1, 0u);
    }
  }
  const double norm = sqrt(sqrt(ts.total[0]));
  return norm > 0.0 ? norm * 1.01 : 1.0;
}

// The FP32 level's anchor terms (anchor_phases over the FP64 slices).
template <class T>
__device__ __noinline__ void team_anchor(const Prob<T>& P, const State<T>& S, const Team& tm) {
  double dummy[1] = {0.0};
  run_phase<1, 1, false, true, kSliceUnroll, false, true>(P.A.ptr, P.A.idx, P.A.val64, P.pae,
                                                          Gather1<double>{S.xr}, StoreRow<1>{S.axr, -1},
                                                          dummy, nullptr, tm.rank);
  run_phase<1, 1, false, true, kSliceUnroll, false, true>(
      P.AT.ptr, P.AT.idx, P.AT.val64, P.pate, Gather1<double>{S.yr},
      AnchorCol{P.c64, P.cl64, P.cu64, S.xr, S.cg, S.dl, S.du}, dummy, nullptr, tm.rank);
}

constexpr unsigned kTeamEvalMask = (kEvalMaxMask << 2) | (kCertMaxMask << 18) | (kFarkasColMaxMask << 25) |
                                   (3u << 28) | (1u << 30);

// The evaluation's passes over the matrices, each in a function of its own for its registers. Bound by
// L2 latency (index and value, then the pair of candidates): kEvalUnroll entries a lane in flight.
constexpr int kEvalUnroll = 8;
template <class T>
__device__ __noinline__ void eval_rows(const Prob<T>& P, const State<T>& S, TeamShared& ts, const Team& tm) {
  double acc[8];
#pragma unroll
  for (int s = 0; s < 8; ++s) acc[s] = 0.0;
  RowEval<T, 2> re{P.dr, P.rl0, P.ru0, nullptr, nullptr, nullptr, nullptr, S.yc};
  run_phase<2, 8, false, true, kEvalUnroll, true>(P.A.ptr, P.A.idx, P.A.val64, P.pae, GatherPair{S.xc}, re, acc,
                                                  nullptr, tm.rank);
  team_part<8, kEvalMaxMask & 0xffu>(ts, 2, acc);
}
template <class T>
__device__ __noinline__ void eval_columns(const Prob<T>& P, const State<T>& S, TeamShared& ts, const Team& tm) {
  double acc[8];
#pragma unroll
  for (int s = 0; s < 8; ++s) acc[s] = 0.0;
  ColEval<T, 2, 8> ce{P.dc, P.cl0, P.cu0, P.c0, nullptr, nullptr, nullptr, nullptr, nullptr, S.xc};
  run_phase<2, 8, false, true, kEvalUnroll, true>(P.AT.ptr, P.AT.idx, P.AT.val64, P.pate, GatherPair{S.yc}, ce,
                                                  acc, nullptr, tm.rank);
  team_part<8, (kEvalMaxMask >> 8)>(ts, 10, acc);
}
template <class T>
__device__ __noinline__ void eval_certificates(const Prob<T>& P, const State<T>& S, const T* ray_from, int cur,
                                               int prev, TeamShared& ts, const Team& tm) {
  double fk[3] = {0.0, 0.0, 0.0};
  if constexpr (kDelta<T>) {
    run_phase<1, 3, false, true>(P.AT.ptr, P.AT.idx, P.AT.val64, P.pate, Gather1<T>{S.y[cur]},
                                 FarkasCol{P.dc, P.cl0, P.cu0}, fk, nullptr, tm.rank);
  } else {
    run_phase<1, 3, false, true>(P.AT.ptr, P.AT.idx, P.AT.val64, P.pate, DiffGather<T, double>{S.y[cur], S.yr},
                                 FarkasCol{P.dc, P.cl0, P.cu0}, fk, nullptr, tm.rank);
  }
  team_part<3, kFarkasColMaxMask>(ts, 25, fk);
  double rr[2] = {0.0, 0.0};
  run_phase<1, 2, false, true>(P.A.ptr, P.A.idx, P.A.val64, P.pae, DiffGather<T, T>{ray_from, S.x[prev]},
                               RayRow{P.dr, P.rl0, P.ru0}, rr, nullptr, tm.rank);
  team_part<2, 3u>(ts, 28, rr);
}

// One evaluation (evaluate_kernel's steps and slots, one reduction at the end). Slot 30 carries
// rank 0's reading of the clock against the LP's deadline. Leaves c.state at kRunning, a final
// state or a certificate candidate, and ts.flags as evaluate_kernel's.
template <class T>
__device__ __noinline__ void team_evaluate(const Prob<T>& P, const State<T>& S, TeamShared& ts, const Team& tm) {
  Ctrl& c = ts.c;
  const int cur = c.cur, prev = cur_prev_slot(c);
  const bool has_average = c.averaged > 0;
  const double count = (double)c.averaged;
  const bool test_cert = c.farkas_cooldown == 0 && (c.evaluations % kCertEvery) == kCertEvery - 1;
  const bool halpern = c.halpern != 0;
  const T* ray_from = halpern ? S.xt : S.x[cur];
  const int base = tm.rank * kThreads + threadIdx.x, stride = tm.cs * kThreads;
  {
    double mv[2] = {0.0, 0.0};
    double ec[kCertSlots];
#pragma unroll
    for (int s = 0; s < kCertSlots; ++s) ec[s] = 0.0;
    for (int j = base; j < P.n; j += stride) {
      const double xo = ld(S.x[cur] + j);
      double second = 0.0;
      if (halpern) {
        second = ld(S.xt + j);
      } else {
        const double xs = S.xsum[j] + (c.pending ? xo : 0.0);
        S.xsum[j] = xs;
        second = xs / count;
      }
      const double r = S.xr[j];
      const double d = kDelta<T> ? xo : xo - r;
      S.xc[j] = kDelta<T> ? make_double2(r + xo, has_average ? r + second : 0.0)
                          : make_double2(xo, has_average ? second : 0.0);
      mv[0] += d * d;
      if (test_cert) {
        const double t = __ldg(P.dc + j) * (ld(ray_from + j) - ld(S.x[prev] + j));
        ray_col_terms(t, __ldg(P.cl0 + j), __ldg(P.cu0 + j), __ldg(P.c0 + j), ec);
      }
    }
    for (int i = base; i < P.m; i += stride) {
      const double yo = ld(S.y[cur] + i);
      double second = 0.0;
      if (halpern) {
        second = ld(S.yt + i);
      } else {
        const double ys = S.ysum[i] + (c.pending ? yo : 0.0);
        S.ysum[i] = ys;
        second = ys / count;
      }
      const double r = S.yr[i];
      const double d = kDelta<T> ? yo : yo - r;
      S.yc[i] = kDelta<T> ? make_double2(r + yo, has_average ? r + second : 0.0)
                          : make_double2(yo, has_average ? second : 0.0);
      mv[1] += d * d;
      if (test_cert) farkas_row_terms(-__ldg(P.dr + i) * d, __ldg(P.rl0 + i), __ldg(P.ru0 + i), ec);
    }
    team_part<2, 0u>(ts, 0, mv);
    if (test_cert) team_part<kCertSlots, kCertMaxMask>(ts, 18, ec);
  }
  tm.sync();
  SIH26_TEAM_MARK(12);
  eval_rows(P, S, ts, tm);
  eval_columns(P, S, ts, tm);
  if (test_cert) {
    eval_certificates(P, S, ray_from, cur, prev, ts, tm);
  } else if ((threadIdx.x & 31) == 0) {
    for (int s = 18; s < 30; ++s) ts.warp[threadIdx.x >> 5][s] = 0.0;
  }
  if ((threadIdx.x & 31) == 0)
    ts.warp[threadIdx.x >> 5][30] =
        tm.rank == 0 && threadIdx.x == 0 && c.deadline_ns != 0ull && global_ns() > c.deadline_ns ? 1.0 : 0.0;
  SIH26_TEAM_MARK(13);
  team_total(ts, tm, kTeamSlots, kTeamEvalMask);
  SIH26_TEAM_MARK(14);
  // every block takes the same decisions from the same totals
  if (threadIdx.x == 0) {
    ts.before = c;
    double mv[2], t[kEvalSlots];
    for (int s = 0; s < 2; ++s) mv[s] = ts.total[s];
    for (int s = 0; s < kEvalSlots; ++s) t[s] = ts.total[2 + s];
    evaluation_decision(c, t, mv, has_average, ts.flags);
    ts.flags[3] = 0;
    if (c.farkas_cooldown > 0) --c.farkas_cooldown;
    if (test_cert && c.state != kConverged) {
      double ec[kCertSlots], fk[3], rr[2];
      for (int s = 0; s < kCertSlots; ++s) ec[s] = ts.total[18 + s];
      for (int s = 0; s < 3; ++s) fk[s] = ts.total[25 + s];
      for (int s = 0; s < 2; ++s) rr[s] = ts.total[28 + s];
      const int kind = certificate_test(c, ec, fk, rr);
      if (kind != 0) {
        // keep the restart anchor and step state: the certificate is read from them, and the
        // LP resumes from them if the host turns it down
        const double margin = c.farkas_margin;
        c = ts.before;
        ++c.evaluations;
        c.pending = 0;
        c.farkas_margin = margin;
        c.state = kind == 1 ? kInfeasible : kUnbounded;
        ts.flags[0] = ts.flags[1] = ts.flags[2] = 0;
        ts.flags[3] = kind;
      }
    }
    if (c.state == kRunning && ts.total[30] > 0.0) c.state = kTimeLimit;
  }
  __syncthreads();
  const int best = ts.flags[0], restart = ts.flags[1], average = ts.flags[2], kind = ts.flags[3];
  const double scale = kind == 1 ? ts.total[19] : ts.total[21];
  if (best || restart || kind) {
    for (int j = base; j < P.n; j += stride) {
      const double2 xcj = S.xc[j];
      if (kind == 2) S.cert_col[j] = __ldg(P.dc + j) * (ld(ray_from + j) - ld(S.x[prev] + j)) / scale;
      if (best) S.best_x[j] = average ? xcj.y : xcj.x;
      if (restart) {
        S.xr[j] = xcj.x;
        S.xsum[j] = 0.0;
        if constexpr (kDelta<T>) S.x[cur][j] = T(0);
      }
    }
    for (int i = base; i < P.m; i += stride) {
      const double2 yci = S.yc[i];
      if (kind == 1) {
        const double d = kDelta<T> ? ld(S.y[cur] + i) : ld(S.y[cur] + i) - ld(S.yr + i);
        S.cert_row[i] = -__ldg(P.dr + i) * d / scale;
      }
      if (best) S.best_y[i] = average ? yci.y : yci.x;
      if (restart) {
        S.yr[i] = yci.x;
        S.ysum[i] = 0.0;
        if constexpr (kDelta<T>) {
          S.y[cur][i] = T(0);
          S.ax[cur][i] = 0.0;
        } else {
          if (halpern) S.axr[i] = S.ax[cur][i];  // A x_0 of the new restart point
        }
      }
    }
  }
  tm.sync();
  if constexpr (kDelta<T>) {
    // a restart moved the anchor: form its terms
    if (restart) {
      team_anchor(P, S, tm);
      tm.sync();
    }
  }
}

// Report of one finished LP (report_kernel's, pdhg.cpp:647-661): unscaled point, reduced costs,
// multipliers, the residual block of the best point into c.best and the quality slots.
template <class T>
__device__ __noinline__ void team_report(const Prob<T>& P, const State<T>& S, double* x_out, double* red_out,
                                         double* y_out, TeamShared& ts, const Team& tm) {
  Ctrl& c = ts.c;
  tm.sync();  // the totals of the last evaluation have been read in every block
  {
    double acc[kEvalSlots];
#pragma unroll
    for (int s = 0; s < kEvalSlots; ++s) acc[s] = 0.0;
    RowEval<T, 1> re{P.dr, P.rl0, P.ru0, nullptr, nullptr, S.best_y, y_out};
    run_phase<1, kEvalSlots, false, true, kSliceUnroll, true, true>(
        P.A.ptr, P.A.idx, P.A.val64, P.pae, Gather1<double>{S.best_x}, re, acc, nullptr, tm.rank);
    ColEval<T, 1> ce{P.dc, P.cl0, P.cu0, P.c0, nullptr, nullptr, S.best_x, x_out, red_out};
    run_phase<1, kEvalSlots, false, true, kSliceUnroll, true, true>(
        P.AT.ptr, P.AT.idx, P.AT.val64, P.pate, Gather1<double>{S.best_y}, ce, acc, nullptr, tm.rank);
    team_part<kEvalSlots, kReportMaxMask>(ts, 0, acc);
  }
  team_total(ts, tm, kEvalSlots, kReportMaxMask);  // and orders the outputs' writes
  if (threadIdx.x == 0) {
    double t[kEvalSlots];
    for (int s = 0; s < kEvalSlots; ++s) t[s] = ts.total[s];
    c.best = make_residuals(t, 0, c.bound_norm, c.cost_norm);
    c.primal_violation = dmax(0.0, dmax(t[1], t[9]));
  }
  double qv[kQualitySlots];
#pragma unroll
  for (int k = 0; k < kQualitySlots; ++k) qv[k] = 0.0;
  quality_pass(P, S.best_x, S.best_y, x_out, y_out, red_out, tm.rank * kWarps + (int)(threadIdx.x >> 5),
               tm.cs * kWarps, qv);
  team_part<kQualitySlots, 0xFFu>(ts, 0, qv);
  tm.sync();
  team_total(ts, tm, kQualitySlots, 0xFFu);
  if (threadIdx.x < kQualitySlots) c.quality[threadIdx.x] = ts.total[threadIdx.x];
  __syncthreads();
}

// ---- one LP on one team ---------------------------------------------------------------------------

// A section's device time, by thread 0 of rank 0, whose control block goes back. Out of line: in the caller's
// registers the clock cost the FP64 loop 0.2 us an iteration (2,000 x 5,000, Halpern: 5.68 and 5.89).
static __device__ __noinline__ void section_begins(TeamShared& ts, const Team& tm) {
  if (threadIdx.x == 0 && tm.rank == 0) ts.section_start = global_ns();
}
static __device__ __noinline__ void section_ends(TeamShared& ts, const Team& tm, unsigned long long Ctrl::*total) {
  if (threadIdx.x == 0 && tm.rank == 0) ts.c.*total += global_ns() - ts.section_start;
}

// Runs the LP from its stored state: to a final state, `max_evaluations` evaluations or
// `max_attempts` attempts, whichever comes first. A final state comes with its report. kHalpern:
// 1 / 0 for an LP of that operator alone, -1 for either (the batched engine). kOnlyL2: for LPs gathered out of
// L2 alone.
template <class T, int kHalpern, bool kOnlyL2 = false>
__device__ __forceinline__ void team_solve(const Prob<T>& P, const State<T>& S, const ResidentPlan& pl,
                                           const ResidentPlan& pl64, double* x_out, double* red_out, double* y_out,
                                           TeamShared& ts, SideView<T>& sp, SideView<T>& sd, SideView<double>& sp64,
                                           SideView<double>& sd64, const Team& tm,
                                           long long max_attempts, int max_evaluations) {
  constexpr bool kStreams = kHalpern < 0;
  Ctrl& c = ts.c;
  if (threadIdx.x == 0) c = *S.ctrl;
  if constexpr (kHalpern >= 0) section_begins(ts, tm);
  tm.sync();  // every block has started: its shared memory may be written
  const bool setup = c.state == kSetup;
  SIH26_TEAM_MARK(-1);
  const bool halpern = kHalpern >= 0 ? kHalpern != 0 : c.halpern != 0;
  const bool outside = kOnlyL2 || (kHalpern < 0 && pl.outside != kInside);
  const bool turns = !kOnlyL2 && outside && pl.outside == kInTurns;
  if (c.state == kSetup) {
    SIH26_TEAM_MARK(7);
    if (pl64.cs > 0 && !outside) {
      load_side(sp64, pl64.side[0], Csr<double>{P.AT.ptr, P.AT.idx, P.AT.val64, P.AT.val64}, P.pate, P.pate, tm.rank);
      load_side(sd64, pl64.side[1], Csr<double>{P.A.ptr, P.A.idx, P.A.val64, P.A.val64}, P.pae, P.pae, tm.rank);
    }
    double norm;
    const int nnz = __ldg(P.A.ptr + P.m);
    if constexpr (kHalpern < 0) {
      norm = turns     ? vector_setup<true>(P, S, nnz, ts, tm)
             : outside ? vector_setup<false>(P, S, nnz, ts, tm)
                       : team_power<T, kStreams || kDelta<T>>(P, S, nnz, pl64, sp64, sd64, ts, tm);
    } else {
      norm = team_power<T, kStreams || kDelta<T>>(P, S, nnz, pl64, sp64, sd64, ts, tm);
    }
    if (threadIdx.x == 0) {
      c.spectral_norm = norm;
      c.eta = norm > 0.0 ? 1.0 / norm : 1.0;
      if (halpern) c.eta = 0.998 / dmax(norm, 1e-12);  // constant: tau sigma ||A||^2 < 1
      c.eta_ceiling = 1.0e3 / dmax(norm, 1e-12);
    }
    SIH26_TEAM_MARK(8);
    if constexpr (kDelta<T>) team_anchor(P, S, tm);
    tm.sync();
  }
  SIH26_TEAM_MARK(9);
  const bool resident = !outside;
  if (outside && c.state == kSetup) {
    __syncthreads();
    if (threadIdx.x == 0) c.state = kRunning;
    tm.sync();
  }
  if (resident && (c.state == kSetup || c.state == kRunning)) {
    tm.sync();  // no block still stores the norm estimate's vectors into this one's memory
    if (kDelta<T> || c.state == kRunning) {
      load_side(sp, pl.side[0], P.AT, P.pati, P.pate, tm.rank);
      load_side(sd, pl.side[1], P.A, P.pai, P.pae, tm.rank);
    }
    load_vectors(P, S, pl, c.cur);
    __syncthreads();
    if (c.state == kSetup) {
      if constexpr (!kDelta<T>) {
        // A x_0 with the iteration's sums; also the Halpern anchor's
        TeamStoreAx st{S.ax[c.cur], S.axr};
        side_phase<kStreams>(sd, reinterpret_cast<const T*>(team_memory() + pl.x[c.cur]), st);
        __syncthreads();
      }
      if (threadIdx.x == 0) c.state = kRunning;
    }
    load_epilogues(P, S, sp, sd, halpern, c.cur);
    tm.sync();
  }
  SIH26_TEAM_MARK(10);
  if constexpr (kHalpern >= 0) {
    if (setup) section_ends(ts, tm, &Ctrl::setup_ns);
  }
  long long left = max_attempts;
  int evaluations = max_evaluations;
  while (c.state == kRunning) {
    // loop top (pdhg.cpp:384-385)
    if (c.iteration >= c.iteration_limit || c.time_up) {
      __syncthreads();
      if (threadIdx.x == 0) c.state = c.iteration >= c.iteration_limit ? kIterationLimit : kTimeLimit;
      __syncthreads();
      break;
    }
    if (left <= 0 || evaluations <= 0) break;
    SIH26_TEAM_MARK(6);
    if (halpern) {
      long long steps = 40 - c.iteration % 40;
      if (steps > c.iteration_limit - c.iteration) steps = c.iteration_limit - c.iteration;
      if (steps > left) steps = left;
      if (resident) {
        team_halpern<T, kStreams>(S, pl, sp, sd, ts, tm, static_cast<int>(steps));
      } else {
        if constexpr (kHalpern < 0) {
          if (turns) vector_halpern<true>(P, S, ts, tm, static_cast<int>(steps));
          else vector_halpern<false>(P, S, ts, tm, static_cast<int>(steps));
        }
      }
      left -= steps;
    } else {
      do {
        if (resident) {
          team_attempt<T, kStreams>(pl, sp, sd, ts, tm);
        } else {
          if constexpr (kHalpern < 0) {
            if (turns) vector_attempt<true>(P, S, ts, tm);
            else vector_attempt<false>(P, S, ts, tm);
          }
        }
        --left;
      } while (c.state == kRunning && left > 0 && c.iteration < c.iteration_limit);
      if (resident) spill(S, pl, sp, sd, c);
      tm.sync();
    }
    if (c.state == kNeedEval) {
      SIH26_TEAM_MARK(4);
      if constexpr (kHalpern >= 0) section_begins(ts, tm);
      team_evaluate(P, S, ts, tm);
      if constexpr (kHalpern >= 0) section_ends(ts, tm, &Ctrl::evaluate_ns);
      SIH26_TEAM_MARK(5);
      --evaluations;
      if (resident && c.state == kRunning) {
        const bool refill = kDelta<T> && ts.flags[1] != 0;  // the same in every block
        if (refill) load_vectors(P, S, pl, c.cur);
        if (ts.flags[1] || !halpern) load_epilogues(P, S, sp, sd, halpern, c.cur);
        // The Halpern operator's next step stores into every block's only copy of x: not before they have all
        // been refilled, or a block that is behind writes the restart's zeros over a new entry. Some 500
        // cycles a restart.
        if (refill) tm.sync();
        else __syncthreads();
      }
    }
  }
  if (c.state == kConverged || c.state == kIterationLimit || c.state == kTimeLimit || c.state == kInfeasible ||
      c.state == kUnbounded) {
    if constexpr (kHalpern >= 0) section_begins(ts, tm);
    team_report(P, S, x_out, red_out, y_out, ts, tm);
    if constexpr (kHalpern >= 0) section_ends(ts, tm, &Ctrl::report_ns);
  }
  SIH26_TEAM_MARK(11);
  if (threadIdx.x == 0 && tm.rank == 0) *S.ctrl = c;
  tm.sync();
}

// The single-LP path's kernel: one cluster, one LP.
template <class T, bool kHalpern>
__global__ void __launch_bounds__(kThreads, 1)
    resident_kernel(const __grid_constant__ Prob<T> P, const __grid_constant__ State<T> S,
                    const __grid_constant__ ResidentPlan pl, const __grid_constant__ ResidentPlan pl64,
                    double* x_out, double* red_out, double* y_out, long long max_attempts, int max_evaluations) {
  __shared__ TeamShared ts;
  __shared__ SideView<T> sp, sd;
  // the norm estimate's FP64 view: the FP64 level's own, or before the FP32 level loads its
  __shared__ SideView<double> other[2];
  SideView<double>*sp64 = other, *sd64 = other + 1;
  if constexpr (!kDelta<T>) {
    sp64 = &sp;
    sd64 = &sd;
  }
  const Team tm{pl.cs, pl.cs > 1 ? (int)cooperative_groups::this_cluster().block_rank() : 0};
  team_solve<T, kHalpern ? 1 : 0>(P, S, pl, pl64, x_out, red_out, y_out, ts, sp, sd, *sp64, *sd64, tm,
                                  max_attempts, max_evaluations);
}

}  // namespace sih26
