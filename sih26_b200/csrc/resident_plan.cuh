// Where an LP's vectors and matrix sit in the shared memory of the cluster that solves it (resident.cuh).
// Host code.
#pragma once

#include <algorithm>
#include <vector>

#include "pdhg_host.cuh"

namespace sih26 {

constexpr int kMaxTeam = 16;                  // blocks of the largest cluster
constexpr int kResidentBytes = 212 * 1024;    // dynamic shared memory a plan may take (the kernels hold 12 KB more)
constexpr int kWholeVector = kResidentBytes / 8;  // FP64 entries of a vector that fits alone

// Where everything sits in a block's dynamic shared memory (bytes; the same in every block of
// the cluster, sized for the block with the most of each). side[0]: rows of A' (phase P),
// side[1]: rows of A (phase D).
struct ResidentPlan {
  int cs;      // blocks of the cluster; 0: the LP has no plan
  int bytes;
  int outside;         // how an LP whose vectors do not fit beside each other is solved: below
  int x[2], y[2];      // equal: one buffer (the Halpern operator always accepts its step)
  struct Side {
    int resident;      // the entries are in shared memory too
    int items, segs, longs, seg_sum, len, gptr, epi, idx, val;
    int stride;        // slots: length of each epilogue array
  } side[2];
};

// Epilogue arrays of the plan's two sides (see above).
__host__ __device__ constexpr int team_column_arrays() { return 4; }
__host__ __device__ constexpr int team_row_arrays(bool halpern, bool delta) {
  return halpern ? 4 : (delta ? 7 : 5);
}

// The plan of an LP over the blocks of its two partitions (pat: rows of A', pa: rows of A, both
// sliced). value_bytes: of the level. `streams`: a side whose entries do not fit may stay in global
// memory. cs = 0 when the LP does not fit, which 65,536 rows or columns (16-bit indices) already
// decide.
inline ResidentPlan plan_resident(int m, int n, const std::vector<int>& at_ptr, const std::vector<int>& a_ptr,
                                  const HostPart& pat, const HostPart& pa, int cs, int value_bytes, bool halpern,
                                  bool streams) {
  ResidentPlan pl{};
  if (m > 65536 || n > 65536) return pl;
  long long bytes = 0;
  const auto put = [&](long long count, int size) {
    const long long at = bytes;
    bytes += (count * size + 15) & ~15ll;
    return static_cast<int>(std::min<long long>(at, 1 << 30));
  };
  for (int k = 0; k < 2; ++k) {
    if (k == 1 && halpern) {
      pl.x[1] = pl.x[0];
      pl.y[1] = pl.y[0];
    } else {
      pl.x[k] = put(n, value_bytes);
      pl.y[k] = put(m, value_bytes);
    }
  }
  long long entries[2] = {0, 0};
  for (int o = 0; o < 2; ++o) {
    const HostPart& hp = o == 0 ? pat : pa;
    const std::vector<int>& ptr = o == 0 ? at_ptr : a_ptr;
    long long items = 0, segs = 0, longs = 0, slots = 0;
    for (int b = 0; b < cs; ++b) {
      long long sl = hp.blk_long_begin[b + 1] - hp.blk_long_begin[b], en = 0;
      for (int q = hp.blk_seg_begin[b]; q < hp.blk_seg_begin[b + 1]; ++q) en += hp.segs[q].z - hp.segs[q].y;
      for (int q = hp.blk_item_begin[b]; q < hp.blk_item_begin[b + 1]; ++q) {
        const int4& it = hp.items[q];
        sl += it.y - it.x;
        en += it.z < 0 ? 32ll * -it.z : ptr[it.y] - ptr[it.x];
      }
      items = std::max<long long>(items, hp.blk_item_begin[b + 1] - hp.blk_item_begin[b]);
      segs = std::max<long long>(segs, hp.blk_seg_begin[b + 1] - hp.blk_seg_begin[b]);
      longs = std::max<long long>(longs, hp.blk_long_begin[b + 1] - hp.blk_long_begin[b]);
      slots = std::max(slots, sl);
      entries[o] = std::max(entries[o], en);
    }
    ResidentPlan::Side& s = pl.side[o];
    s.items = put(items, 16);
    s.segs = put(segs, 16);
    s.longs = put(longs, 16);
    s.seg_sum = put(segs, 8);
    s.len = put(slots, 2);
    s.gptr = put(slots, 4);
    s.stride = static_cast<int>(slots);
    s.epi = put(slots * (o == 0 ? team_column_arrays() : team_row_arrays(halpern, value_bytes == 4)), 8);
  }
  for (int o = 0; o < 2; ++o) {
    ResidentPlan::Side& s = pl.side[o];
    const long long before = bytes;
    s.idx = put(entries[o], 2);
    s.val = put(entries[o], value_bytes);
    s.resident = bytes <= kResidentBytes ? 1 : 0;
    if (!s.resident) {
      if (!streams) return pl;
      bytes = before;
    }
  }
  if (bytes > kResidentBytes) return pl;
  pl.cs = cs;
  pl.bytes = static_cast<int>(bytes);
  return pl;
}

// An LP whose vectors do not fit beside each other keeps its state in global memory.
enum {
  kInside = 0,
  kInTurns = 1,  // the gathered vector is copied into shared memory, x and y in turn (turn_phase)
  kFromL2 = 2    // its entries are gathered out of L2, in a launch without dynamic shared memory
};

// The plan of such an LP: in turns while either vector fits alone. FP64, us per Halpern iteration of one LP on
// 8 blocks, and of each of 36 at once, in turns and from L2: 9,000 x 20,000 with 160,000 nonzeros 27 and 18-25,
// 2.3 and 3.8. Longer vectors in pieces that fit were measured too, and lose: 20,000 x 50,000 with 450,000
// nonzeros in two pieces 83 and 74 from L2, 11.8 and 8.1 at once; 100,000 x 250,000 with 2.5 million in ten 1,051
// and 519, 136 and 50; 1,000,000 x 2,500,000 with 10 million in 93 alone 64,831 and 2,834.
inline ResidentPlan plan_outside(int m, int n, int cs) {
  ResidentPlan pl{};
  pl.cs = cs;
  pl.outside = std::max(m, n) <= kWholeVector ? kInTurns : kFromL2;
  pl.bytes = pl.outside == kInTurns ? kResidentBytes : 0;
  return pl;
}

}  // namespace sih26
