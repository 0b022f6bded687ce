// Walking a range of entries in chunks, for ranges that end anywhere up to 2^31 - 1.
#pragma once

namespace sih26 {

// Where the chunk of at most kSize entries that begins at `at` ends; the next one begins there. at < last.
// Stepping by kSize instead passes 2^31 - 1 behind the last chunk of such a range and goes on at negative
// positions.
template <int kSize>
#ifdef __CUDACC__
__host__ __device__ __forceinline__
#else
inline
#endif
    int
    chunk_end(int at, int last) {
  return last - at > kSize ? at + kSize : last;
}

}  // namespace sih26
