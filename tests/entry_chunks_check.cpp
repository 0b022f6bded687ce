// The residual check's walk over a column range's entries (sih26_b200/csrc/entry_chunks.cuh): contiguous chunks
// of at most the chunk's size that cover the range and end with it, up to 2^31 - 1. Built with -ftrapv.
#include <climits>
#include <cstdio>
#include <initializer_list>

#include "entry_chunks.cuh"

int main() {
  const int ends[] = {1, 127, 128, 129, 1000, INT_MAX - 129, INT_MAX - 128, INT_MAX - 1, INT_MAX};
  for (int last : ends)
    for (int length : {1, 5, 127, 128, 129, 256, 700}) {
      const int first = last > length ? last - length : 0;
      int at = first, chunks = 0;
      while (at < last) {
        const int end = sih26::chunk_end<128>(at, last);
        if (end <= at || end > last || end - at > 128 || (end < last && end - at != 128) || ++chunks > 8) {
          std::printf("range [%d, %d): chunk [%d, %d)\n", first, last, at, end);
          return 1;
        }
        at = end;
      }
    }
  std::puts("ok");
  return 0;
}
