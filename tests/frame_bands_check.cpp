// Host check of csrc/frame_bands.h: over frames of every height, limits and
// amounts of memory that can be had, the band fits the limit and the memory or
// is the smallest, and is as large as they allow up to halving.  Prints the
// number of wrong answers and of cases.
#include <stdio.h>

#include "frame_bands.h"

int main() {
  long long bad = 0, n = 0;
  const int heights[] = {1, 2, 3, 4, 5, 7, 8, 9, 63, 64, 65, 1080, 2160, 5121};
  for (int rows : heights)
    for (size_t per_row : {size_t(84), size_t(1000), size_t(4096) * 596})
      for (size_t limit : {size_t(1), per_row * 4, per_row * 5 + 256, per_row * 64 + 256, per_row * 1001, per_row * 100000})
        for (size_t memory : {size_t(0), per_row * 4 + 256, per_row * 9 + 256, per_row * 300 + 256, per_row * 100000}) {
          int tries = 0;
          size_t got = 0;
          static char somewhere;
          const auto bytes = [&](int r) { return 256 + per_row * size_t(r); };
          const mbr::FrameBands b = mbr::frame_bands(rows, limit, bytes, [&](size_t want) {
            tries++;
            if (want > memory) return static_cast<void *>(nullptr);
            got = want;
            return static_cast<void *>(&somewhere);
          });
          const int least = rows < 4 ? rows : 4;
          bool ok = b.rows >= least && b.rows <= rows && (b.rows == rows || b.rows % 4 == 0) && tries < 20;
          if (b.rows > least) ok = ok && bytes(b.rows) <= limit;
          ok = ok && (b.scratch != nullptr) == (bytes(least) <= memory);
          if (b.scratch) ok = ok && got == bytes(b.rows);
          if (bytes(rows) <= limit && bytes(rows) <= memory) ok = ok && b.rows == rows;
          if (b.rows < rows) ok = ok && (bytes(b.rows + 4) > limit || bytes(2 * b.rows + 8) > memory);
          bad += !ok;
          n++;
        }
  printf("%lld %lld\n", bad, n);
  return bad != 0;
}
