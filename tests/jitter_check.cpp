// Host check of csrc/jitter.h: tenthousandths(k) == k / 10000.0 for every draw
// k = 0 .. 1000 of the march jitter.  Prints the number of mismatches.
#include <stdio.h>

#include "jitter.h"

int main() {
  int bad = 0;
  for (int k = 0; k <= 1000; k++) {
    volatile double d = double(k), n = 10000.0;
    bad += mbr::tenthousandths(k) != d / n;
  }
  printf("%d\n", bad);
  return bad != 0;
}
