// Host check of csrc/bailout.h: r2 > largest_square(b) == sqrt(r2) > b for
// the squares next to the edge, random squares, zero, infinity and NaN,
// over bailouts of every magnitude.  Prints the number of mismatches and of
// comparisons.
#include <stdio.h>

#include "bailout.h"

static unsigned long long rng = 0x9E3779B97F4A7C15ull;
static unsigned long long next() {
  rng ^= rng << 13;
  rng ^= rng >> 7;
  rng ^= rng << 17;
  return rng;
}

template <class T>
static void check(T b, long long &bad, long long &n) {
  const T inf = std::numeric_limits<T>::infinity();
  const T x = mbr::largest_square(b);
  const auto one = [&](T r2) {
    volatile T root = std::sqrt(r2);
    bad += (root > b) != (r2 > x);
    n++;
  };
  T up = x < T(0) ? T(0) : x, down = up;
  for (int k = 0; k < 64; k++) {
    one(up);
    one(down);
    up = std::nextafter(up, inf);
    down = std::nextafter(down, T(0));
  }
  for (int k = 0; k < 64; k++) one(std::fabs(x) * T(0.5 + double(next() >> 11) * 0x1p-53));
  one(T(0));
  one(inf);
  one(std::numeric_limits<T>::max());
  one(std::numeric_limits<T>::denorm_min());
  one(std::numeric_limits<T>::quiet_NaN());
}

int main() {
  long long bad = 0, n = 0;
  const double some[] = {0.0, -1.0, 1e-320, 1e-160, 0.1, 1.0, 2.0, 10.0, 100.0, 1e19, 1e20, 1e38, 3.4e38, 1e154, 1.5e154,
                         1e300, 1.7e308, std::numeric_limits<double>::infinity()};
  for (double b : some) {
    check<double>(b, bad, n);
    check<float>(float(b), bad, n);
  }
  for (int k = 0; k < 20000; k++) {
    const double b = std::ldexp(1.0 + double(next() >> 11) * 0x1p-53, int(next() % 120) - 60);
    check<double>(b, bad, n);
    check<float>(float(b), bad, n);
  }
  printf("%lld %lld\n", bad, n);
  return bad != 0;
}
