// bailout.h - the bailout test |z| > b without the square root.
//
// The square root is correctly rounded on the host and on the device, hence
// monotonic: there is a largest value X with sqrt(X) <= b, and for every r2
// (infinities and NaN included) sqrt(r2) > b exactly when r2 > X.  An orbit
// loop can then compare |z|^2 with X and take the root once, when the orbit
// ends; the iteration counts are those of the test on |z|.
#pragma once
#include <cmath>
#include <limits>

namespace mbr {

template <class T>
inline T largest_square(T b) {
  const T inf = std::numeric_limits<T>::infinity();
  if (b != b || b == inf) return inf;  // no |z| lies above
  if (b < T(0)) return T(-1);          // every |z| lies above
  T x = b * b;
  if (!(x < inf)) return std::numeric_limits<T>::max();  // finite squares have roots below such a b
  while (std::sqrt(x) > b) x = std::nextafter(x, T(0));
  for (T up = std::nextafter(x, inf); std::sqrt(up) <= b; up = std::nextafter(x, inf)) x = up;
  return x;
}

}  // namespace mbr
