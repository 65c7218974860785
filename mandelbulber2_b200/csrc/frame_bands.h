// frame_bands.h - the bands of rows in which a staged plain frame is rendered,
// one after another over one scratch, so that a frame of any size needs at most
// `limit` bytes (the scratch of a whole frame grows with its AO rays: 3840x2160
// with 64 rays takes 4.9 GB).  A band's pixels come out as the whole frame's do.
#pragma once
#include <stddef.h>

#include <algorithm>

namespace mbr {

struct FrameBands {
  void *scratch;  // null: not even the smallest band's could be had
  int rows;       // rows per band, a multiple of 4 (a row of the stages' 8x4 tiles) unless it is all
};

// bytes(r): the scratch of a band of r rows, increasing with r; alloc(b): b
// bytes or null.  Tries the largest band within the limit, then smaller ones.
template <class Bytes, class Alloc>
FrameBands frame_bands(int rows, size_t limit, Bytes bytes, Alloc alloc) {
  int band = rows;
  while (band > 4 && bytes(band) > limit) {
    const double share = double(limit) / double(bytes(band));
    band = std::max(4, std::min(band - 1, int(band * share)) / 4 * 4);
  }
  for (;;) {
    void *p = alloc(bytes(band));
    if (p || band <= 4) return {p, band};
    band = std::max(4, band / 8 * 4);
  }
}

}  // namespace mbr
