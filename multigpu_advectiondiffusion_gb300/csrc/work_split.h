// work_split.h -- how a launch's (tile, z-plane) pairs, tile-major, are shared among its CTAs.
#pragma once
#include <algorithm>
#include <cstdint>

namespace adv {

// `parts` shares of every group of pairs (all of them, or one tile's planes): each = pairs / parts, one
// more for the first `extra` shares, with the divisions made on the host (a 64-bit division costs every
// thread about 100 instructions). The longer shares come first, so that consecutive CTAs, which go to
// different SMs, take them; spread evenly they alternated, and with an even number of SMs half the SMs got
// all of them (heat FP64 O4 128^3: 314 -> 292 us per step; FP32 O2 128^3: 5.6 -> 5.1, 192^3: 11.4 -> 10.4).
struct WorkSplit {
  int64_t each = 0;
  unsigned extra = 0, parts = 1;
  unsigned ctas = 1;  // parts times the groups
  unsigned ratio = 1u << 31;  // of longer shares among the first CTAs, times 2^31 (split_range_whole)
};

// At most `most` CTAs (one wave, or a few) of at least min_share planes for `tiles` tiles of nz planes. A
// share that crosses into the next tile starts a second segment, whose halo planes cost as much as
// `restart` planes; shares cut tile by tile cross none but cannot use every CTA slot. The cheaper of the two
// by that count (Burgers FP32 128^3: 41.3 -> 38.4 us per stage tile by tile, adjoint 96^3: 50.6 -> 45.1; but
// FP64 121 x 101 x 97, where a segment's start costs little: 2369 -> 2617).
inline WorkSplit work_split(int64_t tiles, int nz, int64_t most, int64_t min_share, double restart) {
  const int64_t total = tiles * nz;
  most = std::max<int64_t>(1, std::min<int64_t>(most, total / min_share));
  const int64_t c = std::min<int64_t>(most / tiles, std::max<int64_t>(1, nz / min_share));
  const bool by_tile = c >= 1 && (double)((nz + c - 1) / c) + restart < (double)((total + most - 1) / most) + 2 * restart;
  const int64_t pairs = by_tile ? nz : total, parts = by_tile ? c : most;
  WorkSplit w;
  w.each = pairs / parts;
  w.extra = (unsigned)(pairs % parts);
  w.parts = (unsigned)parts;
  w.ctas = (unsigned)(by_tile ? tiles * c : most);
  return w;
}

}  // namespace adv
