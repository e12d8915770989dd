// heatk_rows.h -- where the rows around a thread's nodes lie in the heat-with-k(x) kernels, in elements.
#pragma once

#ifdef __CUDACC__
#define ADV_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define ADV_HOST_DEVICE inline
#endif

namespace adv {

// Offsets from the thread's first row y: its rows (those past the grid: the last one), and the rows y-1 and
// y+RY beside them (clamped to its own first / last). 32 bits hold them for the rows of up to 2^30 nodes that the
// solver accepts, the row below two rows only without a sign (64-bit offsets would spill the FP32 adjoint, at 126
// registers of 128).
template <int RY>
struct HeatKRows {
  static_assert(RY <= 2, "a row of 2^30 nodes: dr fits an int, below an unsigned");
  int dr[RY];
  int above;
  unsigned below;
  ADV_HOST_DEVICE void set(int y, int nx, int ny) {
    auto row = [&](int r) { return (unsigned)(y + r < ny ? r : ny - 1 - y) * (unsigned)nx; };
    for (int r = 0; r < RY; ++r) dr[r] = (int)row(r);
    above = y > 0 ? -nx : 0;
    below = row(RY);
  }
};

}  // namespace adv
