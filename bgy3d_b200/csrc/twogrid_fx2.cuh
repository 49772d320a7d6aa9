// twogrid_fx2.cuh -- launchers of the x-axis grid transfers that run both
// sides by FFT (k_restrict_fx2 / k_prolong_fx2 of twogrid_fft.cuh), one struct
// per fine half row M over the coarse half rows MC that the coarse-grid rule
// can pair with it: pairs without a kernel fall back to the (K+1) x Nc table
// product (fine rows of the older shapes) or the dense tiles, at 162 -> 54
// points 107 us per restriction and 153 us per prolongation against 34 and 63
// here.  Instantiated by the twogrid_fx2*.cu translation units.
#pragma once
#include <cuda_runtime.h>

namespace rism {

// Fine half rows with these transfers.
#define RISM_FX2_LENS(X)                                                                                      \
  X(24) X(27) X(32) X(36) X(48) X(54) X(64) X(72) X(81) X(96) X(108) X(128) X(144) X(162) X(192) X(216) X(243) \
  X(256)
#define RISM_FX2_COARSE(X) X(16) X(18) X(24) X(27) X(32) X(36) X(48) X(54) X(64) X(128)

// Spacings of 0.75 or 1 A on the coarse side and 0.16 A and more on the fine
// one: ratios of 1.3 to 4.6 (a 256-point coarse axis under 512 points only).
constexpr bool fx2_pair(int M, int MC) {
  return MC == 128 ? M == 256 : 13 * MC <= 10 * M && 10 * M <= 46 * MC;
}

template <int M> struct Fx2 {
  template <typename T>
  static bool restrict_x(int MC, long long rows, const T *in, float s, const float2 *post, const float2 *tw,
                         const float2 *postc, const float2 *twc, float *out, cudaStream_t st);
  template <typename T>
  static bool prolong_x(int MC, long long rows, const float *y, const float2 *post, const float2 *tw,
                        const float2 *postc, const float2 *twc, const T *r, double s, T *out, cudaStream_t st);
};

}  // namespace rism
