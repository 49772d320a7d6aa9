// twogrid_fx2_impl.cuh -- definitions of twogrid_fx2.cuh.
#pragma once
#include "twogrid_fft.cuh"
#include "twogrid_fx2.cuh"

namespace rism {

namespace {

template <typename T, int M, int MC>
bool run_restrict(long long rows, const T *in, float s, const float2 *post, const float2 *tw, const float2 *postc,
                  const float2 *twc, float *out, cudaStream_t st) {
  constexpr int RX = x_rx<T, M>();
  static_assert(fx2_smem<M, MC, RX>() <= 48 * 1024, "no opt-in needed");
  k_restrict_fx2<T, M, MC, RX>
      <<<(unsigned)((rows + RX - 1) / RX), kFx2Threads, fx2_smem<M, MC, RX>(), st>>>(rows, in, s, post, tw, postc, twc, out);
  return true;
}
template <typename T, int M, int MC>
bool run_prolong(long long rows, const float *y, const float2 *post, const float2 *tw, const float2 *postc,
                 const float2 *twc, const T *r, double s, T *out, cudaStream_t st) {
  constexpr int RX = x_rx<T, M>();
  static_assert(fx2_smem<M, MC, RX>() <= 48 * 1024, "no opt-in needed");
  k_prolong_fx2<T, T, M, MC, RX>
      <<<(unsigned)((rows + RX - 1) / RX), kFx2Threads, fx2_smem<M, MC, RX>(), st>>>(rows, y, post, tw, postc, twc, r, s, out);
  return true;
}

}  // namespace

// out[rows][2 MC] = restriction of s * in[rows][2 M].  false: no kernel for
// this pair (the caller then uses the table form).
template <int M>
template <typename T>
bool Fx2<M>::restrict_x(int MC, long long rows, const T *in, float s, const float2 *post, const float2 *tw,
                        const float2 *postc, const float2 *twc, float *out, cudaStream_t st) {
#define FX2_R(B)                                                                                            \
  if constexpr (fx2_pair(M, B)) {                                                                           \
    if (MC == B) return run_restrict<T, M, B>(rows, in, s, post, tw, postc, twc, out, st); \
  }
  RISM_FX2_COARSE(FX2_R)
#undef FX2_R
  return false;
}

// out[rows][2 M] = prolongation of y[rows][2 MC] - s r.
template <int M>
template <typename T>
bool Fx2<M>::prolong_x(int MC, long long rows, const float *y, const float2 *post, const float2 *tw,
                       const float2 *postc, const float2 *twc, const T *r, double s, T *out, cudaStream_t st) {
#define FX2_P(B)                                                                                              \
  if constexpr (fx2_pair(M, B)) {                                                                             \
    if (MC == B) return run_prolong<T, M, B>(rows, y, post, tw, postc, twc, r, s, out, st); \
  }
  RISM_FX2_COARSE(FX2_P)
#undef FX2_P
  return false;
}

#define RISM_INST_FX2_T(M, T)                                                                                  \
  template bool Fx2<M>::restrict_x<T>(int, long long, const T *, float, const float2 *, const float2 *,        \
                                      const float2 *, const float2 *, float *, cudaStream_t);                  \
  template bool Fx2<M>::prolong_x<T>(int, long long, const float *, const float2 *, const float2 *,            \
                                     const float2 *, const float2 *, const T *, double, T *, cudaStream_t);
#define RISM_INST_FX2(M) RISM_INST_FX2_T(M, float) RISM_INST_FX2_T(M, double)

}  // namespace rism
