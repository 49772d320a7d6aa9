// twogrid_fx2_impl.cuh -- definitions of twogrid_fx2.cuh.
#pragma once
#include <algorithm>
#include <cstdlib>

#include "twogrid_fft.cuh"
#include "twogrid_fx2.cuh"

namespace rism {

namespace {

constexpr int kRX = 16;  // rows per batch, as the table-product kernels

// Rows per batch of the 128-point half rows (the 256^3 grid): 16 or 32
// (RISM3D_FX2_ROWS, read once).
inline int rows_128() {
  static const int r = [] {
    const char *e = std::getenv("RISM3D_FX2_ROWS");
    return e && std::atoi(e) == 32 ? 32 : 16;
  }();
  return r;
}

// Persistent CTAs: as many as fit at once, at most `work`; also raises the
// kernel's dynamic shared-memory limit when it needs more than 48 KB.
// Returns 0 when the tile does not fit on this device.
inline unsigned fx2_grid(const void *fn, size_t smem, unsigned work) {
  int dev = 0, sms = 0, optin = 0, per = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return 0;
  if (smem + 4096 > (size_t)optin) return 0;
  if (smem > 48 * 1024 && cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, 256, smem) != cudaSuccess || per < 1) return 0;
  return std::max(1u, std::min((unsigned)per * (unsigned)sms, work));
}

template <typename T, int M, int MC, int RX>
bool run_restrict(long long rows, const T *in, float s, const float2 *post, const float2 *tw, const float2 *postc,
                  const float2 *twc, float *out, cudaStream_t st) {
  const size_t sm = fx2_smem<M, MC, RX>();
  const unsigned g = fx2_grid((const void *)k_restrict_fx2<T, M, MC, RX>, sm, (unsigned)((rows + RX - 1) / RX));
  if (g == 0) return false;
  k_restrict_fx2<T, M, MC, RX><<<g, 256, sm, st>>>(rows, in, s, post, tw, postc, twc, out);
  return true;
}
template <typename T, int M, int MC, int RX>
bool run_prolong(long long rows, const float *y, const float2 *post, const float2 *tw, const float2 *postc,
                 const float2 *twc, const T *r, double s, T *out, cudaStream_t st) {
  const size_t sm = fx2_smem<M, MC, RX>();
  const unsigned g = fx2_grid((const void *)k_prolong_fx2<T, T, M, MC, RX>, sm, (unsigned)((rows + RX - 1) / RX));
  if (g == 0) return false;
  k_prolong_fx2<T, T, M, MC, RX><<<g, 256, sm, st>>>(rows, y, post, tw, postc, twc, r, s, out);
  return true;
}

}  // namespace

// out[rows][2 MC] = restriction of s * in[rows][2 M].  false: no kernel for
// this pair or its tile does not fit (the caller then uses the table form).
template <int M>
template <typename T>
bool Fx2<M>::restrict_x(int MC, long long rows, const T *in, float s, const float2 *post, const float2 *tw,
                        const float2 *postc, const float2 *twc, float *out, cudaStream_t st) {
#define FX2_R(B)                                                                                            \
  if constexpr (fx2_pair(M, B)) {                                                                           \
    if (MC == B) {                                                                                          \
      if constexpr (M == 128) {                                                                             \
        if (rows_128() == 32) return run_restrict<T, M, B, 32>(rows, in, s, post, tw, postc, twc, out, st); \
      }                                                                                                     \
      return run_restrict<T, M, B, kRX>(rows, in, s, post, tw, postc, twc, out, st);                        \
    }                                                                                                       \
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
    if (MC == B) {                                                                                            \
      if constexpr (M == 128) {                                                                               \
        if (rows_128() == 32) return run_prolong<T, M, B, 32>(rows, y, post, tw, postc, twc, r, s, out, st);  \
      }                                                                                                       \
      return run_prolong<T, M, B, kRX>(rows, y, post, tw, postc, twc, r, s, out, st);                         \
    }                                                                                                         \
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
