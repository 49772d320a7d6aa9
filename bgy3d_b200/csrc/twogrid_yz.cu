// twogrid_yz.cu -- the y and z grid transfers of the two-grid preconditioner
// by FFT (sm_100a).
//
// Along one axis the band-limited restriction R (N -> Nc points) and
// prolongation P (Nc -> N) of twogrid.cuh are
//
//   R v = (1/N)  IDFT_Nc( truncate_w( DFT_N v ) ),
//   P c = (1/Nc) IDFT_N ( pad_w     ( DFT_Nc c ) ),
//
// truncate_w keeping the modes |k| < Nc/2 and folding +-Nc/2 into the
// coarse Nyquist mode with weight 1/2 each, pad_w its transpose (the coarse
// Nyquist mode split in halves onto +-Nc/2, zeros elsewhere).  Both are real
// operators, so two adjacent real columns (a, b) -- one float2 in memory --
// go through as the complex column a + ib and come out as Ra + iRb.
//
// A CTA takes 16 (or 8) such columns, rows of 128 (64) bytes, and each of its
// threads one DFT of every step: the first reads its rows from global memory,
// the second leaves the spectrum of the tile in shared memory, in the order of
// its two steps (fft_static.cuh); the third gathers the kept modes from there
// and the last writes its rows to global memory.  One read and one write of
// each field and four barriers; with whole transforms through shared memory
// there were eight.  At 256^3, us per launch on average of y and z: 256 -> 64 points
// 24.3 -> 11.7, 64 -> 256 18.2 -> 10.3 (4.9 TB/s of the larger field along y).
#include <cuda_runtime.h>

#include "fft_static.cuh"

namespace rism {

namespace {

// Complex column pairs per tile: 16 (128-byte rows) where both tiles and the
// twiddles fit the default 48 KB of shared memory, else 8.
template <int NI, int NO> __host__ __device__ constexpr int yz_cols() {
  return (NI + NO) * (16 + 1) * 8 <= 48 * 1024 && SplitSq<NI>::R1 <= 16 && SplitSq<NO>::R1 <= 16 ? 16 : 8;
}

template <int NI, int NO> __host__ __device__ constexpr size_t yz_smem() {
  return sizeof(float2) * ((size_t)(NI + NO) * yz_cols<NI, NO>() + NI + NO);
}

// in [outer][NI][inner] -> out [outer][NO][inner] floats, inner even.
template <int NI, int NO>
__global__ void __launch_bounds__(256) k_transfer_fft(int outer, int inner, const float *__restrict__ in,
                                                      const float2 *__restrict__ twi, const float2 *__restrict__ two,
                                                      float *__restrict__ out) {
  constexpr int B = yz_cols<NI, NO>();
  using SI = SplitSq<NI>;
  using SO = SplitSq<NO>;
  static_assert(SI::R1 * SI::R2 == NI && SO::R1 * SO::R2 == NO, "two-step splits");
  static_assert(SI::R1 * B <= 256 && SI::R2 * B <= 256 && SO::R1 * B <= 256 && SO::R2 * B <= 256,
                "one DFT of every step per thread");
  extern __shared__ __align__(16) unsigned char yz_raw[];
  float2 *X = reinterpret_cast<float2 *>(yz_raw);  // [NI][B], row R2 k1 + k2: mode k1 + R1 k2
  float2 *Y = X + NI * B;                            // [NO][B]
  float2 *ti = Y + NO * B;
  float2 *to = ti + NI;
  const int tid = threadIdx.x;
  const int c = tid % B, w = tid / B;  // column, work item of the column
  const int ntile = (inner + 2 * B - 1) / (2 * B);
  const int o = blockIdx.x / ntile;
  const int i0 = (blockIdx.x - o * ntile) * 2 * B;
  const bool in_row = i0 + 2 * c < inner;
  {
    const float *src = in + (long long)o * NI * inner + i0 + 2 * c;
    float2 u[SI::R1];
    if (w < SI::R2) {
#pragma unroll
      for (int n1 = 0; n1 < SI::R1; ++n1)
        u[n1] = in_row ? *reinterpret_cast<const float2 *>(src + (long long)(SI::R2 * n1 + w) * inner)
                       : make_float2(0.f, 0.f);
    }
    for (int q = tid; q < NI; q += 256) ti[q] = twi[q];
    for (int q = tid; q < NO; q += 256) to[q] = two[q];
    __syncthreads();
    if (w < SI::R2) {
      fwd_step1<SI>(u, w, ti);
#pragma unroll
      for (int k1 = 0; k1 < SI::R1; ++k1) X[(SI::R2 * k1 + w) * B + c] = u[k1];
    }
  }
  __syncthreads();
  if (w < SI::R1) {
    float2 u[SI::R2];
    float2 *p = X + SI::R2 * w * B + c;
#pragma unroll
    for (int n2 = 0; n2 < SI::R2; ++n2) u[n2] = p[n2 * B];
    fwd_step2<SI>(u, ti);
#pragma unroll
    for (int k2 = 0; k2 < SI::R2; ++k2) p[k2 * B] = u[k2];
  }
  __syncthreads();
  if (w < SO::R1) {
    const float scale = 1.0f / (float)NI;
    auto mode = [&](int k) { return X[perm_pos<SI>(k) * B + c]; };
    float2 u[SO::R2];
#pragma unroll
    for (int k2 = 0; k2 < SO::R2; ++k2) {
      const int k = w + SO::R1 * k2;
      float2 v = make_float2(0.f, 0.f);
      if (NO < NI) {  // truncate: coarse mode k from the fine spectrum
        if (2 * k == NO) {
          const float2 a = mode(k), b = mode(NI - k);
          v = make_float2(0.5f * (a.x + b.x), 0.5f * (a.y + b.y));
        } else {
          v = mode(2 * k < NO ? k : NI - NO + k);
        }
      } else {  // pad: fine mode k from the coarse spectrum
        if (2 * k == NI || 2 * (NO - k) == NI) {
          const float2 a = mode(NI / 2);
          v = make_float2(0.5f * a.x, 0.5f * a.y);
        } else if (2 * k < NI) {
          v = mode(k);
        } else if (2 * (NO - k) < NI) {
          v = mode(NI - NO + k);
        }
      }
      u[k2] = make_float2(v.x * scale, v.y * scale);
    }
    inv_step1<SO>(u, w, to);
    float2 *p = Y + SO::R2 * w * B + c;
#pragma unroll
    for (int n2 = 0; n2 < SO::R2; ++n2) p[n2 * B] = u[n2];
  }
  __syncthreads();
  if (w < SO::R2 && in_row) {
    float2 u[SO::R1];
#pragma unroll
    for (int k1 = 0; k1 < SO::R1; ++k1) u[k1] = Y[(SO::R2 * k1 + w) * B + c];
    inv_step2<SO>(u, to);
    float *dst = out + (long long)o * NO * inner + i0 + 2 * c;
#pragma unroll
    for (int n1 = 0; n1 < SO::R1; ++n1)
      *reinterpret_cast<float2 *>(dst + (long long)(SO::R2 * n1 + w) * inner) = u[n1];
  }
}

template <int NI, int NO>
bool launch_fft(int outer, int inner, const float *in, const float2 *twi, const float2 *two, float *out,
                cudaStream_t st) {
  constexpr int B = yz_cols<NI, NO>();
  constexpr size_t sm = yz_smem<NI, NO>();
  static_assert(sm <= 48 * 1024, "tile exceeds the default shared memory");
  const long long tiles = (long long)outer * ((inner + 2 * B - 1) / (2 * B));
  if (tiles > 0x7fffffffLL) return false;
  k_transfer_fft<NI, NO><<<(unsigned)tiles, 256, sm, st>>>(outer, inner, in, twi, two, out);
  return true;
}

// The pairs of axis lengths with a kernel in both directions: as along x
// (ratios of 1.3 to 4.6; 512 points down to 96).
constexpr bool yz_pair(int F, int C) { return 13 * C <= 10 * F && (10 * F <= 46 * C || (F == 512 && C == 96)); }

template <int F, int C>
bool run_pair(int n_in, int outer, int inner, const float *in, const float2 *twi, const float2 *two, float *out,
              cudaStream_t st) {
  if constexpr (yz_pair(F, C))
    return n_in == F ? launch_fft<F, C>(outer, inner, in, twi, two, out, st)
                     : launch_fft<C, F>(outer, inner, in, twi, two, out, st);
  else
    return false;
}

template <int F>
bool run_fine(int n_coarse, int n_in, int outer, int inner, const float *in, const float2 *twi, const float2 *two,
              float *out, cudaStream_t st) {
  switch (n_coarse) {
#define YZ_COARSE(C) \
  case C: return run_pair<F, C>(n_in, outer, inner, in, twi, two, out, st);
    YZ_COARSE(32) YZ_COARSE(36) YZ_COARSE(48) YZ_COARSE(54) YZ_COARSE(64) YZ_COARSE(72) YZ_COARSE(96) YZ_COARSE(108)
    YZ_COARSE(128)
#undef YZ_COARSE
    default: return false;
  }
}

}  // namespace

// out [outer][n_out][inner] = transfer of in [outer][n_in][inner] along the
// middle axis (restriction when n_out < n_in); twi / two: the FP32 twiddle
// tables exp(-2 pi i q / n) of lengths n_in / n_out.  False: no kernel for
// this pair, or inner odd.
bool yz_fft_transfer(int outer, int n_in, int n_out, int inner, const float *in, const float2 *twi,
                     const float2 *two, float *out, cudaStream_t st) {
  if (inner % 2 != 0 || outer < 1) return false;
  const int fine = n_in > n_out ? n_in : n_out, coarse = n_in > n_out ? n_out : n_in;
  switch (fine) {
#define YZ_FINE(F) \
  case F: return run_fine<F>(coarse, n_in, outer, inner, in, twi, two, out, st);
    YZ_FINE(48) YZ_FINE(54) YZ_FINE(64) YZ_FINE(72) YZ_FINE(96) YZ_FINE(108) YZ_FINE(128) YZ_FINE(144) YZ_FINE(162)
    YZ_FINE(192) YZ_FINE(216) YZ_FINE(256) YZ_FINE(288) YZ_FINE(324) YZ_FINE(384) YZ_FINE(432) YZ_FINE(486)
    YZ_FINE(512)
#undef YZ_FINE
    default: return false;
  }
}

}  // namespace rism
