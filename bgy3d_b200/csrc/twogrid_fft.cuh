// twogrid_fft.cuh -- the x-axis grid transfers of the two-grid
// preconditioner by FFT, for the row lengths with shape-specialised
// transforms (N0 = 2M).
//
// Restriction of a row x (N0 reals) to Nc coarse points, K = Nc/2:
//   out_i = (s/N0) [X_0 + 2 sum_{0<k<K} Re(e^{2 pi i k i/Nc} X_k) + Re(e^{2 pi i K i/Nc} X_K)],
// X = r2c(x) -- only X_0..X_K are formed after the row transform.
// Prolongation of a coarse row y (Nc reals) with the residual term:
//   out_j = c2r(X)_j - s r_j,  X_k = f_k sum_i y_i e^{-2 pi i k i/Nc},
// f_k = 1/Nc for k < K, 1/(2 Nc) at the Nyquist k = K, X_k = 0 above K.
// Both equal the dense band-limited transfers of twogrid.cuh (the same
// R and P) at about a third of the arithmetic: the row transform is the
// half-length complex FFT of the x passes plus the r2c untangle, and the
// coarse side is a (K+1) x Nc table product.  Transforms run in FP32.
#pragma once
#include <type_traits>

#include "kernels_static.cuh"

namespace rism {

template <typename T> __device__ __forceinline__ float2 ld_pair(const T *p);
template <> __device__ __forceinline__ float2 ld_pair<float>(const float *p) {
  return *reinterpret_cast<const float2 *>(p);
}
template <> __device__ __forceinline__ float2 ld_pair<double>(const double *p) {
  const double2 v = *reinterpret_cast<const double2 *>(p);
  return make_float2((float)v.x, (float)v.y);
}

template <int M, int RX> __host__ __device__ constexpr int fx_buf() { return RX * LayRow<M, SplitRow<M>::R2>::RS; }

// Shared memory of the two kernels (bytes) for K = Nc/2: twiddles, the row
// tiles, the coarse-side table, the kept spectrum (and the coarse rows).
template <int M, int RX> inline size_t fx_smem_restrict(int K, int Nc) {
  return sizeof(float2) * (size_t)(M + fx_buf<M, RX>() + (K + 1) * Nc + RX * (K + 1));
}
template <int M, int RX> inline size_t fx_smem_prolong(int K, int Nc) {
  return sizeof(float2) * (size_t)(M + fx_buf<M, RX>() + (K + 1) * Nc + RX * (K + 1)) +
         sizeof(float) * (size_t)RX * Nc;
}

// Vector access of 2 complex values (4 reals) of a row.
template <typename T> struct Quad;
template <> struct Quad<float> {
  using type = float4;
  __device__ __forceinline__ static void split(const float4 &v, float2 &a, float2 &b) {
    a = make_float2(v.x, v.y);
    b = make_float2(v.z, v.w);
  }
};
template <> struct Quad<double> {
  struct type { double2 a, b; };
  __device__ __forceinline__ static void split(const type &v, float2 &a, float2 &b) {
    a = make_float2((float)v.a.x, (float)v.a.y);
    b = make_float2((float)v.b.x, (float)v.b.y);
  }
};

// out[row][i] (rows x Nc, FP32) = restriction of s * in[row][.] (rows x 2M).
// ctab[k][i] = c_k e^{2 pi i k i / Nc} / N0, c = 1, 2, ..., 2, 1.
// Persistent: each CTA stages the twiddles and the table once and walks
// batches of RX rows with stride gridDim.x; the next batch's rows are loaded
// into registers while the current one is transformed.
template <typename TI, int M, int RX>
__global__ void __launch_bounds__(256) k_restrict_fx(long long rows, int Nc, int K, const TI *__restrict__ in,
                                                     float s, const float2 *__restrict__ post,
                                                     const float2 *__restrict__ twg,
                                                     const float2 *__restrict__ ctab, float *__restrict__ out) {
  using V = float2;
  using Lay = LayRow<M, SplitRow<M>::R2>;
  using Q = typename Quad<TI>::type;
  constexpr int N0 = 2 * M, PER = M / 2, CNT = (RX * PER + 255) / 256;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  V *tw = reinterpret_cast<V *>(smem_raw);
  V *buf = tw + M;
  V *C = buf + fx_buf<M, RX>();
  const int K1 = K + 1;
  V *X = C + K1 * Nc;
  const int tid = threadIdx.x;
  const long long nbat = (rows + RX - 1) / RX;
  long long bat = blockIdx.x;
  Q ra[CNT];
#define FX_LOAD_ROWS(BAT)                                                                           \
  {                                                                                                 \
    const long long r0 = (BAT) * RX;                                                                \
    _Pragma("unroll") for (int it = 0; it < CNT; ++it) {                                            \
      const int e = tid + it * 256;                                                                 \
      const int row = e / PER, jj = (e % PER) * 2;                                                  \
      if (e < RX * PER && r0 + row < rows) ra[it] = *reinterpret_cast<const Q *>(in + (r0 + row) * N0 + 2 * jj); \
    }                                                                                               \
  }
  if (bat < nbat) FX_LOAD_ROWS(bat)
  for (int q = tid; q < M; q += 256) tw[q] = twg[q];
  for (int q = tid; q < K1 * Nc; q += 256) C[q] = ctab[q];
  for (; bat < nbat; bat += gridDim.x) {
    const long long row0 = bat * RX;
#pragma unroll
    for (int it = 0; it < CNT; ++it) {
      const int e = tid + it * 256;
      if (e >= RX * PER) break;
      const int row = e / PER, jj = (e % PER) * 2;
      V a = make_float2(0.f, 0.f), b = a;
      if (row0 + row < rows) {
        Quad<TI>::split(ra[it], a, b);
        a.x *= s; a.y *= s; b.x *= s; b.y *= s;
      }
      buf[Lay::at(jj, row)] = a;
      buf[Lay::at(jj + 1, row)] = b;
    }
    if (bat + gridDim.x < nbat) FX_LOAD_ROWS(bat + gridDim.x)
    __syncthreads();
    fft2<M, RX, 256, false, false, Lay, SplitRow<M>>(buf, tw);
    for (int e = tid; e < RX * K1; e += 256) {
      const int row = e / K1, k = e - row * K1;
      const V zk = buf[Lay::at(k, row)];
      const V zm = buf[Lay::at(k == 0 ? 0 : M - k, row)];
      V E, O;
      E.x = (zk.x + zm.x) * 0.5f;
      E.y = (zk.y - zm.y) * 0.5f;
      O.x = (zk.y + zm.y) * 0.5f;
      O.y = -(zk.x - zm.x) * 0.5f;
      X[row * K1 + k] = cadd(E, cmul(post[k], O));
    }
    __syncthreads();
    // (K+1) x Nc table product, register-blocked 2 rows x 4 outputs per
    // thread: 6 shared loads per 8 complex products (shared-memory bandwidth
    // bounds this loop)
    {
      const int NQ = (Nc + 3) / 4;
      for (int e = tid; e < (RX / 2) * NQ; e += 256) {
        const int r2 = (e / NQ) * 2, i0 = (e % NQ) * 4;
        float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
        for (int k = 0; k < K1; ++k) {
          const V x0 = X[r2 * K1 + k], x1 = X[(r2 + 1) * K1 + k];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const V c = i0 + q < Nc ? C[k * Nc + i0 + q] : make_float2(0.f, 0.f);
            acc[0][q] = fmaf(c.x, x0.x, fmaf(-c.y, x0.y, acc[0][q]));
            acc[1][q] = fmaf(c.x, x1.x, fmaf(-c.y, x1.y, acc[1][q]));
          }
        }
#pragma unroll
        for (int rr = 0; rr < 2; ++rr) {
          if (row0 + r2 + rr >= rows) continue;
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (i0 + q < Nc) out[(row0 + r2 + rr) * Nc + i0 + q] = acc[rr][q];
        }
      }
    }
    __syncthreads();
  }
#undef FX_LOAD_ROWS
}

// out[row][j] (rows x 2M) = prolongation of y[row][.] (rows x Nc, FP32) - s r.
// dtab[i][k] = f_k e^{-2 pi i k i / Nc} (k fastest).  Persistent as
// k_restrict_fx: the next batch's coarse rows and subtracted fine rows are
// in flight while the current batch is transformed.
template <typename TO, typename TR, int M, int RX>
__global__ void __launch_bounds__(256) k_prolong_fx(long long rows, int Nc, int K, const float *__restrict__ y,
                                                    const float2 *__restrict__ post, const float2 *__restrict__ twg,
                                                    const float2 *__restrict__ dtab, const TR *__restrict__ r,
                                                    double s, TO *__restrict__ out) {
  using V = float2;
  using Lay = LayRow<M, SplitRow<M>::R2>;
  using QR = typename Quad<TR>::type;
  constexpr int N0 = 2 * M, H = M / 2 + 1, PER = M / 2, CNT = (RX * PER + 255) / 256;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  V *tw = reinterpret_cast<V *>(smem_raw);
  V *buf = tw + M;
  const int K1 = K + 1;
  V *D = buf + fx_buf<M, RX>();
  V *X = D + K1 * Nc;
  float *ys = reinterpret_cast<float *>(X + RX * K1);
  const int tid = threadIdx.x;
  const long long nbat = (rows + RX - 1) / RX;
  const int YC = (RX * Nc + 255) / 256;  // coarse values per thread; Nc < 2M <= 256 keeps it <= RX
  long long bat = blockIdx.x;
  QR rr[CNT], rn[CNT];
  float yv[RX];
#define FX_LOAD(BAT, RR)                                                                            \
  {                                                                                                 \
    const long long r0 = (BAT) * RX;                                                                \
    _Pragma("unroll") for (int it = 0; it < CNT; ++it) {                                            \
      const int e = tid + it * 256;                                                                 \
      const int row = e / PER, jj = (e % PER) * 2;                                                  \
      if (e < RX * PER && r0 + row < rows) RR[it] = *reinterpret_cast<const QR *>(r + (r0 + row) * N0 + 2 * jj); \
    }                                                                                               \
    _Pragma("unroll") for (int q = 0; q < RX; ++q) {                                                \
      const int e = tid + q * 256;                                                                  \
      if (q < YC) yv[q] = (e < RX * Nc && r0 + e / Nc < rows) ? y[r0 * Nc + e] : 0.f;               \
    }                                                                                               \
  }
  if (bat < nbat) FX_LOAD(bat, rr)
  for (int q = tid; q < M; q += 256) tw[q] = twg[q];
  for (int q = tid; q < K1 * Nc; q += 256) D[q] = dtab[q];
  for (; bat < nbat; bat += gridDim.x) {
    const long long row0 = bat * RX;
#pragma unroll
    for (int q = 0; q < RX; ++q) {
      const int e = tid + q * 256;
      if (q < YC && e < RX * Nc) ys[e] = yv[q];
    }
    const bool more = bat + gridDim.x < nbat;
    if (more) FX_LOAD(bat + gridDim.x, rn)
    __syncthreads();
    // Nc x (K+1) table product, register-blocked 2 rows x 3 coefficients
    // per thread: 5 shared loads per 6 complex products
    {
      const int KQ = (K1 + 2) / 3;
      for (int e = tid; e < (RX / 2) * KQ; e += 256) {
        const int r2 = (e / KQ) * 2, k0 = (e % KQ) * 3;
        float ax[2][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}}, ay[2][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
        for (int i = 0; i < Nc; ++i) {
          const float v0 = ys[r2 * Nc + i], v1 = ys[(r2 + 1) * Nc + i];
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            const V d = k0 + q < K1 ? D[i * K1 + k0 + q] : make_float2(0.f, 0.f);
            ax[0][q] = fmaf(d.x, v0, ax[0][q]);
            ay[0][q] = fmaf(d.y, v0, ay[0][q]);
            ax[1][q] = fmaf(d.x, v1, ax[1][q]);
            ay[1][q] = fmaf(d.y, v1, ay[1][q]);
          }
        }
#pragma unroll
        for (int rr = 0; rr < 2; ++rr)
#pragma unroll
          for (int q = 0; q < 3; ++q)
            if (k0 + q < K1) X[(r2 + rr) * K1 + k0 + q] = make_float2(ax[rr][q], ay[rr][q]);
      }
    }
    __syncthreads();
    for (int e = tid; e < RX * H; e += 256) {
      const int row = e / H, k = e - row * H;
      V xk = make_float2(0.f, 0.f), xm = make_float2(0.f, 0.f);
      if (k <= K) xk = X[row * K1 + k];
      if (M - k <= K) xm = X[row * K1 + (M - k)];
      if (k == 0) { xk.y = 0.f; xm.y = 0.f; }
      V Aa, Dd;
      Aa.x = xk.x + xm.x; Aa.y = xk.y - xm.y;
      Dd.x = xk.x - xm.x; Dd.y = xk.y + xm.y;
      const V Pp = cmul(Dd, cconj(post[k]));
      V zk, zm;
      zk.x = Aa.x - Pp.y; zk.y = Aa.y + Pp.x;
      zm.x = Aa.x + Pp.y; zm.y = -(Aa.y - Pp.x);
      buf[Lay::at(k, row)] = zk;
      if (k != 0 && M - k != k) buf[Lay::at(M - k, row)] = zm;
    }
    __syncthreads();
    fft2<M, RX, 256, true, false, Lay, SplitRow<M>>(buf, tw);
#pragma unroll
    for (int it = 0; it < CNT; ++it) {
      const int e = tid + it * 256;
      if (e >= RX * PER) break;
      const int row = e / PER, jj = (e % PER) * 2;
      if (row0 + row >= rows) continue;
      V ra, rb;
      Quad<TR>::split(rr[it], ra, rb);
      const V za = buf[Lay::at(jj, row)], zb = buf[Lay::at(jj + 1, row)];
      TO *o = out + (row0 + row) * N0 + 2 * jj;
      // the subtracted term in the output precision (r kept exact for FP64)
      const TR *rx = r + (row0 + row) * N0 + 2 * jj;
      if (sizeof(TR) == 8) {
        o[0] = (TO)((double)za.x - s * (double)rx[0]);
        o[1] = (TO)((double)za.y - s * (double)rx[1]);
        o[2] = (TO)((double)zb.x - s * (double)rx[2]);
        o[3] = (TO)((double)zb.y - s * (double)rx[3]);
      } else {
        const float sf = (float)s;
        o[0] = (TO)(za.x - sf * ra.x);
        o[1] = (TO)(za.y - sf * ra.y);
        o[2] = (TO)(zb.x - sf * rb.x);
        o[3] = (TO)(zb.y - sf * rb.y);
      }
    }
    if (more) {
#pragma unroll
      for (int it = 0; it < CNT; ++it) rr[it] = rn[it];
    }
    __syncthreads();
  }
#undef FX_LOAD
}

// ---- both sides by FFT: the coarse side as a packed row transform of
// length Nc = 2 MC instead of the (K+1) x Nc table product (K = MC).
//
// Restriction: out = c2r_Nc(X_0..X_K) / N0 (Im X_0, Im X_K dropped, as the
// table's c_k weights do), i.e. the K+1 kept coefficients are packed into
// MC complex values and transformed by the MC-point inverse FFT; the packed
// result z_j = out_{2j} + i out_{2j+1}.
// Prolongation: X_k = f_k r2c_Nc(y)_k from the MC-point forward FFT of the
// coarse row and its untangle, then the fine packed c2r as before.
// twc / postc: the twiddles of the MC-point transform and exp(-2 pi i k / Nc),
// k in [0, MC] (the coarse grid's own x tables).
//
// Bound by latency (a chain of barriers over 10 KB of rows), so as the x
// passes: small CTAs of one batch each, a thread's loads all in flight, both
// transforms in the order of their two steps (perm_pos), the untangling of one
// side and the packing of the other in one step between the two tiles, and the
// last step's outputs from its registers: five CTA barriers instead of ten.
// us, persistent CTAs of 256 threads with whole transforms -> here: 162 -> 54
// points FP32, restriction 62 -> 34, prolongation 79 -> 63; 128 -> 48 FP64 37 ->
// 19 and 57 -> 27.
constexpr int kFx2Threads = 128;
template <int M, int MC, int RX> __host__ __device__ constexpr size_t fx2_smem() {
  return sizeof(float2) * (size_t)(M + MC + RX * (LayRow<M, SplitRow<M>::R2>::RS + LayRow<MC, SplitRow<MC>::R2>::RS));
}

// The two steps of a forward transform of RX rows in place, spectrum in
// permuted order; ends synchronised.
template <int M, int RX, class S, class Lay> __device__ __forceinline__ void fx2_fwd(float2 *buf, const float2 *tw) {
#pragma unroll
  for (int q = threadIdx.x; q < RX * S::R2; q += kFx2Threads) {
    const int row = q / S::R2, n2 = q % S::R2;
    float2 u[S::R1];
#pragma unroll
    for (int n1 = 0; n1 < S::R1; ++n1) u[n1] = buf[Lay::at(S::R2 * n1 + n2, row)];
    fwd_step1<S>(u, n2, tw);
#pragma unroll
    for (int k1 = 0; k1 < S::R1; ++k1) buf[Lay::at(S::R2 * k1 + n2, row)] = u[k1];
  }
  __syncthreads();
#pragma unroll
  for (int q = threadIdx.x; q < RX * S::R1; q += kFx2Threads) {
    const int row = q / S::R1, k1 = q % S::R1;
    float2 u[S::R2];
#pragma unroll
    for (int n2 = 0; n2 < S::R2; ++n2) u[n2] = buf[Lay::at(S::R2 * k1 + n2, row)];
    fwd_step2<S>(u, tw);
#pragma unroll
    for (int k2 = 0; k2 < S::R2; ++k2) buf[Lay::at(S::R2 * k1 + k2, row)] = u[k2];
  }
  __syncthreads();
}
// The first step of the inverse transform in place; ends synchronised.
template <int M, int RX, class S, class Lay> __device__ __forceinline__ void fx2_inv1(float2 *buf, const float2 *tw) {
#pragma unroll
  for (int q = threadIdx.x; q < RX * S::R1; q += kFx2Threads) {
    const int row = q / S::R1, k1 = q % S::R1;
    float2 u[S::R2];
#pragma unroll
    for (int k2 = 0; k2 < S::R2; ++k2) u[k2] = buf[Lay::at(S::R2 * k1 + k2, row)];
    inv_step1<S>(u, k1, tw);
#pragma unroll
    for (int n2 = 0; n2 < S::R2; ++n2) buf[Lay::at(S::R2 * k1 + n2, row)] = u[n2];
  }
  __syncthreads();
}

// X_k of the row transform of length 2 M from its packed transform (k <= M),
// and the packed pair (Z_k, Z_{M-k}) of the inverse from (X_k, X_{M-k}).
template <int M, class S, class Lay>
__device__ __forceinline__ float2 fx2_untangle(const float2 *buf, int row, int k, const float2 *post) {
  const float2 zk = buf[Lay::at(perm_pos<S>(k == M ? 0 : k), row)];
  const float2 zm = buf[Lay::at(perm_pos<S>(k == 0 || k == M ? 0 : M - k), row)];
  const float2 E = make_float2((zk.x + zm.x) * 0.5f, (zk.y - zm.y) * 0.5f);
  const float2 O = make_float2((zk.y + zm.y) * 0.5f, -(zk.x - zm.x) * 0.5f);
  return cadd(E, cmul(post[k], O));
}
template <int M, class S, class Lay>
__device__ __forceinline__ void fx2_pack(float2 *buf, int row, int k, float2 xk, float2 xm, const float2 *post) {
  if (k == 0) { xk.y = 0.f; xm.y = 0.f; }
  const float2 Aa = make_float2(xk.x + xm.x, xk.y - xm.y), Dd = make_float2(xk.x - xm.x, xk.y + xm.y);
  const float2 Pp = cmul(Dd, cconj(post[k]));
  buf[Lay::at(perm_pos<S>(k), row)] = make_float2(Aa.x - Pp.y, Aa.y + Pp.x);
  if (k != 0 && M - k != k) buf[Lay::at(perm_pos<S>(M - k), row)] = make_float2(Aa.x + Pp.y, -(Aa.y - Pp.x));
}

template <typename TI, int M, int MC, int RX>
__global__ void __launch_bounds__(kFx2Threads) k_restrict_fx2(long long rows, const TI *__restrict__ in, float s,
                                                              const float2 *__restrict__ post, const float2 *__restrict__ twg,
                                                              const float2 *__restrict__ postc,
                                                              const float2 *__restrict__ twcg, float *__restrict__ out) {
  using S = SplitRow<M>;
  using SC = SplitRow<MC>;
  using Lay = LayRow<M, S::R2>;
  using LayC = LayRow<MC, SC::R2>;
  using VEC = typename VecW<TI, M>::vec;
  static_assert(MC < M, "the coarse row is the shorter one");
  constexpr int THR = kFx2Threads, VW = VecW<TI, M>::n, PER_ROW = M / VW, CNT = (RX * PER_ROW + THR - 1) / THR;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  float2 *tw = reinterpret_cast<float2 *>(smem_raw);
  float2 *twc = tw + M;
  float2 *buf = twc + MC;
  float2 *bc = buf + RX * Lay::RS;
  const int tid = threadIdx.x;
  const long long row0 = (long long)blockIdx.x * RX;
  VEC ra[CNT];
#pragma unroll
  for (int it = 0; it < CNT; ++it) {
    const int e = tid + it * THR;
    if (e < RX * PER_ROW && row0 + e / PER_ROW < rows)
      ra[it] = *reinterpret_cast<const VEC *>(in + (row0 + e / PER_ROW) * (2 * M) + 2 * VW * (e % PER_ROW));
  }
  for (int q = tid; q < M; q += THR) tw[q] = twg[q];
  for (int q = tid; q < MC; q += THR) twc[q] = twcg[q];
#pragma unroll
  for (int it = 0; it < CNT; ++it) {
    const int e = tid + it * THR;
    if (e >= RX * PER_ROW) break;
    const int row = e / PER_ROW, jj = (e % PER_ROW) * VW;
    const TI *v = reinterpret_cast<const TI *>(&ra[it]);
    const bool in_range = row0 + row < rows;
#pragma unroll
    for (int w = 0; w < VW; ++w)
      buf[Lay::at(jj + w, row)] =
          in_range ? make_float2((float)v[2 * w] * s, (float)v[2 * w + 1] * s) : make_float2(0.f, 0.f);
  }
  __syncthreads();
  fx2_fwd<M, RX, S, Lay>(buf, tw);
  constexpr int H = MC / 2 + 1;
#pragma unroll 2
  for (int e = tid; e < RX * H; e += THR) {
    const int row = e / H, k = e % H;
    fx2_pack<MC, SC, LayC>(bc, row, k, fx2_untangle<M, S, Lay>(buf, row, k, post),
                           fx2_untangle<M, S, Lay>(buf, row, MC - k, post), postc);
  }
  __syncthreads();
  fx2_inv1<MC, RX, SC, LayC>(bc, twc);
  const float inv_n0 = 1.0f / (float)(2 * M);
#pragma unroll
  for (int q = tid; q < RX * SC::R2; q += THR) {
    const int row = q / SC::R2, n2 = q % SC::R2;
    float2 u[SC::R1];
#pragma unroll
    for (int k1 = 0; k1 < SC::R1; ++k1) u[k1] = bc[LayC::at(SC::R2 * k1 + n2, row)];
    inv_step2<SC>(u, twc);
    if (row0 + row >= rows) continue;
    float2 *o = reinterpret_cast<float2 *>(out + (row0 + row) * (2 * MC)) + n2;
#pragma unroll
    for (int n1 = 0; n1 < SC::R1; ++n1) o[SC::R2 * n1] = make_float2(u[n1].x * inv_n0, u[n1].y * inv_n0);
  }
}

// The subtracted term s r is taken in r's precision.  The last step's outputs
// leave from its registers where its lanes cover whole sectors (R2 complex
// values in a row), else through shared memory.
template <typename TO, typename TR, int M, int MC, int RX>
__global__ void __launch_bounds__(kFx2Threads) k_prolong_fx2(long long rows, const float *__restrict__ y,
                                                             const float2 *__restrict__ post, const float2 *__restrict__ twg,
                                                             const float2 *__restrict__ postc,
                                                             const float2 *__restrict__ twcg, const TR *__restrict__ r,
                                                             double s, TO *__restrict__ out) {
  using S = SplitRow<M>;
  using SC = SplitRow<MC>;
  using Lay = LayRow<M, S::R2>;
  using LayC = LayRow<MC, SC::R2>;
  static_assert(std::is_same<TO, TR>::value && MC < M, "one field type; the coarse row is the shorter one");
  constexpr int THR = kFx2Threads;
  constexpr bool direct = S::R2 * 2 * sizeof(TR) % 32 == 0;
  constexpr int VW = direct ? 1 : VecW<TR, M>::n;
  using C2 = typename Cx<TR>::type;
  using VEC = std::conditional_t<direct, C2, typename VecW<TR, M>::vec>;
  constexpr int PER_ROW = M / VW;
  constexpr int ITEMS = (RX * S::R2 + THR - 1) / THR;
  constexpr int CNT = direct ? ITEMS * S::R1 : (RX * PER_ROW + THR - 1) / THR;
  constexpr int YC = (RX * MC + THR - 1) / THR;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  float2 *tw = reinterpret_cast<float2 *>(smem_raw);
  float2 *twc = tw + M;
  float2 *buf = twc + MC;
  float2 *bc = buf + RX * Lay::RS;
  const int tid = threadIdx.x;
  const long long row0 = (long long)blockIdx.x * RX;
  // element `it` of this thread: (row, complex index), or row < 0
  auto where = [&](int it, int &row, int &jj) {
    if (direct) {
      const int q = tid + (it / S::R1) * THR;
      row = q < RX * S::R2 ? q / S::R2 : -1;
      jj = S::R2 * (it % S::R1) + q % S::R2;
    } else {
      const int e = tid + it * THR;
      row = e < RX * PER_ROW ? e / PER_ROW : -1;
      jj = (e % PER_ROW) * VW;
    }
    if (row0 + row >= rows) row = -1;
  };
  float2 yv[YC];
#pragma unroll
  for (int it = 0; it < YC; ++it) {
    const int e = tid + it * THR;
    yv[it] = e < RX * MC && row0 + e / MC < rows ? *reinterpret_cast<const float2 *>(y + row0 * (2 * MC) + 2 * e)
                                                 : make_float2(0.f, 0.f);
  }
  VEC rin[CNT];
#pragma unroll
  for (int it = 0; it < CNT; ++it) {
    int row, jj;
    where(it, row, jj);
    if (row >= 0) rin[it] = *reinterpret_cast<const VEC *>(r + (row0 + row) * (2 * M) + 2 * jj);
  }
  for (int q = tid; q < M; q += THR) tw[q] = twg[q];
  for (int q = tid; q < MC; q += THR) twc[q] = twcg[q];
#pragma unroll
  for (int it = 0; it < YC; ++it) {
    const int e = tid + it * THR;
    if (e < RX * MC) bc[LayC::at(e % MC, e / MC)] = yv[it];
  }
  __syncthreads();
  fx2_fwd<MC, RX, SC, LayC>(bc, twc);
  // untangle to the Nc-point r2c with weights f_k (1/Nc, half at the Nyquist
  // K, real there), zero above K, and pack for the fine side
  constexpr float fk = 1.0f / (float)(2 * MC);
  auto spec = [&](int row, int k) {
    if (k > MC) return make_float2(0.f, 0.f);
    const float2 x = fx2_untangle<MC, SC, LayC>(bc, row, k, postc);
    return k == MC ? make_float2(x.x * (0.5f * fk), 0.f) : make_float2(x.x * fk, x.y * fk);
  };
  constexpr int H = M / 2 + 1;
#pragma unroll 2
  for (int e = tid; e < RX * H; e += THR) {
    const int row = e / H, k = e % H;
    fx2_pack<M, S, Lay>(buf, row, k, spec(row, k), spec(row, M - k), post);
  }
  __syncthreads();
  fx2_inv1<M, RX, S, Lay>(buf, tw);
  const TR sr = (TR)s;
  auto put = [&](int it, int row, int jj, const float2 *z) {
    if (row < 0) return;
    const TR *rr = reinterpret_cast<const TR *>(&rin[it]);
    VEC o;
    TR *oo = reinterpret_cast<TR *>(&o);
#pragma unroll
    for (int w = 0; w < VW; ++w) {
      oo[2 * w] = (TR)z[w].x - sr * rr[2 * w];
      oo[2 * w + 1] = (TR)z[w].y - sr * rr[2 * w + 1];
    }
    *reinterpret_cast<VEC *>(out + (row0 + row) * (2 * M) + 2 * jj) = o;
  };
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const int q = tid + i * THR;
    if (q >= RX * S::R2) break;
    const int row = q / S::R2, n2 = q % S::R2;
    float2 u[S::R1];
#pragma unroll
    for (int k1 = 0; k1 < S::R1; ++k1) u[k1] = buf[Lay::at(S::R2 * k1 + n2, row)];
    inv_step2<S>(u, tw);
#pragma unroll
    for (int n1 = 0; n1 < S::R1; ++n1) {
      if constexpr (direct)
        put(i * S::R1 + n1, row0 + row < rows ? row : -1, S::R2 * n1 + n2, &u[n1]);
      else
        buf[Lay::at(S::R2 * n1 + n2, row)] = u[n1];
    }
  }
  if constexpr (!direct) {
    __syncthreads();
#pragma unroll
    for (int it = 0; it < CNT; ++it) {
      int row, jj;
      where(it, row, jj);
      float2 z[VW];
#pragma unroll
      for (int w = 0; w < VW; ++w) z[w] = row >= 0 ? buf[Lay::at(jj + w, row)] : float2{};
      put(it, row, jj, z);
    }
  }
}

}  // namespace rism
