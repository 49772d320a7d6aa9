// kernels_static.cuh -- shape-specialised FFT passes of the 3D-RISM residual
// (the same five passes as kernels.cuh, for compile-time transform lengths).
//
//   k_xfwd_s  closure (or its linearisation) + r2c along x: RX contiguous rows
//             per CTA, vector loads, padded shared-memory rows;
//   k_y_s     one [N1][B] column tile per CTA, loaded and stored by TMA;
//   k_z_s     the m [N2][B] tiles of one (ky, kx-block), TMA in and out, with
//             the OZ contraction between the forward and inverse transforms;
//   k_xinv_s  c2r along x with "- t" and the residual norms.
//
// B columns of a y/z tile are 128 bytes (16 float2 or 8 double2): one TMA box
// row per transform index, so every HBM access is a whole 128-byte line.
#pragma once
#include <type_traits>

#include "fft_static.cuh"
#include "kernels.cuh"

namespace rism {

constexpr uint32_t kMbarPolls = 1u << 26;  // bounded mbarrier wait (seconds)

// Complex values per vector load in the x passes: 16 bytes, or one value
// where an odd half row leaves every other row off a 16-byte boundary.
template <typename T, int M> struct VecW { static constexpr int n = 1; using vec = typename Cx<T>::type; };
template <int M> struct VecW<float, M> {
  static constexpr int n = M % 2 == 0 ? 2 : 1;
  using vec = std::conditional_t<M % 2 == 0, float4, float2>;
};

// The x passes take RX rows with 128 threads (256 in the FP32 forward pass, whose
// exponentials want the warps): about 8 KB of a field per CTA, so that a thread
// has all its loads in flight and several small CTAs share an SM.  Sixteen rows
// of 512 points in FP64 took 256 registers of loads, and long FP32 rows fell
// back to a loop of two loads in flight.  Inverse pass, us, with 256 threads and
// whole transforms through shared memory -> here: 128^3 FP32 21.7 -> 20.7, FP64
// 46 -> 34; 256^3 133 -> 110, 288 -> 241; 512^3 1413 -> 888, 3985 -> 2352.
constexpr int kXThreads = 128;
template <typename T> __host__ __device__ constexpr int xfwd_threads() { return sizeof(T) == 4 ? 256 : 128; }
__host__ __device__ constexpr int x_rows(bool f64, int M) {
  return f64 ? (M <= 64 ? 16 : M <= 162 ? 8 : 4) : (M <= 128 ? 16 : 8);
}
template <typename T, int M> __host__ __device__ constexpr int x_rx() { return x_rows(sizeof(T) == 8, M); }

// x forward (see k_xfwd): MODE_F c = closure(p B, A); MODE_J c = B (p A);
// MODE_S c = closure'(p B, Tv) A.  In FP64 the spectrum stays in the order of
// the two transform steps (perm_pos) and the untangling indexes it there (J at
// 256^3 207 -> 197 us); in FP32 the natural order is the faster one (125 -> 116).
template <typename T, int MODE, int M, int RX>
__global__ void __launch_bounds__(xfwd_threads<T>()) k_xfwd_s(Geo g, const T *__restrict__ A, const T *__restrict__ Bv,
                                                     const T *__restrict__ Tv, T p, int closure,
                                                     typename Cx<T>::type *__restrict__ W,
                                                     const typename Cx<T>::type *__restrict__ post,
                                                     const typename Cx<T>::type *__restrict__ twg) {
  using V = typename Cx<T>::type;
  using S = SplitRow<M>;
  using Lay = LayRow<M, S::R2>;
  constexpr int THR = xfwd_threads<T>();
  constexpr bool PERM = sizeof(T) == 8;
  constexpr int VW = VecW<T, M>::n;
  using VEC = typename VecW<T, M>::vec;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  V *tw = reinterpret_cast<V *>(smem_raw);
  V *buf = tw + M;
  const int tid = threadIdx.x;
  const int rows_total = g.N1 * g.N2;
  const int row0 = blockIdx.x * RX;
  const int site = blockIdx.y;
  for (int q = tid; q < M; q += THR) tw[q] = twg[q];
  const long long sbase = (long long)site * g.Nr;
  constexpr int PER_ROW = M / VW;
  constexpr int CNT = (RX * PER_ROW + THR - 1) / THR;
  // all loads of the thread in flight before any use
  VEC ra[CNT], rb[CNT], rt[MODE == MODE_S ? CNT : 1];
#pragma unroll
  for (int it = 0; it < CNT; ++it) {
    const int e = tid + it * THR;
    const int row = e / PER_ROW, jj = (e % PER_ROW) * VW;
    if (e < RX * PER_ROW && row0 + row < rows_total) {
      const long long off = sbase + (long long)(row0 + row) * g.N0 + 2 * jj;
      ra[it] = *reinterpret_cast<const VEC *>(A + off);
      rb[it] = *reinterpret_cast<const VEC *>(Bv + off);
      if (MODE == MODE_S) rt[it] = *reinterpret_cast<const VEC *>(Tv + off);
    }
  }
#pragma unroll
  for (int it = 0; it < CNT; ++it) {
    const int e = tid + it * THR;
    if (e >= RX * PER_ROW) break;
    const int row = e / PER_ROW, jj = (e % PER_ROW) * VW;
    const int grow = row0 + row;
    V z[VW];
#pragma unroll
    for (int v = 0; v < VW; ++v) z[v].x = z[v].y = T(0);
    if (grow < rows_total) {
      const T *ar = reinterpret_cast<const T *>(&ra[it]);
      const T *br = reinterpret_cast<const T *>(&rb[it]);
      const T *tr = reinterpret_cast<const T *>(&rt[MODE == MODE_S ? it : 0]);
#pragma unroll
      for (int v = 0; v < VW; ++v) {
        if (MODE == MODE_F) {
          z[v].x = closure_c<T>(closure, p * br[2 * v], ar[2 * v]);
          z[v].y = closure_c<T>(closure, p * br[2 * v + 1], ar[2 * v + 1]);
        } else if (MODE == MODE_S) {
          z[v].x = closure_d<T>(closure, p * br[2 * v], tr[2 * v]) * ar[2 * v];
          z[v].y = closure_d<T>(closure, p * br[2 * v + 1], tr[2 * v + 1]) * ar[2 * v + 1];
        } else {
          z[v].x = br[2 * v] * (ar[2 * v] * p);
          z[v].y = br[2 * v + 1] * (ar[2 * v + 1] * p);
        }
      }
    }
#pragma unroll
    for (int v = 0; v < VW; ++v) buf[Lay::at(jj + v, row)] = z[v];
  }
  __syncthreads();
  if constexpr (PERM) {
#pragma unroll
    for (int q = tid; q < RX * S::R2; q += THR) {
      const int row = q / S::R2, n2 = q % S::R2;
      V u[S::R1];
#pragma unroll
      for (int n1 = 0; n1 < S::R1; ++n1) u[n1] = buf[Lay::at(S::R2 * n1 + n2, row)];
      fwd_step1<S>(u, n2, tw);
#pragma unroll
      for (int k1 = 0; k1 < S::R1; ++k1) buf[Lay::at(S::R2 * k1 + n2, row)] = u[k1];
    }
    __syncthreads();
#pragma unroll
    for (int q = tid; q < RX * S::R1; q += THR) {
      const int row = q / S::R1, k1 = q % S::R1;
      V u[S::R2];
#pragma unroll
      for (int n2 = 0; n2 < S::R2; ++n2) u[n2] = buf[Lay::at(S::R2 * k1 + n2, row)];
      fwd_step2<S>(u, tw);
#pragma unroll
      for (int k2 = 0; k2 < S::R2; ++k2) buf[Lay::at(S::R2 * k1 + k2, row)] = u[k2];
    }
    __syncthreads();
  } else {
    fft2<M, RX, THR, false, false, Lay, S>(buf, tw);
  }
  constexpr int H = M / 2 + 1;
  const long long wbase = (long long)site * g.Nc;
  for (int e = tid; e < RX * H; e += THR) {
    const int row = e / H, k = e % H;
    const int grow = row0 + row;
    if (grow >= rows_total) continue;
    const int km = k == 0 ? 0 : M - k;
    const V zk = buf[Lay::at(PERM ? perm_pos<S>(k) : k, row)];
    const V zm = buf[Lay::at(PERM ? perm_pos<S>(km) : km, row)];
    V E, O;
    E.x = (zk.x + zm.x) * T(0.5);
    E.y = (zk.y - zm.y) * T(0.5);
    O.x = (zk.y + zm.y) * T(0.5);
    O.y = -(zk.x - zm.x) * T(0.5);
    const V wO = cmul(post[k], O);
    V *row_out = W + wbase + (long long)grow * g.Nhp;
    row_out[k] = cadd(E, wO);
    if (M - k != k) row_out[M - k] = cconj(csub(E, wO));
  }
}

// x inverse (see k_xinv): out = scale x - sub In, and, where part is given,
// the residual norms.  The packed input is written in the order that the first
// inverse step works on.  The last step's outputs leave from its registers
// where its lanes cover whole 32-byte sectors (R2 complex values in a row),
// else through shared memory as 16-byte vectors.
template <typename T, int M, int RX>
__global__ void __launch_bounds__(kXThreads) k_xinv_s(Geo g, const typename Cx<T>::type *__restrict__ W,
                                                     const T *__restrict__ In, T *__restrict__ Out, T scale, T sub,
                                                     const typename Cx<T>::type *__restrict__ post,
                                                     const typename Cx<T>::type *__restrict__ twg,
                                                     NormPartial *__restrict__ part) {
  using V = typename Cx<T>::type;
  using S = SplitRow<M>;
  using Lay = LayRow<M, S::R2>;
  constexpr int THR = kXThreads;
  constexpr bool direct = S::R2 * sizeof(V) % 32 == 0;
  constexpr int VW = direct ? 1 : VecW<T, M>::n;
  using VEC = std::conditional_t<direct, V, typename VecW<T, M>::vec>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  V *tw = reinterpret_cast<V *>(smem_raw);
  V *buf = tw + M;
  const int tid = threadIdx.x;
  const int rows_total = g.N1 * g.N2;
  const int row0 = blockIdx.x * RX;
  const int site = blockIdx.y;
  for (int q = tid; q < M; q += THR) tw[q] = twg[q];
  constexpr int H = M / 2 + 1;
  const long long wbase = (long long)site * g.Nc;
  const long long sbase = (long long)site * g.Nr;
  constexpr int PER_ROW = M / VW;
  constexpr int ITEMS = (RX * S::R2 + THR - 1) / THR;  // last-step DFTs per thread
  constexpr int CNT = direct ? ITEMS * S::R1 : (RX * PER_ROW + THR - 1) / THR;
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
    if (row0 + row >= rows_total) row = -1;
  };
  constexpr int CW = (RX * H + THR - 1) / THR;
  // every (X_k, X_{M-k}) pair of this thread and the subtracted input are
  // loaded before the first is used
  V xkv[CW], xmv[CW];
#pragma unroll
  for (int it = 0; it < CW; ++it) {
    const int e = tid + it * THR;
    const int row = e / H, k = e % H;
    xkv[it].x = xkv[it].y = xmv[it].x = xmv[it].y = T(0);
    if (e < RX * H && row0 + row < rows_total) {
      const V *row_in = W + wbase + (long long)(row0 + row) * g.Nhp;
      xkv[it] = row_in[k];
      xmv[it] = row_in[M - k];
    }
  }
  VEC rin[CNT];
#pragma unroll
  for (int it = 0; it < CNT; ++it) {
    int row, jj;
    where(it, row, jj);
    if (row >= 0) rin[it] = *reinterpret_cast<const VEC *>(In + sbase + (long long)(row0 + row) * g.N0 + 2 * jj);
  }
#pragma unroll
  for (int it = 0; it < CW; ++it) {
    const int e = tid + it * THR;
    const int row = e / H, k = e % H;
    if (e >= RX * H) break;
    V xk = xkv[it], xm = xmv[it];
    if (k == 0) { xk.y = T(0); xm.y = T(0); }  // c2r reads only Re X_0, Re X_{N0/2}
    V Aa, D, zk, zm;
    Aa.x = xk.x + xm.x; Aa.y = xk.y - xm.y;
    D.x = xk.x - xm.x;  D.y = xk.y + xm.y;
    const V Pp = cmul(D, cconj(post[k]));
    zk.x = Aa.x - Pp.y; zk.y = Aa.y + Pp.x;
    zm.x = Aa.x + Pp.y; zm.y = -(Aa.y - Pp.x);
    buf[Lay::at(perm_pos<S>(k), row)] = zk;
    if (k != 0 && M - k != k) buf[Lay::at(perm_pos<S>(M - k), row)] = zm;
  }
  __syncthreads();
#pragma unroll
  for (int q = tid; q < RX * S::R1; q += THR) {
    const int row = q / S::R1, k1 = q % S::R1;
    V u[S::R2];
#pragma unroll
    for (int k2 = 0; k2 < S::R2; ++k2) u[k2] = buf[Lay::at(S::R2 * k1 + k2, row)];
    inv_step1<S>(u, k1, tw);
#pragma unroll
    for (int n2 = 0; n2 < S::R2; ++n2) buf[Lay::at(S::R2 * k1 + n2, row)] = u[n2];
  }
  __syncthreads();
  double amax = 0.0, sum2 = 0.0;
  auto put = [&](int it, int row, int jj, const V *z) {
    if (row < 0) return;
    const T *ir = reinterpret_cast<const T *>(&rin[it]);
    VEC o;
    T *orr = reinterpret_cast<T *>(&o);
#pragma unroll
    for (int v = 0; v < VW; ++v) {
      orr[2 * v] = z[v].x * scale - sub * ir[2 * v];
      orr[2 * v + 1] = z[v].y * scale - sub * ir[2 * v + 1];
    }
    *reinterpret_cast<VEC *>(Out + sbase + (long long)(row0 + row) * g.N0 + 2 * jj) = o;
    if (part) {
#pragma unroll
      for (int v = 0; v < 2 * VW; ++v) {
        const double ov = (double)orr[v];
        amax = fmax(amax, fabs(ov));
        sum2 += ov * ov;
      }
    }
  };
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const int q = tid + i * THR;
    if (q >= RX * S::R2) break;
    const int row = q / S::R2, n2 = q % S::R2;
    V u[S::R1];
#pragma unroll
    for (int k1 = 0; k1 < S::R1; ++k1) u[k1] = buf[Lay::at(S::R2 * k1 + n2, row)];
    inv_step2<S>(u, tw);
#pragma unroll
    for (int n1 = 0; n1 < S::R1; ++n1) {
      if constexpr (direct)
        put(i * S::R1 + n1, row0 + row < rows_total ? row : -1, S::R2 * n1 + n2, &u[n1]);
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
      V z[VW];
#pragma unroll
      for (int v = 0; v < VW; ++v) z[v] = row >= 0 ? buf[Lay::at(jj + v, row)] : V{};
      put(it, row, jj, z);
    }
  }
  if (part) block_norms(amax, sum2, part + (blockIdx.y * gridDim.x + blockIdx.x));
}

// A TMA box spans at most 256 elements per dimension: tiles along a longer
// axis move as two boxes of half its rows, or three of a third where half is
// odd: a box lands on a 128-byte boundary of shared memory, and a z row is 64
// bytes.
__host__ __device__ constexpr int tma_rows(int n) { return n <= 256 ? n : (n % 4 == 0 ? n / 2 : n / 3); }
template <typename V, int N, int B> __host__ __device__ constexpr bool tma_tile_ok() {
  return N % tma_rows(N) == 0 && tma_rows(N) <= 256 && (size_t)N * B * sizeof(V) % 128 == 0 &&
         (size_t)tma_rows(N) * B * sizeof(V) % 128 == 0;
}

// y pass: one [N][B] tile (kx0 .. kx0+B-1 at fixed z, site) by TMA.
// tm: W as {2 Nhp, N1, m N2} scalars, box {2B, N1, 1}.  ALONG_Z: the same
// along z, at fixed y (box {2B, 1, N2}): the z transform alone, for the passes
// whose work at a k point is a kernel of its own (k_oz, the forward transform
// of the gradient).
template <typename T, bool INV, int N, int B, bool ALONG_Z = false>
__global__ void __launch_bounds__(SplitY<N>::R1 * B) k_y_s(Geo g, const __grid_constant__ CUtensorMap tm,
                                                         const typename Cx<T>::type *__restrict__ twg,
                                                         int *__restrict__ err) {
  using V = typename Cx<T>::type;
  constexpr int NTHR = SplitY<N>::R1 * B;
  static_assert(tma_tile_ok<V, N, B>(), "every box starts on a 128-byte boundary");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  V *buf = reinterpret_cast<V *>(smem_raw);
  V *tw = buf + N * B;
  uint64_t *bar = reinterpret_cast<uint64_t *>(tw + N);
  const int tid = threadIdx.x;
  const int kx0 = blockIdx.x * B, f = blockIdx.y, site = blockIdx.z;  // f: the fixed z (or y)
  if (tid == 0) mbar_init(bar, 1);
  __syncthreads();
  if (tid == 0) {
    mbar_expect_tx(bar, (uint32_t)(N * B * sizeof(V)));
#pragma unroll
    for (int c = 0; c < N; c += tma_rows(N))
      tma_load_3d(buf + c * B, &tm, bar, 2 * kx0, ALONG_Z ? f : c, site * g.N2 + (ALONG_Z ? c : f));
  }
  for (int q = tid; q < N; q += NTHR) tw[q] = twg[q];
  if (!cta_wait_tile(bar, 0, kMbarPolls, err, ALONG_Z ? 2 : 1)) return;
  fft2<N, B, NTHR, INV, true, LayCol<N, B>, SplitY<N>>(buf, tw);
  fence_proxy_async();
  __syncthreads();
  if (tid == 0) {
#pragma unroll
    for (int c = 0; c < N; c += tma_rows(N))
      tma_store_3d(&tm, buf + c * B, 2 * kx0, ALONG_Z ? f : c, site * g.N2 + (ALONG_Z ? c : f));
    tma_commit();
    tma_wait_read0();
  }
}

// Row pairs whose chi - 1 values a thread has in flight during the z
// contraction: 4 in the FP32 Jacobian pass, 2 where the residual's
// long-range terms or FP64 values take the registers (the FP32 passes stay
// within 128 registers, i.e. the 4 CTAs per SM that shared memory allows).
template <typename T, int MODE> __host__ __device__ constexpr int zpf_default() {
  return sizeof(T) == 4 && MODE == MODE_J ? 4 : 2;
}

// One z tile in shared memory: forward transform along z of the m [N][B]
// site columns, the OZ contraction with chi - 1 (+ the long-range terms in
// MODE_F), inverse transform; ends after a barrier.  Run by the NTHR = R1 B
// threads tid of a group (act false: barriers only); JOINT: the MS site
// tiles (all allocated) transform as one MS B-column tile by R1 B MS threads.
//
// chi - 1 comes from the octant table (k_octant): rows z and N - z of a
// column share its values, so a thread contracts both on one set of loads
// (row 0 is paired with row N / 2, which has values of its own).  The loads
// depend only on where the row sits on the k grid, so a thread keeps those of
// its next ZPF row pairs (and, in MODE_F, their long-range values) in flight
// while it contracts the current one, and issues the first ZPF before the
// forward transforms, under whose latency they arrive.  Same arithmetic as
// the rule evaluated at every element.
template <typename T, int MODE, int N, int B, int MS, bool JOINT = false, int ZPF = zpf_default<T, MODE>(),
          class S = Split<N>>
__device__ __forceinline__ void z_tile_g(const Geo &g, typename Cx<T>::type *buf, const typename Cx<T>::type *tw,
                                         const ZParams<T> &zp, int kx0, int y, int tid, bool act) {
  using V = typename Cx<T>::type;
  constexpr int NTHR = S::R1 * B * (JOINT ? MS : 1);
  constexpr int NP = MS * (MS + 1) / 2;
  constexpr int H = N / 2;
  static_assert(N % 2 == 0, "rows pair up as (z, N - z)");
  constexpr int NIT = (H * B + NTHR - 1) / NTHR;
  constexpr int D = NIT < ZPF ? NIT : ZPF;
  const int m = g.m;
  const int np = m * (m + 1) / 2;
  const int bw = min(B, g.Nh - kx0);
  const bool full = MODE == MODE_F && zp.L != nullptr;
  const long long zstride = (long long)g.N1 * g.Nhp;
  const long long col = (long long)y * g.Nhp + kx0;
  const int OR = oct_row(g);
  const long long orow = (long long)(y <= g.N1 / 2 ? y : g.N1 - y) * (H + 1) * OR + kx0;  // octant row kz = 0
  T tq[D][NP];     // chi - 1 of each pair
  T sq[D][MS];     // beta/eps0 s_i, MODE_F
  V lq[D][2];      // long-range values of rows z and N - z, MODE_F
  auto load = [&](int r, int b, T *tv, T *sv) {
    const long long o = orow + (long long)r * OR + b;
#pragma unroll
    for (int q = 0; q < NP; ++q)
      if (q < np) tv[q] = __ldg(&zp.kt[q * zp.oct + o]);
    if (full && zp.ks != nullptr) {
#pragma unroll
      for (int ii = 0; ii < MS; ++ii)
        if (ii < m) sv[ii] = __ldg(&zp.ks[ii * zp.oct + o]);
    }
  };
  auto fetch = [&](int it, int slot) {
    const int e = tid + it * NTHR;
    const int r = e / B, b = e % B;
    if (!act || e >= H * B || b >= bw) return;
    load(r, b, tq[slot], sq[slot]);
    if (full) {
      lq[slot][0] = __ldg(&zp.L[r * zstride + col + b]);
      lq[slot][1] = __ldg(&zp.L[(r == 0 ? H : N - r) * zstride + col + b]);
    }
  };
  auto contract = [&](int e, const T *xv, const T *sv, V Lk) {
    V c[MS];
#pragma unroll
    for (int j = 0; j < MS; ++j)
      if (j < m) c[j] = buf[j * N * B + e];
    if (full) {
#pragma unroll
      for (int j = 0; j < MS; ++j)
        if (j < m) { c[j].x -= zp.a[j] * Lk.x; c[j].y -= zp.a[j] * Lk.y; }
    }
#pragma unroll
    for (int ii = 0; ii < MS; ++ii) {
      if (ii < m) {
        V t;
        t.x = T(0); t.y = T(0);
#pragma unroll
        for (int j = 0; j < MS; ++j) {
          if (j < m) {
            const T x = xv[ii >= j ? ii * (ii + 1) / 2 + j : j * (j + 1) / 2 + ii];
            t.x += x * c[j].x;
            t.y += x * c[j].y;
          }
        }
        if (full) {
          T bb = zp.bconst[ii];
          if (zp.ks != nullptr) bb += sv[ii];
          t.x -= bb * Lk.x;
          t.y -= bb * Lk.y;
        }
        buf[ii * N * B + e] = t;
      }
    }
  };
#pragma unroll
  for (int s = 0; s < D; ++s) fetch(s, s);
  if (JOINT) fft2g<N, MS * B, NTHR, false, true, LayCol<N, B>, S>(buf, tw, tid, act);
  else
    for (int s = 0; s < m; ++s) fft2g<N, B, NTHR, false, true, LayCol<N, B>, S>(buf + s * N * B, tw, tid, act);
#pragma unroll
  for (int it = 0; it < NIT; ++it) {
    const int slot = it % D;
    const int e = tid + it * NTHR;
    const int r = e / B, b = e % B;
    if (act && e < H * B && b < bw) {
      contract(e, tq[slot], sq[slot], lq[slot][0]);
      if (r == 0) load(H, b, tq[slot], sq[slot]);
      contract((r == 0 ? H : N - r) * B + b, tq[slot], sq[slot], lq[slot][1]);
    }
    if (it + D < NIT) fetch(it + D, slot);
  }
  __syncthreads();
  if (JOINT) fft2g<N, MS * B, NTHR, true, true, LayCol<N, B>, S>(buf, tw, tid, act);
  else
    for (int s = 0; s < m; ++s) fft2g<N, B, NTHR, true, true, LayCol<N, B>, S>(buf + s * N * B, tw, tid, act);
}
// ---- the fused z tile
//
// Forward transform, contraction and inverse transform of the m site columns
// with the middle of all three in registers.  With N = R1 R2, n = R2 n1 + n2
// and k = k1 + R1 k2,
//
//   A  per (site, n2, column): R1-point DFT over n1, times W^(n2 k1), back in
//      place (rows R2 k1 + n2);
//   M  per (k1, column): the R2-point DFTs over n2 of all m sites give
//      X[k1 + R1 k2] for every k2 in registers; contract each k with chi - 1;
//      the inverse R2-point DFTs over k2, times W^(-n2 k1), back in place;
//   E  per (site, n2, column): inverse R1-point DFT over k1, back in place.
//
// Every step reads and writes the thread's own rows, so a tile takes three
// shared-memory round trips and three barriers, where two whole transforms
// per site and a separate contraction took five round trips and 6 m + 1
// barriers: with four 128-thread CTAs per SM the pass was bound by those
// barriers and the latency behind them (2.4 of 6.5 TB/s), not by memory.
// J / F passes before -> after, us: 256^3 FP32 169 / 234 -> 127 / 201, FP64
// 341 / 474 -> 245 / 315; 96^3 FP32 21.9 / 26.0 -> 11.0 / 17.7, FP64 32.5 /
// 42.0 -> 17.3 / 22.4; 512^3 FP32 1923 / 4195 -> 1426 / 2958 (half-width tiles).  What is left is
// the FP64 units (FP64) and twelve resident warps per SM (FP32).
template <typename T, int N> struct ZFused {
  // R2 bounds the registers of M (m R2 complex values): at most 18 in FP32, 9
  // in FP64; R1 those of A and E: at most 32.  FP64 columns of 324 points and
  // more have no such pair and keep the separate transforms.
  static constexpr bool f64 = sizeof(T) == 8;
  static constexpr int R2 =
      f64 ? (N == 32 ? 4 : N == 36 || N == 54 ? 6 : N % 9 == 0 && N > 100 ? 9 : N % 8 == 0 ? 8 : 6)
          : N == 32 ? 4 : N == 36 || N == 48 || N == 54 || N == 72 ? 6 : N == 64 || N == 96 || N == 128 ? 8
          : N == 108 || N == 144 || N == 162 ? 9 : N == 192 || N == 216 || N == 324 ? 12 : N == 486 ? 18 : 16;
  static constexpr int R1 = N / R2;
  static constexpr bool on = R1 * R2 == N && R1 <= 32;
  // chi - 1 (and in MODE_F the long-range values) of the tile staged in shared
  // memory, where the tile leaves room
  static constexpr bool stage = N <= 288;
};

// Shared memory of a tile's staged values: chi - 1 [m(m+1)/2][N/2 + 1][B] and,
// in MODE_F, beta/eps0 s_i [m][N/2 + 1][B] and the long-range field [N][B].
template <typename T, int MODE, int N, int B> __host__ __device__ constexpr size_t zf_stage_bytes(int m) {
  return !(ZFused<T, N>::on && ZFused<T, N>::stage)
             ? 0
             : sizeof(T) * ((size_t)(m * (m + 1) / 2 + (MODE == MODE_F ? m : 0)) * (N / 2 + 1) * B +
                            (MODE == MODE_F ? (size_t)2 * N * B : 0));
}

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Issues the copies of the tile's staged values, which land while the tile
// is loaded and A runs: every thread waits for its own before the barrier
// that follows A.  The long-range rows end at Nhp (even, so whole 16-byte
// pieces in FP32 and FP64); what lies beyond is not read (M skips columns
// past Nh).
template <typename T, int MODE, int N, int B, int NTHR>
__device__ __forceinline__ void zf_stage(const Geo &g, const ZParams<T> &zp, int kx0, int y, T *tab) {
  if constexpr (ZFused<T, N>::on && ZFused<T, N>::stage) {
    using V = typename Cx<T>::type;
    constexpr int H2 = N / 2 + 1;
    constexpr int E16 = 16 / (int)sizeof(T);
    constexpr int PER = B / E16;  // 16-byte pieces per row
    static_assert(PER >= 1, "a table row is at least one 16-byte piece");
    const int OR = oct_row(g);
    const int np = g.m * (g.m + 1) / 2;
    const long long o = (long long)(y <= g.N1 / 2 ? y : g.N1 - y) * H2 * OR + kx0;
    for (int q = 0; q < np + (MODE == MODE_F && zp.ks ? g.m : 0); ++q) {
      const T *src = (q < np ? zp.kt + q * zp.oct : zp.ks + (q - np) * zp.oct) + o;
      for (int e = threadIdx.x; e < H2 * PER; e += NTHR) {
        const int r = e / PER, c = (e % PER) * E16;
        cp_async16(tab + ((size_t)q * H2 + r) * B + c, src + (long long)r * OR + c);
      }
    }
    if (MODE == MODE_F && zp.L) {
      V *ls = reinterpret_cast<V *>(tab + (size_t)(np + g.m) * H2 * B);
      for (int e = threadIdx.x; e < N * 2 * PER; e += NTHR) {
        const int z = e / (2 * PER), c = (e % (2 * PER)) * E16 / 2;
        if (kx0 + c < g.Nhp) cp_async16(ls + z * B + c, zp.L + ((long long)z * g.N1 + y) * g.Nhp + kx0 + c);
      }
    }
  }
}

template <typename T, int MODE, int N, int B, int MS, int NTHR>
__device__ __forceinline__ void z_tile_f(const Geo &g, typename Cx<T>::type *buf, const typename Cx<T>::type *tw,
                                         const T *tab, const ZParams<T> &zp, int kx0, int y) {
  using V = typename Cx<T>::type;
  using Z = ZFused<T, N>;
  constexpr int R1 = Z::R1, R2 = Z::R2;
  constexpr int NP = MS * (MS + 1) / 2;
  constexpr int H2 = N / 2 + 1;
  const int tid = threadIdx.x;
  const int m = g.m;
  const int np = m * (m + 1) / 2;
  const bool full = MODE == MODE_F && zp.L != nullptr;
  // A
#pragma unroll 1
  for (int w = tid; w < m * R2 * B; w += NTHR) {
    const int col = w % B, n2 = (w / B) % R2, s = w / (B * R2);
    V *p = buf + s * N * B + n2 * B + col;
    V u[R1];
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) u[n1] = p[n1 * R2 * B];
    RDft<R1, false, V>::run(u, tw, N / R1);
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) p[k1 * R2 * B] = k1 == 0 ? u[0] : cmul(u[k1], tw[n2 * k1]);
  }
  if constexpr (Z::stage) cp_async_wait_all();
  __syncthreads();
  // M
#pragma unroll 1
  for (int w = tid; w < R1 * B; w += NTHR) {
    const int col = w % B, k1 = w / B;
    V u[MS][R2];
#pragma unroll
    for (int s = 0; s < MS; ++s) {
      if (s < m) {
        const V *p = buf + s * N * B + k1 * R2 * B + col;
#pragma unroll
        for (int n2 = 0; n2 < R2; ++n2) u[s][n2] = p[n2 * B];
        RDft<R2, false, V>::run(u[s], tw, N / R2);
      } else {
#pragma unroll
        for (int n2 = 0; n2 < R2; ++n2) u[s][n2].x = u[s][n2].y = T(0);
      }
    }
    const bool valid = kx0 + col < g.Nh;
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) {
      const int z = k1 + R1 * k2;
      const int zz = z <= N / 2 ? z : N - z;
      T x[NP];
      const long long o = ((long long)(y <= g.N1 / 2 ? y : g.N1 - y) * H2 + zz) * oct_row(g) + kx0 + col;
#pragma unroll
      for (int q = 0; q < NP; ++q)
        if (q < np) x[q] = Z::stage ? tab[((size_t)q * H2 + zz) * B + col] : __ldg(&zp.kt[q * zp.oct + o]);
        else x[q] = T(0);
      V Lk;
      Lk.x = Lk.y = T(0);
      if (full && valid)
        Lk = Z::stage ? reinterpret_cast<const V *>(tab + (size_t)(np + m) * H2 * B)[z * B + col]
                      : __ldg(&zp.L[((long long)z * g.N1 + y) * g.Nhp + kx0 + col]);
      V c[MS];
#pragma unroll
      for (int j = 0; j < MS; ++j) {
        c[j] = u[j][k2];
        if (full && j < m) { c[j].x -= zp.a[j] * Lk.x; c[j].y -= zp.a[j] * Lk.y; }
      }
#pragma unroll
      for (int i = 0; i < MS; ++i) {
        V t;
        t.x = T(0); t.y = T(0);
#pragma unroll
        for (int j = 0; j < MS; ++j) {
          const T xv = x[i >= j ? i * (i + 1) / 2 + j : j * (j + 1) / 2 + i];
          t.x += xv * c[j].x;
          t.y += xv * c[j].y;
        }
        if (full && i < m) {
          T bb = zp.bconst[i];
          if (zp.ks != nullptr)
            bb += Z::stage ? tab[((size_t)(np + i) * H2 + zz) * B + col] : __ldg(&zp.ks[i * zp.oct + o]);
          t.x -= bb * Lk.x;
          t.y -= bb * Lk.y;
        }
        u[i][k2] = t;
      }
    }
#pragma unroll
    for (int s = 0; s < MS; ++s) {
      if (s < m) {
        V *p = buf + s * N * B + k1 * R2 * B + col;
        RDft<R2, true, V>::run(u[s], tw, N / R2);
#pragma unroll
        for (int n2 = 0; n2 < R2; ++n2) p[n2 * B] = n2 == 0 ? u[s][0] : cmul(u[s][n2], cconj(tw[n2 * k1]));
      }
    }
  }
  __syncthreads();
  // E
#pragma unroll 1
  for (int w = tid; w < m * R2 * B; w += NTHR) {
    const int col = w % B, n2 = (w / B) % R2, s = w / (B * R2);
    V *p = buf + s * N * B + n2 * B + col;
    V u[R1];
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) u[k1] = p[k1 * R2 * B];
    RDft<R1, true, V>::run(u, tw, N / R1);
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) p[n1 * R2 * B] = u[n1];
  }
  __syncthreads();
}

// Threads of a z-pass CTA.
template <typename T, int N, int B> __host__ __device__ constexpr int z_threads() {
  return ZFused<T, N>::on ? (ZFused<T, N>::R1 * B + 31) / 32 * 32 : SplitY<N>::R1 * B;
}
template <typename T, int MODE, int N, int B, int MS>
__device__ __forceinline__ void z_tile(const Geo &g, typename Cx<T>::type *buf, const typename Cx<T>::type *tw,
                                       const T *tab, const ZParams<T> &zp, int kx0, int y) {
  if constexpr (ZFused<T, N>::on)
    z_tile_f<T, MODE, N, B, MS, z_threads<T, N, B>()>(g, buf, tw, tab, zp, kx0, y);
  else
    z_tile_g<T, MODE, N, B, MS, false, zpf_default<T, MODE>(), SplitY<N>>(g, buf, tw, zp, kx0, y, (int)threadIdx.x, true);
}
// Rows of the pass in launch order: y and N1 - y, which share their chi - 1
// rows, next to one another (0, 1, N1 - 1, 2, N1 - 2, ...).
__device__ __forceinline__ int z_row(int i, int N1) { return i == 0 ? 0 : ((i & 1) ? (i + 1) / 2 : N1 - i / 2); }

// CTAs per SM that the z pass's registers are bounded for: as many as its
// shared memory admits at m = 3 (3 at 256 points in FP32), while each thread
// keeps the m R2 complex values of M and about 72 registers beside them.
template <typename T, int MODE, int N, int B> __host__ __device__ constexpr int z_min_ctas() {
  if (!ZFused<T, N>::on) return sizeof(T) == 4 ? 4 : 1;
  constexpr int w = sizeof(T) / 4;
  const int smem = (int)(sizeof(T) * 2 * (3 * N * B + N) + zf_stage_bytes<T, MODE, N, B>(3)) + 16 + 1024;
  const int by_smem = 228 * 1024 / smem;
  const int by_regs = 65536 / (z_threads<T, N, B>() * (3 * ZFused<T, N>::R2 * 2 * w + 72));
  const int c = by_smem < by_regs ? by_smem : by_regs;
  return c < 1 ? 1 : c;
}

// z pass: the m [N][B] tiles of one (ky, kx-block) by TMA, forward transform,
// OZ contraction (+ long-range terms in MODE_F), inverse transform, TMA out.
// tm: W as {2 Nhp, N1, m N2} scalars, box {2B, 1, N2}.
template <typename T, int MODE, int N, int B, int MS>
__global__ void __launch_bounds__((z_threads<T, N, B>()), (z_min_ctas<T, MODE, N, B>()))
    k_z_s(Geo g, const __grid_constant__ CUtensorMap tm, const typename Cx<T>::type *__restrict__ twg, ZParams<T> zp,
          int *__restrict__ err) {
  using V = typename Cx<T>::type;
  constexpr int NTHR = z_threads<T, N, B>();
  static_assert(tma_tile_ok<V, N, B>(), "every box starts on a 128-byte boundary");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int m = g.m;
  V *buf = reinterpret_cast<V *>(smem_raw);
  V *tw = buf + m * N * B;
  T *tab = reinterpret_cast<T *>(tw + N);
  uint64_t *bar = reinterpret_cast<uint64_t *>(reinterpret_cast<unsigned char *>(tab) + zf_stage_bytes<T, MODE, N, B>(m));
  const int tid = threadIdx.x;
  const int kx0 = blockIdx.x * B, y = z_row(blockIdx.y, g.N1);
  if (tid == 0) mbar_init(bar, 1);
  __syncthreads();
  if (tid == 0) {
    mbar_expect_tx(bar, (uint32_t)(m * N * B * sizeof(V)));
    for (int s = 0; s < m; ++s)
#pragma unroll
      for (int c = 0; c < N; c += tma_rows(N)) tma_load_3d(buf + s * N * B + c * B, &tm, bar, 2 * kx0, y, s * g.N2 + c);
  }
  zf_stage<T, MODE, N, B, NTHR>(g, zp, kx0, y, tab);
  for (int q = tid; q < N; q += NTHR) tw[q] = twg[q];
  if (!cta_wait_tile(bar, 0, kMbarPolls, err, 2)) {
    cp_async_wait_all();
    return;
  }
  z_tile<T, MODE, N, B, MS>(g, buf, tw, tab, zp, kx0, y);
  fence_proxy_async();
  __syncthreads();
  if (tid == 0) {
    for (int s = 0; s < m; ++s)
#pragma unroll
      for (int c = 0; c < N; c += tma_rows(N)) tma_store_3d(&tm, buf + s * N * B + c * B, 2 * kx0, y, s * g.N2 + c);
    tma_commit();
    tma_wait_read0();
  }
}

// The z pass from persistent CTAs with two tile buffers: the TMA load of the
// next tile is in flight while the current one is transformed, and the
// store of a tile drains while the next is transformed.  Tiles t =
// blockIdx.x, blockIdx.x + gridDim.x, ... (kx-block t % nkx, ky t / nkx).
template <typename T, int MODE, int N, int B, int MS>
__global__ void __launch_bounds__(z_threads<T, N, B>())
    k_z_sp(Geo g, const __grid_constant__ CUtensorMap tm, const typename Cx<T>::type *__restrict__ twg, ZParams<T> zp,
           int *__restrict__ err) {
  using V = typename Cx<T>::type;
  constexpr int NTHR = z_threads<T, N, B>();
  static_assert(tma_tile_ok<V, N, B>(), "every box starts on a 128-byte boundary");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int m = g.m;
  V *bufs[2];
  bufs[0] = reinterpret_cast<V *>(smem_raw);
  bufs[1] = bufs[0] + m * N * B;
  V *tw = bufs[1] + m * N * B;
  T *tab = reinterpret_cast<T *>(tw + N);
  uint64_t *bar = reinterpret_cast<uint64_t *>(reinterpret_cast<unsigned char *>(tab) + zf_stage_bytes<T, MODE, N, B>(m));
  const int tid = threadIdx.x;
  const int nkx = (g.Nh + B - 1) / B;
  const int ntile = nkx * g.N1;
  const uint32_t bytes = (uint32_t)(m * N * B * sizeof(V));
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
  }
  __syncthreads();
  int t = blockIdx.x;
  if (tid == 0 && t < ntile) {
    mbar_expect_tx(&bar[0], bytes);
    for (int s = 0; s < m; ++s)
#pragma unroll
      for (int c = 0; c < N; c += tma_rows(N))
        tma_load_3d(bufs[0] + s * N * B + c * B, &tm, &bar[0], 2 * (t % nkx) * B, t / nkx, s * g.N2 + c);
  }
  for (int q = tid; q < N; q += NTHR) tw[q] = twg[q];
  for (int it = 0; t < ntile; t += gridDim.x, ++it) {
    const int cur = it & 1;
    const int tn = t + gridDim.x;
    if (tid == 0 && tn < ntile) {
      // the other buffer's last store must have read shared memory first
      tma_wait_read0();
      mbar_expect_tx(&bar[cur ^ 1], bytes);
      for (int s = 0; s < m; ++s)
#pragma unroll
        for (int c = 0; c < N; c += tma_rows(N))
          tma_load_3d(bufs[cur ^ 1] + s * N * B + c * B, &tm, &bar[cur ^ 1], 2 * (tn % nkx) * B, tn / nkx,
                      s * g.N2 + c);
    }
    const int kx0 = (t % nkx) * B, y = t / nkx;
    zf_stage<T, MODE, N, B, NTHR>(g, zp, kx0, y, tab);
    const bool ok = mbar_wait(&bar[cur], (uint32_t)((it >> 1) & 1), kMbarPolls);
    if (__syncthreads_or(!ok)) {
      cp_async_wait_all();
      // a CTA-uniform exit: both buffers' loads (this tile's and the
      // prefetch of the next) get one more bounded wait, and the stores
      // drain, before the CTA leaves
      if (tid == 0) {
        atomicExch(err, 2);
        mbar_wait(&bar[cur], (uint32_t)((it >> 1) & 1), kMbarPolls);
        if (tn < ntile) mbar_wait(&bar[cur ^ 1], (uint32_t)(((it + 1) >> 1) & 1), kMbarPolls);
        tma_wait0();
      }
      __syncthreads();
      return;
    }
    z_tile<T, MODE, N, B, MS>(g, bufs[cur], tw, tab, zp, kx0, y);
    fence_proxy_async();
    __syncthreads();
    if (tid == 0) {
      for (int s = 0; s < m; ++s)
#pragma unroll
        for (int c = 0; c < N; c += tma_rows(N))
          tma_store_3d(&tm, bufs[cur] + s * N * B + c * B, 2 * kx0, y, s * g.N2 + c);
      tma_commit();
    }
  }
  if (tid == 0) tma_wait0();
}

}  // namespace rism
