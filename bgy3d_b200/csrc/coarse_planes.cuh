// coarse_planes.cuh -- the persistent coarse GMRES (coarse_pk.cuh) in plane
// form: every CTA owns whole (site, z) planes, so that the y transforms ride
// in the x phases and a step has three grid barriers,
//
//   XY   V_j -= sum_{i<j} c_i V_i (with its |.|^2 partials), c'_H V_j, r2c
//        along x, forward along y, one contiguous store of the plane of W;
//   Z    along z, the OZ contraction, inverse along z;
//   YXI  one contiguous load of the plane, inverse along y, c2r along x,
//        V_{j+1} = (X / N - V_j) / s_j and the dot partials <V_i, V_{j+1}>.
//
// The phases are chains of L2 round trips and CTA barriers over little data (a
// 64^3 plane is 16 KB), and a grid barrier's acquire drops the L1 cache, so
// what the x phases read again in every step is kept in shared memory: the
// rows of the first NRES basis vectors that belong to the CTA's first plane.
// Up to 48^3 there are no more planes than SMs, the CTA has an SM to itself
// and the whole basis is resident (NRES = 17) beside c'_H; only W goes
// through L2.  Larger grids have more planes than SMs, two CTAs per SM and
// room for a part of the basis; the rest, and the further planes of a CTA
// whose grid has fewer CTAs than planes, are read from global memory.
//
// The transforms leave out the reordering between their two steps (the x
// untangling and the z phase index the permuted order instead), the steps next
// to W move between registers and global memory directly, and the reductions
// are one warp per value with its partials in flight together: an item of XY or
// YXI has six CTA barriers, a round of Z tiles five, and the kernels up to 48^3
// spill nothing, the others 60 to 252 bytes a thread.  16 steps, us, before -> after: 32^3 298 -> 204, 36^3 364 -> 209, 48^3
// 489 -> 256, 54^3 532 -> 390, 64^3 628 -> 440, 72^3 1117 -> 630, 96^3 2056 ->
// 1463.  What is left: the grid barrier (1.3 us, three per step), two or three
// L2 round trips per phase, and above 48^3 the rest of the basis through L2 on
// SMs that own two planes.
#pragma once
#include "coarse_pk.cuh"

namespace rism {

// Complex values per row of W's planes: Nhp = M + 1 rounded up to even.
template <int M> __host__ __device__ constexpr int pl_ncp() { return (M + 2) & ~1; }

// Splits of the row and column transforms.
template <int M> using PlRow = SplitRow<M>;
template <int N> using PlCol = SplitSq<N>;

template <int M> struct PlShape {
  static constexpr int N = 2 * M;
  // whole basis resident, one CTA per SM: planes of up to 9.2 KB, at most 144
  static constexpr bool res = M <= 24;
  static constexpr int THR = res ? 512 : 288;
  static constexpr int PER_SM = res ? 1 : 2;
  static constexpr int NV = M * M;  // float4 per plane of a basis vector
  static constexpr size_t plane = sizeof(float4) * NV;
  static constexpr size_t xs = sizeof(float2) * (size_t)N * (LayRow<M, PlRow<M>::R2>::RS + pl_ncp<M>());
  static constexpr int ZG = PlCol<N>::R1 * kPkBz * 3;  // threads of a z tile
  static constexpr int ZGPC = THR / ZG;                // z tiles at once
  static constexpr size_t zs = sizeof(float2) * (size_t)ZGPC * 3 * N * kPkBz;
  static constexpr size_t tile = ((xs > zs ? xs : zs) + 15) & ~(size_t)15;
  static constexpr size_t tw = sizeof(float2) * (size_t)(M + M % 2 + N);
  // 228 KB per SM less 1 KB reserved and the static shared memory per CTA
  static constexpr size_t room = (size_t)(228 * 1024) / PER_SM - 1024 - (res ? 6144 : 4352) - tw - tile;
  static constexpr int fit = (int)(room / plane);
  static constexpr int NRES = res ? kPkMaxSteps + 1 : (fit < kPkMaxSteps + 1 ? fit : kPkMaxSteps + 1);
  static constexpr bool dres = fit > NRES;  // c'_H of the first plane resident too
  static constexpr size_t smem = tw + tile + plane * (NRES + (dres ? 1 : 0));
  static_assert(!res || fit >= NRES, "the whole basis fits");
};

// The basis of one item: vector i < nres in shared memory, the others (and all
// of an item without residency) in global memory at `base`.
template <int M> struct PlBasis {
  float4 *res;        // [NRES][NV]
  float *const *V;
  long long base;     // first value of the item
  int nres;
  __device__ __forceinline__ float4 *at(int i) const {
    return i < nres ? res + (size_t)i * PlShape<M>::NV : reinterpret_cast<float4 *>(V[i] + base);
  }
};

// Basis vectors whose loads a thread keeps in flight together.
template <int CNT> __host__ __device__ constexpr int pl_group() { return CNT <= 2 ? 4 : 2; }

template <int M>
__device__ __forceinline__ void pl_xy(const PkArgs &a, float *const *V, float4 *res, const float4 *dres, int j,
                                      const float *cf, bool fft, float2 *buf, const float2 *tw, const float2 *twy,
                                      double &nrm2) {
  using S = PlShape<M>;
  constexpr int N = S::N, THR = S::THR, NV = S::NV;
  using PX = PlRow<M>;
  using PY = PlCol<N>;
  using Lay = LayRow<M, PX::R2>;
  constexpr int NCP = pl_ncp<M>();
  float2 *T = buf + N * Lay::RS;  // the column tile
  constexpr int CNT = (NV + THR - 1) / THR;
  constexpr int GV = pl_group<CNT>();
  constexpr int H = M / 2 + 1;
  const int tid = threadIdx.x;
  const int nitems = a.g.m * N;
  for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
    const bool first = item == (int)blockIdx.x;
    const PlBasis<M> B{res, V, (long long)item * 4 * NV, first ? S::NRES : 0};
    float4 *w = B.at(j);
    const float4 *ds = S::dres && first ? dres : reinterpret_cast<const float4 *>(a.d + B.base);
    float4 x[CNT];
#pragma unroll
    for (int it = 0; it < CNT; ++it) {
      const int e = tid + it * THR;
      x[it] = e < NV ? w[e] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (j > 0) {
      // the basis vectors in groups, all loads of a group in flight
      for (int i0 = 0; i0 < j; i0 += GV) {
        float4 b[GV][CNT];
#pragma unroll
        for (int u = 0; u < GV; ++u) {
          const float4 *p = B.at(i0 + u < j ? i0 + u : i0);
#pragma unroll
          for (int it = 0; it < CNT; ++it) {
            const int e = tid + it * THR;
            b[u][it] = e < NV ? p[e] : make_float4(0.f, 0.f, 0.f, 0.f);
          }
        }
#pragma unroll
        for (int u = 0; u < GV; ++u) {
          const float c = i0 + u < j ? cf[i0 + u] : 0.f;
#pragma unroll
          for (int it = 0; it < CNT; ++it) {
            x[it].x -= c * b[u][it].x;
            x[it].y -= c * b[u][it].y;
            x[it].z -= c * b[u][it].z;
            x[it].w -= c * b[u][it].w;
          }
        }
      }
#pragma unroll
      for (int it = 0; it < CNT; ++it) {
        const int e = tid + it * THR;
        if (e < NV) {
          w[e] = x[it];
          nrm2 += (double)(x[it].x * x[it].x + x[it].y * x[it].y + x[it].z * x[it].z + x[it].w * x[it].w);
        }
      }
    }
    if (!fft) continue;
#pragma unroll
    for (int it = 0; it < CNT; ++it) {
      const int e = tid + it * THR;
      if (e >= NV) break;
      const float4 d = ds[e];
      // rows may end inside a float4 (odd M)
      buf[Lay::at((2 * e) % M, (2 * e) / M)] = make_float2(d.x * x[it].x, d.y * x[it].y);
      buf[Lay::at((2 * e + 1) % M, (2 * e + 1) / M)] = make_float2(d.z * x[it].z, d.w * x[it].w);
    }
    __syncthreads();
    // along x: step 1, step 2 in place (index k1 + R1 k2 at PX::pos)
    for (int q = tid; q < N * PX::R2; q += THR) {
      const int row = q / PX::R2, n2 = q % PX::R2;
      float2 u[PX::R1];
#pragma unroll
      for (int n1 = 0; n1 < PX::R1; ++n1) u[n1] = buf[Lay::at(PX::R2 * n1 + n2, row)];
      fwd_step1<PX>(u, n2, tw);
#pragma unroll
      for (int k1 = 0; k1 < PX::R1; ++k1) buf[Lay::at(PX::R2 * k1 + n2, row)] = u[k1];
    }
    __syncthreads();
    for (int q = tid; q < N * PX::R1; q += THR) {
      const int row = q / PX::R1, k1 = q % PX::R1;
      float2 u[PX::R2];
#pragma unroll
      for (int n2 = 0; n2 < PX::R2; ++n2) u[n2] = buf[Lay::at(PX::R2 * k1 + n2, row)];
      fwd_step2<PX>(u, tw);
#pragma unroll
      for (int k2 = 0; k2 < PX::R2; ++k2) buf[Lay::at(PX::R2 * k1 + k2, row)] = u[k2];
    }
    __syncthreads();
    for (int e = tid; e < N * H; e += THR) {
      const int row = e / H, kk = e % H;
      const float2 zk = buf[Lay::at(perm_pos<PX>(kk), row)];
      const float2 zm = buf[Lay::at(perm_pos<PX>(kk == 0 ? 0 : M - kk), row)];
      float2 E, O;
      E.x = (zk.x + zm.x) * 0.5f;
      E.y = (zk.y - zm.y) * 0.5f;
      O.x = (zk.y + zm.y) * 0.5f;
      O.y = -(zk.x - zm.x) * 0.5f;
      const float2 wO = cmul(__ldg(&a.post[kk]), O);
      T[row * NCP + kk] = cadd(E, wO);
      if (M - kk != kk) T[row * NCP + M - kk] = cconj(csub(E, wO));
    }
    __syncthreads();
    // along y: step 1 in place, step 2 from registers to W (row R2 k1 + k2
    // holds ky = k1 + R1 k2, which the Z phase undoes)
    for (int q = tid; q < PY::R2 * (M + 1); q += THR) {
      const int col = q % (M + 1), n2 = q / (M + 1);
      float2 u[PY::R1];
#pragma unroll
      for (int n1 = 0; n1 < PY::R1; ++n1) u[n1] = T[(PY::R2 * n1 + n2) * NCP + col];
      fwd_step1<PY>(u, n2, twy);
#pragma unroll
      for (int k1 = 0; k1 < PY::R1; ++k1) T[(PY::R2 * k1 + n2) * NCP + col] = u[k1];
    }
    __syncthreads();
    float2 *Wp = a.W + (long long)item * N * NCP;
    for (int q = tid; q < PY::R1 * (M + 1); q += THR) {
      const int col = q % (M + 1), k1 = q / (M + 1);
      float2 u[PY::R2];
#pragma unroll
      for (int n2 = 0; n2 < PY::R2; ++n2) u[n2] = T[(PY::R2 * k1 + n2) * NCP + col];
      fwd_step2<PY>(u, twy);
#pragma unroll
      for (int k2 = 0; k2 < PY::R2; ++k2) Wp[(PY::R2 * k1 + k2) * NCP + col] = u[k2];
    }
    __syncthreads();  // the tiles are refilled by the next item
  }
}

template <int M>
__device__ __forceinline__ void pl_yxi(const PkArgs &a, float *const *V, float4 *res, int j, float sc, float sub,
                                       float2 *buf, const float2 *tw, const float2 *twy,
                                       double (*sdot)[PlShape<M>::THR / 32]) {
  using S = PlShape<M>;
  constexpr int N = S::N, THR = S::THR, NV = S::NV;
  using PX = PlRow<M>;
  using PY = PlCol<N>;
  using Lay = LayRow<M, PX::R2>;
  constexpr int NCP = pl_ncp<M>();
  float2 *T = buf + N * Lay::RS;
  constexpr int CNT = (NV + THR - 1) / THR;
  constexpr int GV = pl_group<CNT>();
  constexpr int H = M / 2 + 1;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int nitems = a.g.m * N;
  const int nv = j + 1;
  for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
    const PlBasis<M> B{res, V, (long long)item * 4 * NV, item == (int)blockIdx.x ? S::NRES : 0};
    const float2 *Wp = a.W + (long long)item * N * NCP;
    for (int q = tid; q < PY::R1 * (M + 1); q += THR) {
      const int col = q % (M + 1), k1 = q / (M + 1);
      float2 u[PY::R2];
#pragma unroll
      for (int k2 = 0; k2 < PY::R2; ++k2) u[k2] = Wp[(PY::R2 * k1 + k2) * NCP + col];
      inv_step1<PY>(u, k1, twy);
#pragma unroll
      for (int n2 = 0; n2 < PY::R2; ++n2) T[(PY::R2 * k1 + n2) * NCP + col] = u[n2];
    }
    __syncthreads();
    for (int q = tid; q < PY::R2 * (M + 1); q += THR) {
      const int col = q % (M + 1), n2 = q / (M + 1);
      float2 u[PY::R1];
#pragma unroll
      for (int k1 = 0; k1 < PY::R1; ++k1) u[k1] = T[(PY::R2 * k1 + n2) * NCP + col];
      inv_step2<PY>(u, twy);
#pragma unroll
      for (int n1 = 0; n1 < PY::R1; ++n1) T[(PY::R2 * n1 + n2) * NCP + col] = u[n1];
    }
    __syncthreads();
    for (int e = tid; e < N * H; e += THR) {
      const int row = e / H, kk = e % H;
      float2 xk = T[row * NCP + kk];
      float2 xm = T[row * NCP + M - kk];
      if (kk == 0) { xk.y = 0.f; xm.y = 0.f; }  // c2r reads only Re X_0, Re X_{N0/2}
      float2 Aa, D;
      Aa.x = xk.x + xm.x; Aa.y = xk.y - xm.y;
      D.x = xk.x - xm.x;  D.y = xk.y + xm.y;
      const float2 Pp = cmul(D, cconj(__ldg(&a.post[kk])));
      float2 zk, zm;
      zk.x = Aa.x - Pp.y; zk.y = Aa.y + Pp.x;
      zm.x = Aa.x + Pp.y; zm.y = -(Aa.y - Pp.x);
      buf[Lay::at(perm_pos<PX>(kk), row)] = zk;
      if (kk != 0 && M - kk != kk) buf[Lay::at(perm_pos<PX>(M - kk), row)] = zm;
    }
    __syncthreads();
    for (int q = tid; q < N * PX::R1; q += THR) {
      const int row = q / PX::R1, k1 = q % PX::R1;
      float2 u[PX::R2];
#pragma unroll
      for (int k2 = 0; k2 < PX::R2; ++k2) u[k2] = buf[Lay::at(PX::R2 * k1 + k2, row)];
      inv_step1<PX>(u, k1, tw);
#pragma unroll
      for (int n2 = 0; n2 < PX::R2; ++n2) buf[Lay::at(PX::R2 * k1 + n2, row)] = u[n2];
    }
    __syncthreads();
    for (int q = tid; q < N * PX::R2; q += THR) {
      const int row = q / PX::R2, n2 = q % PX::R2;
      float2 u[PX::R1];
#pragma unroll
      for (int k1 = 0; k1 < PX::R1; ++k1) u[k1] = buf[Lay::at(PX::R2 * k1 + n2, row)];
      inv_step2<PX>(u, tw);
#pragma unroll
      for (int n1 = 0; n1 < PX::R1; ++n1) buf[Lay::at(PX::R2 * n1 + n2, row)] = u[n1];
    }
    float4 rin[CNT];
    const float4 *vin = B.at(j);
#pragma unroll
    for (int it = 0; it < CNT; ++it) {
      const int e = tid + it * THR;
      if (e < NV) rin[it] = vin[e];
    }
    __syncthreads();
    float4 o[CNT];
    float4 *vout = B.at(j + 1);
#pragma unroll
    for (int it = 0; it < CNT; ++it) {
      const int e = tid + it * THR;
      o[it] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (e < NV) {
        const float2 z0 = buf[Lay::at((2 * e) % M, (2 * e) / M)];
        const float2 z1 = buf[Lay::at((2 * e + 1) % M, (2 * e + 1) / M)];
        o[it] = make_float4(z0.x * sc - sub * rin[it].x, z0.y * sc - sub * rin[it].y, z1.x * sc - sub * rin[it].z,
                            z1.y * sc - sub * rin[it].w);
        vout[e] = o[it];
      }
    }
    // dots against the basis, GV vectors' loads in flight at a time; each
    // group reduced over the warp (lane 0 adds it to the warp's slot)
    for (int i0 = 0; i0 < nv; i0 += GV) {
      float4 b[GV][CNT];
#pragma unroll
      for (int u = 0; u < GV; ++u) {
        const float4 *p = B.at(i0 + u < nv ? i0 + u : i0);
#pragma unroll
        for (int it = 0; it < CNT; ++it) {
          const int e = tid + it * THR;
          b[u][it] = e < NV ? p[e] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
      double dd[GV];
#pragma unroll
      for (int u = 0; u < GV; ++u) {
        dd[u] = 0.0;
#pragma unroll
        for (int it = 0; it < CNT; ++it)
          dd[u] += (double)(o[it].x * b[u][it].x + o[it].y * b[u][it].y + o[it].z * b[u][it].z +
                            o[it].w * b[u][it].w);
      }
#pragma unroll
      for (int q = 16; q > 0; q >>= 1)
#pragma unroll
        for (int u = 0; u < GV; ++u) dd[u] += __shfl_xor_sync(0xffffffffu, dd[u], q);
#pragma unroll
      for (int u = 0; u < GV; ++u)
        if (lane == 0 && i0 + u < nv) sdot[i0 + u][wid] += dd[u];
    }
    __syncthreads();
  }
}

// Z: tiles of [N][4] columns of the three sites, R1 4 3 threads each, tile t
// to CTA t mod grid first.  Step 1 reads W, the last step writes it, both from
// registers; in between the tile [3][N][4] is in shared memory with row
// R2 k1 + k2 holding kz = k1 + R1 k2.  The chi - 1 values of a thread's rows
// are fetched before step 1.  Every thread of the CTA reaches every barrier.
template <int M> __device__ __forceinline__ void pl_z(const PkArgs &a, float2 *smem, const float2 *tw) {
  using S = PlShape<M>;
  constexpr int N = S::N, B = kPkBz, MS = 3, NG = S::ZG, GPC = S::ZGPC;
  using PZ = PlCol<N>;
  static_assert(GPC >= 1, "a z tile needs at most one CTA of threads");
  constexpr int NP = MS * (MS + 1) / 2;
  constexpr int NIT = (N * B + NG - 1) / NG;
  constexpr int I1 = (PZ::R2 * B * MS + NG - 1) / NG;  // first-step items per thread
  const Geo &g = a.g;
  const int m = g.m, np = m * (m + 1) / 2;
  constexpr int nkx = (M + B) / B;
  constexpr int ntile = nkx * N;
  constexpr int NCP = pl_ncp<M>();
  const int grp = threadIdx.x / NG, tid = threadIdx.x % NG;
  const bool ing = grp < GPC;
  float2 *buf = smem + (ing ? grp : 0) * MS * N * B;
  const int OR = oct_row(g);
  for (int base = blockIdx.x; base < ntile; base += gridDim.x * GPC) {
    const int t = base + grp * gridDim.x;
    const bool act = ing && t < ntile;
    const int kx0 = (t % nkx) * B, y = t / nkx;
    float x[NIT][NP];
    if (act) {
      const int ky = perm_freq<PZ>(y);  // y and z columns are of one length and split
      const float *kt = a.zp.kt + (long long)(ky <= N / 2 ? ky : N - ky) * (N / 2 + 1) * OR + kx0;
#pragma unroll
      for (int it = 0; it < NIT; ++it) {
        const int e = tid + it * NG;
        const int b = e % B, z = perm_freq<PZ>(e / B);
        if (e < N * B) {
#pragma unroll
          for (int q = 0; q < NP; ++q)
            if (q < np) x[it][q] = __ldg(&kt[q * a.zp.oct + (long long)(z <= N / 2 ? z : N - z) * OR + b]);
        }
      }
#pragma unroll
      for (int i = 0; i < I1; ++i) {
        const int q = tid + i * NG;
        const int b = q % B, s = (q / B) % MS, n2 = q / (B * MS);
        if (q >= PZ::R2 * B * MS || s >= m) continue;
        const bool in = kx0 + b < NCP;
        const float2 *w = a.W + ((long long)s * N * N + y) * NCP + kx0 + b;
        float2 u[PZ::R1];
#pragma unroll
        for (int n1 = 0; n1 < PZ::R1; ++n1)
          u[n1] = in ? w[(long long)(PZ::R2 * n1 + n2) * N * NCP] : make_float2(0.f, 0.f);
        fwd_step1<PZ>(u, n2, tw);
#pragma unroll
        for (int k1 = 0; k1 < PZ::R1; ++k1) buf[(s * N + PZ::R2 * k1 + n2) * B + b] = u[k1];
      }
    }
    __syncthreads();
    if (act) {
      // step 2, one item per thread
      const int b = tid % B, s = (tid / B) % MS, k1 = tid / (B * MS);
      if (s < m) {
        float2 u[PZ::R2];
        float2 *p = buf + (s * N + PZ::R2 * k1) * B + b;
#pragma unroll
        for (int n2 = 0; n2 < PZ::R2; ++n2) u[n2] = p[n2 * B];
        fwd_step2<PZ>(u, tw);
#pragma unroll
        for (int k2 = 0; k2 < PZ::R2; ++k2) p[k2 * B] = u[k2];
      }
    }
    __syncthreads();
    if (act) {
#pragma unroll
      for (int it = 0; it < NIT; ++it) {
        const int e = tid + it * NG;
        if (e >= N * B) break;
        float2 c[MS];
#pragma unroll
        for (int s = 0; s < MS; ++s) c[s] = s < m ? buf[s * N * B + e] : make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < MS; ++i) {
          if (i >= m) break;
          float2 o = make_float2(0.f, 0.f);
#pragma unroll
          for (int s = 0; s < MS; ++s) {
            if (s < m) {
              const float xv = x[it][i >= s ? i * (i + 1) / 2 + s : s * (s + 1) / 2 + i];
              o.x += xv * c[s].x;
              o.y += xv * c[s].y;
            }
          }
          buf[i * N * B + e] = o;
        }
      }
    }
    __syncthreads();
    if (act) {
      const int b = tid % B, s = (tid / B) % MS, k1 = tid / (B * MS);
      if (s < m) {
        float2 u[PZ::R2];
        float2 *p = buf + (s * N + PZ::R2 * k1) * B + b;
#pragma unroll
        for (int k2 = 0; k2 < PZ::R2; ++k2) u[k2] = p[k2 * B];
        inv_step1<PZ>(u, k1, tw);
#pragma unroll
        for (int n2 = 0; n2 < PZ::R2; ++n2) p[n2 * B] = u[n2];
      }
    }
    __syncthreads();
    if (act) {
#pragma unroll
      for (int i = 0; i < I1; ++i) {
        const int q = tid + i * NG;
        const int b = q % B, s = (q / B) % MS, n2 = q / (B * MS);
        if (q >= PZ::R2 * B * MS || s >= m) continue;
        float2 u[PZ::R1];
#pragma unroll
        for (int k1 = 0; k1 < PZ::R1; ++k1) u[k1] = buf[(s * N + PZ::R2 * k1 + n2) * B + b];
        inv_step2<PZ>(u, tw);
        float2 *w = a.W + ((long long)s * N * N + y) * NCP + kx0 + b;
        if (kx0 + b < NCP) {
#pragma unroll
          for (int n1 = 0; n1 < PZ::R1; ++n1) w[(long long)(PZ::R2 * n1 + n2) * N * NCP] = u[n1];
        }
      }
    }
    __syncthreads();  // the tile is refilled in the next round
  }
}

// out[v] = sum_{b < nb} part[v * ld + b] for v < nv, one warp per value, in a
// fixed order (identical in every CTA); by the warps w0 .. w0 + nw - 1.
__device__ __forceinline__ void pl_sum(const double *part, int ld, int nb, int nv, double *out, int w0, int nw) {
  const int wid = threadIdx.x / 32 - w0, lane = threadIdx.x & 31;
  if (wid < 0 || wid >= nw) return;
  for (int v = wid; v < nv; v += nw) {
    double s = 0.0;
    for (int b0 = lane; b0 < nb; b0 += 8 * 32) {
      double p[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) p[u] = b0 + 32 * u < nb ? part[(long long)v * ld + b0 + 32 * u] : 0.0;
#pragma unroll
      for (int u = 0; u < 8; ++u) s += p[u];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) out[v] = s;
  }
}

template <int M>
__global__ void __launch_bounds__(PlShape<M>::THR, PlShape<M>::PER_SM) k_coarse_planes(PkArgs a) {
  using S = PlShape<M>;
  constexpr int N = S::N, THR = S::THR, NV = S::NV;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  float2 *twx = reinterpret_cast<float2 *>(smem_raw);
  float2 *twy = twx + M;
  float2 *tile = reinterpret_cast<float2 *>(smem_raw + S::tw);
  float4 *res = reinterpret_cast<float4 *>(smem_raw + S::tw + S::tile);  // [NRES][NV]
  float4 *dres = res + (size_t)S::NRES * NV;                             // c'_H of the first plane
  __shared__ double sH[kPkMaxSteps * (kPkMaxSteps + 1)];
  __shared__ double sS[kPkMaxSteps + 1];  // s_j = |V_j|
  __shared__ double sD[kVecMax];          // summed dot partials
  __shared__ float sC[kPkMaxSteps];       // update coefficients D_i / s_i^2
  __shared__ double sY[kPkMaxSteps];
  __shared__ double sdot[kPkMaxSteps][THR / 32];
  __shared__ float *sV[kPkMaxSteps + 1];  // the basis pointers, indexed at run time
  const int tid = threadIdx.x;
  const int k = a.k;
  const int nitems = a.g.m * N;
  if (tid <= kPkMaxSteps) sV[tid] = a.V[tid];
  if (a.trace && blockIdx.x == 0 && tid == 0) a.trace[0] = global_ns();
  for (int q = tid; q < M; q += THR) twx[q] = a.twx[q];
  for (int q = tid; q < N; q += THR) twy[q] = a.twy[q];  // y and z are of one length
  const float scale = 1.0f / (float)a.g.Nr;
  unsigned gen = 0;
  __syncthreads();  // sV and the twiddles are written before any thread reads them

  // P0: |r|^2, and the resident copies of r and c'_H
  {
    double s2 = 0.0;
    for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
      const bool first = item == (int)blockIdx.x;
      for (int e = tid; e < NV; e += THR) {
        const float4 v = reinterpret_cast<const float4 *>(sV[0])[(long long)item * NV + e];
        if (first && S::NRES > 0) res[e] = v;
        if (first && S::dres) dres[e] = reinterpret_cast<const float4 *>(a.d)[(long long)item * NV + e];
        s2 += (double)(v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w);
      }
    }
    pk_block_sum<THR>(s2, a.pnrm);
  }
  if (!grid_sync(a.bar, ++gen, a.err, a.trace, a.trace_cta)) return;
  pl_sum(a.pnrm, 0, gridDim.x, 1, sD, 0, 1);
  if (tid == 0) sS[0] = sqrt(fmax(sD[0], 0.0));
  __syncthreads();

  for (int j = 0; j <= k; ++j) {
    // the Gram-Schmidt update of V_j against V_0 .. V_{j-1} (coefficients
    // from the dot partials of the last YXI phase), then its transform
    double nrm2 = 0.0;
    if (j > 0) {
      pl_sum(a.pdot, gridDim.x, gridDim.x, j, sD, 0, THR / 32);
      __syncthreads();
      if (tid < j) {
        const double si = sS[tid];
        sH[(j - 1) * (k + 1) + tid] = si > 0.0 ? sD[tid] / si : 0.0;  // h_{i,j-1} = <V_i/s_i, J V_{j-1}/s_{j-1}>
        sC[tid] = si > 0.0 ? (float)(sD[tid] / (si * si)) : 0.f;
      }
      __syncthreads();
    }
    pl_xy<M>(a, sV, res, dres, j, sC, j < k, tile, twx, twy, nrm2);
    if (j > 0) pk_block_sum<THR>(nrm2, a.pnrm + (j & 1) * gridDim.x);
    if (!grid_sync(a.bar, ++gen, a.err, a.trace, a.trace_cta)) return;
    // |V_j| by the last warp (idle in most z tiles); read after the barriers below
    if (j > 0 && tid >= THR - 32) {
      pl_sum(a.pnrm + (j & 1) * gridDim.x, 0, gridDim.x, 1, sD, THR / 32 - 1, 1);
      if (tid == THR - 32) {
        sS[j] = sqrt(fmax(sD[0], 0.0));
        sH[(j - 1) * (k + 1) + j] = sS[j];
      }
    }
    if (j == k) break;
    pl_z<M>(a, tile, twy);
    if (!grid_sync(a.bar, ++gen, a.err, a.trace, a.trace_cta)) return;
    // V_{j+1} = J (V_j / s_j) = (X / N - V_j) / s_j
    const double sj = sS[j];
    const float inv = sj > 0.0 ? (float)(1.0 / sj) : 0.f;
    for (int q = tid; q < kPkMaxSteps * (THR / 32); q += THR) (&sdot[0][0])[q] = 0.0;
    __syncthreads();
    pl_yxi<M>(a, sV, res, j, scale * inv, inv, tile, twx, twy, sdot);
    if (tid <= j) {
      double t = 0.0;
      for (int w = 0; w < THR / 32; ++w) t += sdot[tid][w];
      a.pdot[(long long)tid * gridDim.x + blockIdx.x] = t;
    }
    if (!grid_sync(a.bar, ++gen, a.err, a.trace, a.trace_cta)) return;
  }

  // least squares (every CTA, bitwise alike), then out = sum_j y_j V_j / s_j
  __syncthreads();
  pk_finish(a, sH, sS, sY);
  __syncthreads();
  for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
    const PlBasis<M> B{res, sV, (long long)item * 4 * NV, item == (int)blockIdx.x ? S::NRES : 0};
    for (int e = tid; e < NV; e += THR) {
      float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
      for (int q = 0; q < k; ++q) {
        const float c = (float)sY[q];
        const float4 v = B.at(q)[e];
        o.x += c * v.x; o.y += c * v.y; o.z += c * v.z; o.w += c * v.w;
      }
      reinterpret_cast<float4 *>(a.out + B.base)[e] = o;
    }
  }
  if (a.trace && blockIdx.x == 0 && tid == 0) a.trace[gen + 1] = global_ns();
}

}  // namespace rism
