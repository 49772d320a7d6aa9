// passes_impl.cuh -- definitions of the pass launchers of passes.cuh, for the
// translation units that instantiate them.
#pragma once
#include <algorithm>

#include "passes.cuh"

namespace rism {

template <typename T, int M> constexpr size_t xs_smem() {
  return sizeof(typename Cx<T>::type) * (size_t)(M + x_rx<T, M>() * LayRow<M, SplitRow<M>::R2>::RS);
}
template <typename T, int N> constexpr size_t ys_smem() {
  return sizeof(typename Cx<T>::type) * (size_t)(N * static_B<T>() + N) + 16;
}
template <typename T, int MODE, int N, int B = static_Bz<T>()> size_t zs_smem(int m) {
  return sizeof(typename Cx<T>::type) * (size_t)(m * N * B + N) + zf_stage_bytes<T, MODE, N, B>(m) + 16;
}
template <typename T, int MODE, int N> size_t zsp_smem(int m) {  // two tile buffers, two mbarriers
  return sizeof(typename Cx<T>::type) * (size_t)(2 * m * N * static_Bz<T>() + N) +
         zf_stage_bytes<T, MODE, N, static_Bz<T>()>(m) + 16;
}

template <typename T, int M>
void XPass<T, M>::fwd(int mode, const Geo &g, const T *A, const T *B, const T *t, T p, int closure, V *W,
                      const V *post, const V *tw, cudaStream_t st) {
  constexpr int RX = x_rx<T, M>();
  constexpr size_t sm = xs_smem<T, M>();
  const dim3 grid((unsigned)((g.N1 * g.N2 + RX - 1) / RX), g.m);
  if (mode == MODE_F)
    k_xfwd_s<T, MODE_F, M, RX><<<grid, xfwd_threads<T>(), sm, st>>>(g, A, B, nullptr, p, closure, W, post, tw);
  else if (mode == MODE_S)
    k_xfwd_s<T, MODE_S, M, RX><<<grid, xfwd_threads<T>(), sm, st>>>(g, A, B, t, p, closure, W, post, tw);
  else
    k_xfwd_s<T, MODE_J, M, RX><<<grid, xfwd_threads<T>(), sm, st>>>(g, A, B, nullptr, p, closure, W, post, tw);
}
template <typename T, int M>
void XPass<T, M>::inv(const Geo &g, const V *W, const T *In, T *Out, T scale, T sub, const V *post, const V *tw,
                      NormPartial *part, cudaStream_t st) {
  constexpr int RX = x_rx<T, M>();
  const dim3 grid((unsigned)((g.N1 * g.N2 + RX - 1) / RX), g.m);
  k_xinv_s<T, M, RX><<<grid, kXThreads, xs_smem<T, M>(), st>>>(g, W, In, Out, scale, sub, post, tw, part);
}
template <typename T, int M> void XPass<T, M>::kernels(std::vector<PassKernel> &k) {
  constexpr int RX = x_rx<T, M>();
  k.push_back({(const void *)k_xfwd_s<T, MODE_F, M, RX>, xs_smem<T, M>()});
  k.push_back({(const void *)k_xfwd_s<T, MODE_J, M, RX>, xs_smem<T, M>()});
  k.push_back({(const void *)k_xfwd_s<T, MODE_S, M, RX>, xs_smem<T, M>()});
  k.push_back({(const void *)k_xinv_s<T, M, RX>, xs_smem<T, M>()});
}

template <typename T, int N>
void YPass<T, N>::run(bool inv, const Geo &g, const CUtensorMap &tm, const V *tw, int *err, cudaStream_t st) {
  constexpr int B = static_B<T>();
  const dim3 grid((g.Nh + B - 1) / B, g.N2, g.m);
  if (inv) k_y_s<T, true, N, B><<<grid, SplitY<N>::R1 * B, ys_smem<T, N>(), st>>>(g, tm, tw, err);
  else k_y_s<T, false, N, B><<<grid, SplitY<N>::R1 * B, ys_smem<T, N>(), st>>>(g, tm, tw, err);
}
template <typename T, int N> void YPass<T, N>::kernels(std::vector<PassKernel> &k) {
  constexpr int B = static_B<T>();
  k.push_back({(const void *)k_y_s<T, true, N, B>, ys_smem<T, N>()});
  k.push_back({(const void *)k_y_s<T, false, N, B>, ys_smem<T, N>()});
}

template <int N>
void ZAxis<N>::run(bool inv, const Geo &g, const CUtensorMap &tm, const double2 *tw, int *err, cudaStream_t st) {
  constexpr int B = static_B<double>();
  const dim3 grid((g.Nh + B - 1) / B, g.N1, g.m);
  if (inv) k_y_s<double, true, N, B, true><<<grid, SplitY<N>::R1 * B, ys_smem<double, N>(), st>>>(g, tm, tw, err);
  else k_y_s<double, false, N, B, true><<<grid, SplitY<N>::R1 * B, ys_smem<double, N>(), st>>>(g, tm, tw, err);
}
template <int N> void ZAxis<N>::kernels(std::vector<PassKernel> &k) {
  constexpr int B = static_B<double>();
  k.push_back({(const void *)k_y_s<double, true, N, B, true>, ys_smem<double, N>()});
  k.push_back({(const void *)k_y_s<double, false, N, B, true>, ys_smem<double, N>()});
}

template <typename T, int MODE, int N>
void z_run(int B, bool persistent, const Geo &g, const CUtensorMap &tm, const typename Cx<T>::type *tw,
           const ZParams<T> &zp, int *err, cudaStream_t st) {
  constexpr int BW = static_Bz<T>(), BN = BW / 2;  // wide / narrow tiles
  if constexpr (z_has_variants(N)) {
    if (persistent) {
      int dev = 0, sms = 1, per = 1;
      const size_t sm = zsp_smem<T, MODE, N>(g.m);
      constexpr int thr = z_threads<T, N, BW>();
      cudaGetDevice(&dev);
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_z_sp<T, MODE, N, BW, 3>, thr, sm);
      const int nt = ((g.Nh + BW - 1) / BW) * g.N1;
      k_z_sp<T, MODE, N, BW, 3><<<std::min(std::max(1, per) * sms, nt), thr, sm, st>>>(g, tm, tw, zp, err);
      return;
    }
    if constexpr (sizeof(T) == 4) {
      if (B != BW) {
        const dim3 grid((g.Nh + BN - 1) / BN, g.N1);
        k_z_s<T, MODE, N, BN, 3><<<grid, z_threads<T, N, BN>(), zs_smem<T, MODE, N, BN>(g.m), st>>>(g, tm, tw, zp, err);
        return;
      }
    }
  }
  const dim3 grid((g.Nh + BW - 1) / BW, g.N1);
  k_z_s<T, MODE, N, BW, 3><<<grid, z_threads<T, N, BW>(), zs_smem<T, MODE, N, BW>(g.m), st>>>(g, tm, tw, zp, err);
}
template <typename T, int N>
void ZPass<T, N>::run(int mode, int B, bool persistent, const Geo &g, const CUtensorMap &tm, const V *tw,
                      const ZParams<T> &zp, int *err, cudaStream_t st) {
  if (mode == MODE_F) z_run<T, MODE_F, N>(B, persistent, g, tm, tw, zp, err, st);
  else z_run<T, MODE_J, N>(B, persistent, g, tm, tw, zp, err, st);
}
template <typename T, int MODE, int N> void z_kernels(int m, std::vector<PassKernel> &k) {
  constexpr int BW = static_Bz<T>(), BN = BW / 2;
  k.push_back({(const void *)k_z_s<T, MODE, N, BW, 3>, zs_smem<T, MODE, N, BW>(m)});
  if constexpr (z_has_variants(N)) {
    k.push_back({(const void *)k_z_sp<T, MODE, N, BW, 3>, zsp_smem<T, MODE, N>(m)});
    if constexpr (sizeof(T) == 4) k.push_back({(const void *)k_z_s<T, MODE, N, BN, 3>, zs_smem<T, MODE, N, BN>(m)});
  }
}
template <typename T, int N> void ZPass<T, N>::kernels(int m, std::vector<PassKernel> &k) {
  z_kernels<T, MODE_F, N>(m, k);
  z_kernels<T, MODE_J, N>(m, k);
}

#define RISM_INST_X(M)              \
  template struct XPass<float, M>; \
  template struct XPass<double, M>;
#define RISM_INST_Y(N)              \
  template struct YPass<float, N>; \
  template struct YPass<double, N>; \
  template struct ZAxis<N>;
#define RISM_INST_Z(N)              \
  template struct ZPass<float, N>; \
  template struct ZPass<double, N>;

}  // namespace rism
