// passes.cuh -- launchers of the shape-specialised FFT passes
// (kernels_static.cuh), one struct per axis length and precision.  The
// definitions are in passes_impl.cuh and are instantiated by the passes_*.cu
// translation units, which compile side by side; rism3d.cu only sees the
// declarations here.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <vector>

#include "kernels_static.cuh"

namespace rism {

// Half-row lengths M of the x passes and axis lengths of the y / z passes:
// every grid of 32 .. 512 points (even 2^a 3^b), along each axis.  The
// runtime-length passes (one barrier pair per radix, indices divided at run
// time) are several times slower at every one of them, so a shape is here if
// its two-step split fits registers; axes below 32 points keep them, and so
// does the z pass of more than three solvent sites or a 3D chi.  FP32 J.v, all five passes,
// runtime-length -> here, us: 32^3 48 -> 14, 54^3 98 -> 20, 108^3 373 -> 59,
// 162^3 1265 -> 182, 288^3 6160 -> 822, 486^3 31100 -> 6060.
#define RISM_X_LENS(X)                                                                                      \
  X(16) X(18) X(24) X(27) X(32) X(36) X(48) X(54) X(64) X(72) X(81) X(96) X(108) X(128) X(144) X(162) X(192) \
  X(216) X(243) X(256)
#define RISM_YZ_LENS(X)                                                                                        \
  X(32) X(36) X(48) X(54) X(64) X(72) X(96) X(108) X(128) X(144) X(162) X(192) X(216) X(256) X(288) X(324) X(384) \
  X(432) X(486) X(512)
// ... and those with the half-width (FP32) and the persistent z tile beside the
// wide one, among which the context's creation chooses by timing; the others have
// the wide tile alone, and the two forms have not been tried there.  J pass at
// m = 3, us, wide / half-width / persistent: 512^3 FP32 1685 / 1426 / 1934 (F 4130
// / 2958 / 4598), where the wide tile is 98 KB.  Below that the wide tile is the
// fastest or within the timing's margin of the half-width one (256^3 127 / - / 261,
// 96^3 11.1 / - / 12.3, FP64 244 and 17.4 against 406 and 19.0 persistent; 48^3
// coarse problems have been given either).  The persistent form was never chosen:
// two tiles per CTA halve the CTAs of an SM.
#define RISM_Z_VARIANT_LENS(X) X(48) X(64) X(72) X(96) X(128) X(144) X(192) X(256) X(512)

#define RISM_IS(L) if (n == L) return true;
constexpr bool static_len_x(int n) {
  RISM_X_LENS(RISM_IS)
  return false;
}
constexpr bool static_len_yz(int n) {
  RISM_YZ_LENS(RISM_IS)
  return false;
}
constexpr bool z_has_variants(int n) {
  RISM_Z_VARIANT_LENS(RISM_IS)
#undef RISM_IS
  return false;
}

// y tile width: 128-byte rows (16 float2 or 8 double2); z tile width: 64-byte
// rows, so the m-site z tile is half as large and more CTAs share an SM.
template <typename T> constexpr int static_B() { return sizeof(T) == 4 ? 16 : 8; }
template <typename T> constexpr int static_Bz() { return sizeof(T) == 4 ? 8 : 4; }

// A kernel and the dynamic shared memory that it is launched with.
struct PassKernel {
  const void *fn;
  size_t smem;
};

template <typename T, int M> struct XPass {
  using V = typename Cx<T>::type;
  // mode MODE_F, MODE_J or MODE_S (t: the state of MODE_S)
  static void fwd(int mode, const Geo &g, const T *A, const T *B, const T *t, T p, int closure, V *W, const V *post,
                  const V *tw, cudaStream_t st);
  static void inv(const Geo &g, const V *W, const T *In, T *Out, T scale, T sub, const V *post, const V *tw,
                  NormPartial *part, cudaStream_t st);
  static void kernels(std::vector<PassKernel> &k);
};

template <typename T, int N> struct YPass {
  using V = typename Cx<T>::type;
  static void run(bool inv, const Geo &g, const CUtensorMap &tm, const V *tw, int *err, cudaStream_t st);
  static void kernels(std::vector<PassKernel> &k);
};

// The z transform alone (FP64, tiles of the y pass's width).
template <int N> struct ZAxis {
  static void run(bool inv, const Geo &g, const CUtensorMap &tm, const double2 *tw, int *err, cudaStream_t st);
  static void kernels(std::vector<PassKernel> &k);
};

// B: the tile width the tensor map was made for (static_Bz, or half of it
// where z_has_variants); persistent: double-buffered CTAs (wide tiles only).
template <typename T, int N> struct ZPass {
  using V = typename Cx<T>::type;
  static void run(int mode, int B, bool persistent, const Geo &g, const CUtensorMap &tm, const V *tw,
                  const ZParams<T> &zp, int *err, cudaStream_t st);
  static void kernels(int m, std::vector<PassKernel> &k);
};

}  // namespace rism
