// coarse_pk.cu -- instantiations and cooperative launch of the persistent
// coarse GMRES (coarse_pk.cuh) for the cubic coarse grids with
// shape-specialised transforms: (M, N) = (16, 32), (18, 36), (24, 48),
// (27, 54), (32, 64), (36, 72), (48, 96) in the plane form, (64, 128) in the five-phase form.
#include <algorithm>
#include <cstdlib>

#include "coarse_pk.cuh"

namespace rism {

namespace {

struct PkShape {
  const void *fn;
  size_t smem;
  int phases;
  int items;  // work items of the widest phase: more CTAs would only wait at the
              // barriers (48^3: 168 CTAs 489 us, 296 CTAs 524 us)
};

template <int M, int N> constexpr int pk_items() {
  const int rows = 3 * N, ztiles = ((M + kPkBz) / kPkBz) * N, zgroups = kPkThreads / (PkZSplit<N>::R1 * kPkBz * 3);
  return std::max(rows, (ztiles + zgroups - 1) / zgroups);
}

// Forms of a shape: the five-phase one, the plane one (three phases per step;
// where its plane tiles fit two CTAs per SM: coarse x half rows up to 48), or
// both, RISM3D_PK_PLANES=0 selecting the five-phase form (comparison tests).
enum { kPkFive, kPkPlane, kPkBoth };
template <int M, int N, int FORM> PkShape pk_make() {
  if constexpr (FORM != kPkFive) {
    const char *e = FORM == kPkBoth ? std::getenv("RISM3D_PK_PLANES") : nullptr;
    if (!(e && e[0] == '0'))
      return PkShape{(const void *)k_coarse_gmres<M, N, true>, pk_smem<M, N, true>(), pk_phases<true>(),
                     pk_items<M, N>()};
  }
  if constexpr (FORM != kPkPlane)
    return PkShape{(const void *)k_coarse_gmres<M, N, false>, pk_smem<M, N, false>(), pk_phases<false>(), 1 << 20};
  return PkShape{};  // not reached: the plane-only shapes returned above
}

bool pk_shape(int M, int N, PkShape *s) {
  switch (M * 1000 + N) {
#define PK_CASE(MM, NN, FORM)      \
  case MM * 1000 + NN:             \
    *s = pk_make<MM, NN, FORM>(); \
    return true;
    PK_CASE(16, 32, kPkPlane) PK_CASE(18, 36, kPkPlane) PK_CASE(24, 48, kPkBoth) PK_CASE(27, 54, kPkPlane)
    PK_CASE(32, 64, kPkBoth) PK_CASE(36, 72, kPkBoth) PK_CASE(48, 96, kPkBoth) PK_CASE(64, 128, kPkFive)
#undef PK_CASE
    default: return false;
  }
}

}  // namespace

// Grid barriers per GMRES step of the kernel that shape (M, N) runs (0: none).
int coarse_pk_phases(int M, int N) {
  PkShape s{};
  return pk_shape(M, N, &s) ? s.phases : 0;
}

// CTAs of the cooperative grid for shape (M, N): min(per_sm, the resident
// CTAs per SM) x SMs, at most one per work item; 0 when the shape has no kernel or nothing fits.
int coarse_pk_grid(int M, int N, int per_sm) {
  PkShape s{};
  if (!pk_shape(M, N, &s)) return 0;
  int dev = 0, sms = 0, coop = 0, occ = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop) return 0;
  // opt in always: the static shared memory counts against the default 48 KB
  if (cudaFuncSetAttribute(s.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s.smem) != cudaSuccess)
    return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, s.fn, kPkThreads, s.smem) != cudaSuccess || occ < 1)
    return 0;
  return std::min(std::min(occ, std::max(1, per_sm)) * sms, s.items);
}

// One coarse solve: zero the barrier counter, launch the grid.
cudaError_t coarse_pk_launch(const PkArgs &a, int M, int N, int grid, cudaStream_t st) {
  PkShape s{};
  if (!pk_shape(M, N, &s) || a.k < 1 || a.k > kPkMaxSteps || a.g.m > 3) return cudaErrorInvalidValue;
  cudaError_t e = cudaMemsetAsync(a.bar, 0, sizeof(unsigned), st);
  if (e != cudaSuccess) return e;
  PkArgs copy = a;
  void *args[] = {&copy};
  return cudaLaunchCooperativeKernel(s.fn, dim3((unsigned)grid), dim3(kPkThreads), args, s.smem, st);
}

}  // namespace rism
