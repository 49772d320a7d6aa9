// coarse_pk.cu -- instantiations and cooperative launch of the persistent
// coarse GMRES for the cubic coarse grids with shape-specialised transforms:
// the plane form (coarse_planes.cuh) up to 96^3, the five-phase form
// (coarse_pk.cuh) for 128^3.
#include <algorithm>
#include <cstdlib>

#include "coarse_planes.cuh"

namespace rism {

namespace {

struct PkShape {
  const void *fn = nullptr;
  size_t smem = 0;
  int phases = 0;
  int threads = 0;
  int items = 0;  // work items of the widest phase: more CTAs would only wait at the barriers
};

template <int M> PkShape pk_planes() {
  using S = PlShape<M>;
  const int ztiles = ((M + kPkBz) / kPkBz) * S::N;
  PkShape s;
  s.fn = (const void *)k_coarse_planes<M>;
  s.smem = S::smem;
  s.phases = 3;
  s.threads = S::THR;
  s.items = std::max(3 * S::N, ztiles);
  return s;
}
template <int M, int N> PkShape pk_five() {
  PkShape s;
  s.fn = (const void *)k_coarse_gmres<M, N>;
  s.smem = pk_smem<M, N>();
  s.phases = 5;
  s.threads = kPkThreads;
  s.items = 1 << 20;
  return s;
}

// RISM3D_PK_PLANES=0 selects the five-phase form where both exist
// (comparison tests).
template <int M, int N> PkShape pk_both() {
  const char *e = std::getenv("RISM3D_PK_PLANES");
  return e && e[0] == '0' ? pk_five<M, N>() : pk_planes<M>();
}

bool pk_shape(int M, int N, PkShape *s) {
  if (N != 2 * M) return false;
  switch (N) {
    case 32: *s = pk_planes<16>(); return true;
    case 36: *s = pk_planes<18>(); return true;
    case 48: *s = pk_both<24, 48>(); return true;
    case 54: *s = pk_planes<27>(); return true;
    case 64: *s = pk_both<32, 64>(); return true;
    case 72: *s = pk_both<36, 72>(); return true;
    case 96: *s = pk_both<48, 96>(); return true;
    case 128: *s = pk_five<64, 128>(); return true;
    default: return false;
  }
}

}  // namespace

// Grid barriers per GMRES step of the kernel that shape (M, N) runs (0: none).
int coarse_pk_phases(int M, int N) {
  PkShape s;
  return pk_shape(M, N, &s) ? s.phases : 0;
}

// CTAs of the cooperative grid for shape (M, N): min(per_sm, the resident
// CTAs per SM) x SMs, at most one per work item; 0 when the shape has no
// kernel or nothing fits.
int coarse_pk_grid(int M, int N, int per_sm) {
  PkShape s;
  if (!pk_shape(M, N, &s)) return 0;
  int dev = 0, sms = 0, coop = 0, occ = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop) return 0;
  // opt in always: the static shared memory counts against the default 48 KB
  if (cudaFuncSetAttribute(s.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s.smem) != cudaSuccess)
    return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, s.fn, s.threads, s.smem) != cudaSuccess || occ < 1)
    return 0;
  return std::min(std::min(occ, std::max(1, per_sm)) * sms, s.items);
}

// One coarse solve: zero the barrier counter, launch the grid.
cudaError_t coarse_pk_launch(const PkArgs &a, int M, int N, int grid, cudaStream_t st) {
  PkShape s;
  if (!pk_shape(M, N, &s) || a.k < 1 || a.k > kPkMaxSteps || a.g.m > 3) return cudaErrorInvalidValue;
  cudaError_t e = cudaMemsetAsync(a.bar, 0, sizeof(unsigned), st);
  if (e != cudaSuccess) return e;
  PkArgs copy = a;
  void *args[] = {&copy};
  return cudaLaunchCooperativeKernel(s.fn, dim3((unsigned)grid), dim3((unsigned)s.threads), args, s.smem, st);
}

}  // namespace rism
