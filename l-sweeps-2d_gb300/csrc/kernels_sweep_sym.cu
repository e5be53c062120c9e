// Launch of the symmetric-tile sweep kernels (sweep_sym.cuh): shapes, shared
// memory, clusters.
#include "sweep_sym.cuh"

#include <algorithm>

namespace lsw {

namespace {

constexpr SymTable kHostTab;
constexpr int kSmSharedBytes = 233472;   // shared memory of an SM; a CTA takes 1 KB of it besides its own
// producer and one consumer warp per 16 rows
int sym_warps(int max_ny) { return 1 + (max_ny + 15) / 16; }
SymKernel sym_kernel(bool split, int cl) {
  return cl == 1 ? sym_kernel_1(split) : cl == 2 ? sym_kernel_2(split) : sym_kernel_4(split);
}
int input_bytes(int R, bool split, int n16) {
  switch (R) {
    case 1: return split ? sym_input_bytes<1, true>(n16) : sym_input_bytes<1, false>(n16);
    case 2: return split ? sym_input_bytes<2, true>(n16) : sym_input_bytes<2, false>(n16);
    case 4: return split ? sym_input_bytes<4, true>(n16) : sym_input_bytes<4, false>(n16);
    case 8: return split ? sym_input_bytes<8, true>(n16) : sym_input_bytes<8, false>(n16);
    case 12: return split ? sym_input_bytes<12, true>(n16) : sym_input_bytes<12, false>(n16);
    default: return split ? sym_input_bytes<16, true>(n16) : sym_input_bytes<16, false>(n16);
  }
}

// The launch shape of a front whose cells have up to max_ny points per line:
// classes per chunk, ring stages, bytes per stage, shared memory; false if
// nothing fits.  A chunk is two classes on one or two CTAs per half (a wait and
// a release per chunk are ~30 instructions of every warp's line), one on four,
// or the whole line where that is at most 48 KB; two stages at least.
//
// Small cells share an SM: a CTA has only the warps of its rows, and the ring only
// what leaves room for the CTAs that the registers take (a CTA of all twelve rows'
// warps filled an SM whatever the cell).  An apply of sixteen right-hand sides on
// 16 x 16 cells of 21 points: complex64 12.6 -> 4.0 ms (whole blocks 10.1), split
// 12.1 -> 4.5 (10.4); of 53 points 36.2 -> 18.4 (33.6) and 27.3 -> 13.8 (32.0).  Lines of
// more than 112 points fill an SM as before.
bool sym_shape(int max_ny, int max_nx, int R, int CL, bool split, int maxopt, int* cpc, int* ns, int* stage,
               size_t* smem) {
  const int nb = (max_ny + 15) / 16, n16 = 16 * nb;
  if (nb > kSymTilesMax) return false;
  const size_t fixed = kHdr + kTileB + (size_t)2 * input_bytes(R, split, n16) +
                       (size_t)(2 * (CL - 1) + 1) * n16 * R * 8 + 2 * (size_t)((max_nx + 1) & ~1) * 8 +
                       kSymTilesMax * 4 * 3 * 8 + (size_t)n16 * 8 + (size_t)((max_nx + 15) & ~15) +
                       (size_t)R * (sizeof(DevSlot) + sizeof(SlotCoef) + sizeof(OutSlot)) + 16;
  // as many CTAs per SM as the registers take, fewer where the ring would not fit
  const int nq = 4 / CL;
  for (int share = sym_ctas_per_sm(max_ny); share >= 1; --share) {
    const size_t budget = share > 1 ? std::min((size_t)maxopt, (size_t)kSmSharedBytes / share - 1024) : (size_t)maxopt;
    if (fixed >= budget) continue;
    const size_t room = budget - fixed;
    for (int c = nq; c >= 1; c /= 2) {
      int tiles = 0;
      for (int q = 0; q < 4; q += c) tiles = std::max(tiles, kHostTab.first[nb][q + c] - kHostTab.first[nb][q]);
      const size_t st = (size_t)tiles * kTileB;
      const int n = (int)std::min<size_t>(kRingMax, room / st);
      if (n < 2 || (c > 2 && st > 49152)) continue;
      *cpc = c; *ns = n; *stage = (int)st;
      *smem = fixed + (size_t)n * st;
      return true;
    }
  }
  return false;
}

}  // namespace

// (128 registers per thread of an SM's 64 K)
int sym_ctas_per_sm(int max_ny) { return std::max(1, 16 / (1 + (max_ny + 15) / 16)); }

int sym_fit_mask(bool split, int max_ny, int max_nx, int slots) {
  int dev = 0, maxopt = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  cudaDeviceGetAttribute(&maxopt, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  const int R = std::min(front_rpad(std::max(1, slots)), front_rmax(false));
  int mask = 0, cpc, ns, stage;
  size_t smem;
  for (int cl = 1; cl <= 4; cl *= 2)
    if (sym_shape(max_ny, max_nx, R, cl, split, maxopt, &cpc, &ns, &stage, &smem)) mask |= 1 << cl;
  return mask;
}

cudaError_t launch_front_sym(const FrontArgs& a_in, int max_ny, int max_nx, cudaStream_t st) {
  if (a_in.item_count <= 0) return cudaSuccess;
  FrontArgs a = a_in;
  const bool split = a.split != 0;
  const int R = std::min(front_rpad(std::max(1, a.max_slots)), front_rmax(false));
  if (a.cluster < 1) a.cluster = 1;
  if ((a.cluster != 1 && a.cluster != 2 && a.cluster != 4) || max_nx < 5) return cudaErrorInvalidValue;
  int dev = 0, maxopt = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&maxopt, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  size_t smem = 0;
  if (!sym_shape(max_ny, max_nx, R, a.cluster, split, maxopt, &a.ksw, &a.stages, &a.chunk, &smem))
    return cudaErrorInvalidConfiguration;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[1];
  cfg.gridDim = dim3((unsigned)(a.item_count * 2 * a.cluster));
  cfg.blockDim = dim3(32 * sym_warps(max_ny));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)(2 * a.cluster);   // top and bottom halves
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const SymKernel kern = sym_kernel(split, a.cluster);
  // the attribute is an upper bound: always the device maximum, so that
  // host threads launching concurrently never lower it under one another
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, maxopt);
  if (e != cudaSuccess) return e;
  return cudaLaunchKernelEx(&cfg, kern, a);
}

int sym_max_clusters(bool split, int cluster) {
  int dev = 0, maxopt = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  cudaDeviceGetAttribute(&maxopt, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  const SymKernel kern = sym_kernel(split, cluster / 2);
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[1];
  cfg.gridDim = dim3((unsigned)(cluster * 1024));
  cfg.blockDim = dim3(32 * kSymWarps);     // (the cost model counts one CTA per SM)
  cfg.dynamicSmemBytes = (size_t)maxopt;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, maxopt);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, kern, &cfg);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

}  // namespace lsw
