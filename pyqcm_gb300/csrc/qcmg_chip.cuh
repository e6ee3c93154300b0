// Device parts shared by the on-chip recurrences (qcmg_chip.cu,
// qcmg_chip_band.cu).
#pragma once

#include <cooperative_groups.h>

#include "qcmg_chip.h"

namespace cg = cooperative_groups;

namespace qcmg {

constexpr uint32_t kChipStates = 16384;  // largest sector
constexpr int kChipThreads = 512;
constexpr int kTile = 32;  // states per partial sum: one per lane, so that a few hundred
                           // states per CTA still fill the four sub-partitions's FP64 pipes

struct ChipOp {
  uint32_t du, dd, D;
  int L, inter;
  const uint32_t *ell;
  const uint16_t* len;
  const uint32_t *rp_dn, *col_dn, *bin_up, *bin_dn;
  const double *vtab, *val_dn, *diag_up, *diag_dn, *wdn;
  double U;
};

// Diagonal element (iu, id), as the FP64 product forms it.
__device__ __forceinline__ double chip_diag(const ChipOp& A, uint32_t iu, uint32_t id) {
  double d = A.diag_up[iu] + A.diag_dn[id];
  if (A.inter == QCMG_INTER_ONSITE) {
    d += A.U * (double)__popc(A.bin_up[iu] & A.bin_dn[id]);
  } else if (A.inter == QCMG_INTER_GENERAL) {
    uint32_t u = A.bin_up[iu];
    const double* w = A.wdn + (size_t)id * A.L;
    while (u) {
      d += w[__ffs(u) - 1];
      u &= u - 1;
    }
  }
  return d;
}

// (hops of x)_i with x in shared memory
__device__ __forceinline__ double chip_hops(const ChipOp& A, const double* x, uint32_t iu,
                                            uint32_t id, double acc) {
  const double* xs = x + id * A.du;
#pragma unroll 4
  for (int k = 0, n = __ldg(A.len + iu); k < n; ++k) {
    const uint32_t e = __ldg(A.ell + k * A.du + iu);
    acc = fma(__ldg(A.vtab + (e >> 16)), xs[e & 0xffffu], acc);
  }
  const double* xc = x + iu;
#pragma unroll 4
  for (uint32_t k = __ldg(A.rp_dn + id), e = __ldg(A.rp_dn + id + 1); k < e; ++k)
    acc = fma(__ldg(A.val_dn + k), xc[__ldg(A.col_dn + k) * A.du], acc);
  return acc;
}

__device__ __forceinline__ double warp_total(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sum of the tile partials in a fixed order, for every thread of the block:
// slot[0], or with NORM its square root and the root's inverse in slot[0] and
// slot[1].  The block's warp 0 does it: an FP64 instruction costs the SM 16
// cycles per warp (a square root and a division by all 16 warps 3 us), so the
// others wait instead of repeating it.  The root comes from its inverse (a
// third of the latency of a square root and a division; within 2 ulp of the
// root: over 114 solves of 49 to 15,876 states the energies' error is 2.8e-16
// rms, 2.9e-16 on the fixed-point path with its exact sums and rounded root).
// Any fixed order of the tiles is as accurate as another. The last first was
// chosen among 17 orders of equal error: a CDMFT loop whose bath fits stop at
// the rounding of their cost takes 11, 12 or 13 steps with one or another, and
// this is one of those that take the 11 of the recorded loop it is compared with.
__device__ __forceinline__ void root_and_inverse(double s, double* root) {
  const double r = rsqrt(s);
  root[0] = s > 0.0 ? s * r : s;  // 0, or NaN as it came
  root[1] = r;
}
template <bool NORM>
__device__ __forceinline__ void tile_total(const double* part, int nt, double* slot) {
  if (threadIdx.x < 32) {
    double s = 0.0;
    for (int t = nt - 1 - (int)threadIdx.x; t >= 0; t -= 32) s += part[t];
    s = warp_total(s);
    if (threadIdx.x == 0) {
      if (NORM)
        root_and_inverse(s, slot);
      else
        slot[0] = s;
    }
  }
  __syncthreads();
}

inline ChipOp chip_op(const qcmg_hamiltonian* H) {
  ChipOp A;
  A.du = H->du;
  A.dd = H->dd;
  A.D = (uint32_t)H->dim;
  A.L = H->L;
  A.inter = H->inter_kind;
  A.ell = H->up.ell;
  A.len = H->up.len;
  A.vtab = H->up.vtab;
  A.diag_up = H->up.diag.p;
  A.bin_up = H->up.bin.p;
  A.rp_dn = H->dn.rowptr.p;
  A.col_dn = H->dn.col.p;
  A.val_dn = H->dn.val.p;
  A.diag_dn = H->dn.diag.p;
  A.bin_dn = H->dn.bin.p;
  A.wdn = H->wdn.p;
  A.U = H->U;
  return A;
}

// Launches kern on n clusters of C CTAs.
template <class Kern, class... Args>
inline void launch_clusters(Kern kern, int n, int C, size_t smem, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(n * C));
  cfg.blockDim = dim3(kChipThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)C;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  QCMG_CUDA(cudaLaunchKernelEx(&cfg, kern, args...));
}

// Whether clusters of C CTAs with this much shared memory can run (C above
// the portable 8 needs the kernel's consent, given here).
template <class Kern>
inline bool clusters_run(Kern kern, int C, size_t smem) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)C);
  cfg.blockDim = dim3(kChipThreads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)C;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int n = 0;
  const bool ok = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                  cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n > 0;
  if (!ok) cudaGetLastError();
  return ok;
}

}  // namespace qcmg
