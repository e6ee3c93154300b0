// Per-point LU kernels of the lattice integrals (qcmg_points.cuh).
#pragma once

#include "qcmg_internal.h"

namespace qcmg {

constexpr int kMaxPointL = 16;  // largest matrix of the register kernels

// One launch of the point kernels: nk wavevectors of nw frequencies, warps of
// 32 consecutive wavevectors of one frequency.
struct LuArgs {
  int nk = 0, nw = 0;
  const double2* base = nullptr;    // nw x L x L row-major, G(z)^-1 + Gamma(z) - Hdiff
  const short* vidx = nullptr;      // L x L: row of vk holding V(K)_{rc}, or -1
  const double2* vk = nullptr;      // nnz x nk: the nonzero entries of V(K)
  const double2* uk = nullptr;      // L x nk: e^{2 pi i K.x_a} (periodized G)
  const double* det2 = nullptr;     // nw: |det G|^2 = det2 2^dexp
  const int* dexp = nullptr;
  const double* wgt = nullptr;      // nk: weight of each wavevector
  double* part = nullptr;           // functional: nw x part_ld warp sums (this launch's at part)
  int part_ld = 0;
  double2* out = nullptr;           // periodized G: nw x out_ld (this launch's at out)
  int out_ld = 0;
};

// part[w][b] = sum over the 32 wavevectors b of wgt log|det(V G - 1)|
void launch_sef_points(int L, const LuArgs& A, cudaStream_t s);
// out[w][k] = (1/L) u^+ (base_w - V(K))^-1 u
void launch_cpt_points(int L, const LuArgs& A, cudaStream_t s);

// The sums over K of the inverses. The points (their tables as in LuArgs) are
// grouped in rows [row_start[r], row_start[r + 1]); with nf > 1 a row's points
// share (ky, kz).
struct InvArgs {
  int nk = 0, nw = 0, nrow = 0;
  const double2* base = nullptr;
  const short* vidx = nullptr;
  const double2* vk = nullptr;
  const double* wgt = nullptr;
  double scale = 1.0;               // on the weights
  const int* row_start = nullptr;   // nrow + 1
  const int* rep = nullptr;         // flat grid index of each point
  int gx = 1;
  int nf = 1;                       // weight functions: 1 and the rows of wx
  const double* wx = nullptr;       // (nf - 1) x gx: cosine, sine of each distinct |R_x|
  double2* part = nullptr;          // nw x nrow x nf x L x L
};
constexpr int kMaxInvFuncs = 9;

// out (nw x nm x L x L row-major): the means with the phases of nm
// translations. fx[m]: 0, or +-(the cosine's function) by the sign of R_x;
// yz: nm x nrow, the rest of each phase (null: one plain mean).
void launch_inverse_means(int L, const InvArgs& A, int nm, const int* fx, const double2* yz,
                          bool paired, double inv_nk, double2* out, cudaStream_t s);

// |det|^2 as mantissa and exponent: m 2^e *= bv (a squared modulus).  Zeros,
// subnormals and non-finite values go into the mantissa unchanged.
__device__ __forceinline__ void det_mul(double& m, int& e, double bv) {
  const int hi = __double2hiint(bv), ex = (hi >> 20) & 0x7ff;
  if (ex != 0 && ex != 0x7ff) {
    bv = __hiloint2double((hi & 0x000fffff) | 0x3ff00000, __double2loint(bv));
    e += ex - 1023;
  }
  m *= bv;
}

// Size of a pivot candidate for comparison: the larger magnitude of its two
// parts, by their high words (no FP64 instruction; within sqrt(2) of the
// modulus, so the multipliers stay below 1.5).  NaN compares largest.
__device__ __forceinline__ unsigned pivot_key(double x, double y) {
  return max((unsigned)__double2hiint(x) & 0x7fffffffu, (unsigned)__double2hiint(y) & 0x7fffffffu);
}

}  // namespace qcmg
