// One complex L x L LU factorization per (K, z) point, one point per thread:
// the integrand of the Potthoff functional and the periodized Green function.
//
// GB300 issues two FP64 FMAs per SM and cycle, so one warp with independent
// FMAs fills an SM sub-partition's FP64 pipe; what counts is the number of
// FP64 instructions per point and that every sub-partition has a warp.
//  - Left-looking (column by column) factorization: the working column lives
//    in registers and only the strictly lower part of the multipliers is
//    kept, 16 L(L-1)/2 bytes per point in shared memory instead of 16 L^2.
//    At L = 12 that is 1,056 bytes, six one-warp CTAs per SM (a full matrix
//    per thread allowed three warps, so one sub-partition idled).
//  - A multiply-subtract is four FMAs; pivots are compared by the high words
//    of their parts (integer instructions); |det|^2 is one product per pivot
//    with its exponent kept apart, so a point takes one logarithm.
//  - Row interchanges are not applied to the matrix: the permutation is a
//    64-bit word of nibbles and each new column is read through it.
//  - V(K) is tabulated once per call over the wavevectors (coalesced reads
//    from L2, shared by all frequencies).
// 3x4 cluster, 128x128 K x 256 frequencies x 2 spins: 8.39M points (4.20M
// with K and -K paired): 114.1 ms with a full matrix per thread in shared
// memory, 21.8 ms now for the whole call (FP64 pipe floor of the paired
// points: 18 ms; 20.2 ms with the later Green function kernel).  8-site chain,
// 256 K x 512 z: 1,120 -> 609 us per call, 427 with that kernel.
#pragma once

#include "qcmg_points.h"

namespace qcmg {

// entry (i, k), k < i, of the multipliers; row L is the border of the CPT form
__host__ __device__ constexpr int tri(int i, int k) { return i * (i - 1) / 2 + k; }

// CPT = true: g = u^+ M^-1 u is the Schur complement of the bordered matrix
// [[M, u], [u^+, 0]], so it needs neither the upper factor nor a back
// substitution: the border row is eliminated as one more row (never a pivot)
// and the border column as one more column.
template <int L, bool CPT>
__global__ void __launch_bounds__(32) k_lu_points(LuArgs A) {
  constexpr int N = CPT ? L + 1 : L;
  extern __shared__ double2 lf[];  // tri(N, 0) x 32
  const int lane = threadIdx.x;
  const int nkb = (A.nk + 31) >> 5;
  const int w = blockIdx.x / nkb, kb = blockIdx.x - w * nkb;
  const int ik = kb * 32 + lane, k0 = min(ik, A.nk - 1);
  const double2* base = A.base + (size_t)w * (L * L);
  unsigned long long perm = 0xfedcba9876543210ull;  // perm nibble i: matrix row in place i
  double dm = 1.0;
  int de = 0;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    // column j in the current row order
    double mx[N], my[N];
#pragma unroll
    for (int i = 0; i < L; ++i) {
      const int r = (int)(perm >> (4 * i)) & 15;
      if (j < L) {
        const double2 b = __ldg(base + r * L + j);
        const int q = __ldg(A.vidx + r * L + j);
        mx[i] = b.x;
        my[i] = b.y;
        if (q >= 0) {
          const double2 v = __ldg(A.vk + (size_t)q * A.nk + k0);
          mx[i] -= v.x;
          my[i] -= v.y;
        }
      } else {
        const double2 u = __ldg(A.uk + (size_t)r * A.nk + k0);
        mx[i] = u.x;
        my[i] = u.y;
      }
    }
    if (CPT) {
      if (j < L) {
        const double2 u = __ldg(A.uk + (size_t)j * A.nk + k0);
        mx[N - 1] = u.x;
        my[N - 1] = -u.y;
      } else {
        mx[N - 1] = my[N - 1] = 0.0;
      }
    }
    // elimination by the earlier columns
#pragma unroll
    for (int k = 0; k < j; ++k) {
#pragma unroll
      for (int i = k + 1; i < N; ++i) {
        const double2 l = lf[tri(i, k) * 32 + lane];
        mx[i] = fma(-l.x, mx[k], mx[i]);
        my[i] = fma(-l.x, my[k], my[i]);
        mx[i] = fma(l.y, my[k], mx[i]);
        my[i] = fma(-l.y, mx[k], my[i]);
      }
    }
    if (j == L) {
      if (ik < A.nk) A.out[(size_t)w * A.out_ld + ik] = make_double2(mx[N - 1] * (-1.0 / L), my[N - 1] * (-1.0 / L));
      break;
    }
    // pivot among rows j..L-1
    double px = mx[j], py = my[j];
    if (j + 1 < L) {
      unsigned key = pivot_key(px, py);
      int p = j;
#pragma unroll
      for (int i = j + 1; i < L; ++i) {
        const unsigned ki = pivot_key(mx[i], my[i]);
        if (ki > key) {
          key = ki;
          p = i;
          px = mx[i];
          py = my[i];
        }
      }
      if (__any_sync(0xffffffffu, p != j)) {
#pragma unroll
        for (int i = j + 1; i < L; ++i)
          if (p == i) {
            mx[i] = mx[j];
            my[i] = my[j];
          }
        if (p != j) {
          const unsigned long long d = ((perm >> (4 * j)) ^ (perm >> (4 * p))) & 15ull;
          perm ^= (d << (4 * j)) | (d << (4 * p));
          double2* rp = lf + tri(p, 0) * 32 + lane;
#pragma unroll
          for (int k = 0; k < j; ++k) {
            const double2 t = lf[tri(j, k) * 32 + lane];
            lf[tri(j, k) * 32 + lane] = rp[k * 32];
            rp[k * 32] = t;
          }
        }
      }
    }
    const double d2 = fma(px, px, py * py);
    if (!CPT) det_mul(dm, de, d2);
    if (j + 1 < N) {
      const double rd = 1.0 / d2, ix = px * rd, iy = -py * rd;
#pragma unroll
      for (int i = j + 1; i < N; ++i)
        lf[tri(i, j) * 32 + lane] =
            make_double2(fma(mx[i], ix, -my[i] * iy), fma(mx[i], iy, my[i] * ix));
    }
  }
  if constexpr (!CPT) {
    // log|det(V G - 1)| = log|det M| + log|det G|, formed point by point
    // from the mantissas and exponents: at high frequencies both are
    // ~L log|z| and cancel, here in the integer exponents
    double v = 0.5 * (log(dm * __ldg(A.det2 + w)) + (double)(de + __ldg(A.dexp + w)) * 0.6931471805599453094);
    v = ik < A.nk ? v * __ldg(A.wgt + ik) : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) A.part[(size_t)w * A.part_ld + kb] = v;
  }
}

template <bool CPT, int L>
static void launch_lu(int n, const LuArgs& A, cudaStream_t s) {
  if constexpr (L > 0) {
    if (n != L) return launch_lu<CPT, L - 1>(n, A, s);
    const size_t smem = (size_t)tri(CPT ? L + 1 : L, 0) * 32 * sizeof(double2);
    auto kern = k_lu_points<L, CPT>;
    if (smem > 48 * 1024)
      QCMG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const size_t grid = (size_t)A.nw * ((A.nk + 31) / 32);
    QCMG_CHECK_ARG(grid <= 0x7fffffffu, "too many points for one launch");
    kern<<<(unsigned)grid, 32, smem, s>>>(A);
    QCMG_CUDA(cudaGetLastError());
  } else {
    throw Error(QCMG_ERR_ARG, "matrix dimension out of the point kernels' range");
  }
}

}  // namespace qcmg
