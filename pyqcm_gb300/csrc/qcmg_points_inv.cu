// K means of the per-point inverses M(K, z)^-1, with the phases of
// translations: the density of states, the CDMFT projected Green function
// and the lattice averages.
//
// One point per thread, a warp per CTA as in qcmg_points.cuh, but with both
// triangular factors in shared memory (16 L^2 bytes per point: 6 warps per SM
// at L = 8, 27 at L = 4), since every column of the inverse is solved for.
// The inverses themselves are never stored: each column is summed over the
// warp's 32 points as soon as it is solved, by a reduction that halves the
// number of values a lane holds at every step, 2L - 1 additions for 2L
// values (five per value for a plain butterfly).
//
// The phase of translation m at (kx, ky, kz) is split into an x part and the
// rest. A warp takes points of one (ky, kz) row, so it only needs the sums
// of X, X cos(2 pi kx r) and X sin(2 pi kx r) for the few distinct |r| among
// the translations' x components; k_inv_final puts the rest of each phase on
// the row sums.
//
// 2x4 cluster, 64x64 K x 64 w x 2 spins, 9 translations: writing the inverses
// (537 MB per spin) and reading them back once per element and translation
// took 16.9 ms per call, 4.7 ms now; the plaquette's host function (64x64 K x
// 200 w) 2.63 ms, 1.28 ms (0.85 ms with the later Green function kernel). Bound
// by the FP64 pipe.
#include "qcmg_points.h"

namespace qcmg {

constexpr int pow2_at_least(int n) { return n <= 1 ? 1 : 2 * pow2_at_least((n + 1) / 2); }

// Sums each of the V values of the 32 lanes; afterwards lane l holds the sum
// of value (l >> (5 - log2 V)) (V a power of two <= 32).
template <int V>
__device__ __forceinline__ double warp_sums(double (&a)[V], int lane) {
  int o = 16;
#pragma unroll
  for (int n = V; n > 1; n >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < n / 2; ++i) {
      const double give = up ? a[i] : a[i + n / 2], keep = up ? a[i + n / 2] : a[i];
      a[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  double s = a[0];
  for (; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

template <int L>
__global__ void __launch_bounds__(32) k_inv_rows(InvArgs A) {
  constexpr int V = pow2_at_least(2 * L);
  extern __shared__ double2 lu[];  // L L x 32, then the row's sums
  double* acc = (double*)(lu + L * L * 32);
  const int lane = threadIdx.x;
  const int w = blockIdx.x / A.nrow, row = blockIdx.x - w * A.nrow;
  const double2* base = A.base + (size_t)w * (L * L);
  for (int i = lane; i < A.nf * L * 2 * L; i += 32) acc[i] = 0.0;
  for (int h0 = A.row_start[row]; h0 < A.row_start[row + 1]; h0 += 32) {
    const int h = h0 + lane, hc = min(h, A.row_start[row + 1] - 1);
    const double wgt = h == hc ? __ldg(A.wgt + hc) * A.scale : 0.0;
    unsigned long long perm = 0xfedcba9876543210ull;
    __syncwarp();
#pragma unroll
    for (int j = 0; j < L; ++j) {
      double mx[L], my[L];
#pragma unroll
      for (int i = 0; i < L; ++i) {
        const int r = (int)(perm >> (4 * i)) & 15;
        const double2 b = __ldg(base + r * L + j);
        const int q = __ldg(A.vidx + r * L + j);
        mx[i] = b.x;
        my[i] = b.y;
        if (q >= 0) {
          const double2 v = __ldg(A.vk + (size_t)q * A.nk + hc);
          mx[i] -= v.x;
          my[i] -= v.y;
        }
      }
#pragma unroll
      for (int k = 0; k < j; ++k) {
        lu[(k * L + j) * 32 + lane] = make_double2(mx[k], my[k]);  // upper factor
#pragma unroll
        for (int i = k + 1; i < L; ++i) {
          const double2 l = lu[(i * L + k) * 32 + lane];
          mx[i] = fma(-l.x, mx[k], mx[i]);
          my[i] = fma(-l.x, my[k], my[i]);
          mx[i] = fma(l.y, my[k], mx[i]);
          my[i] = fma(-l.y, mx[k], my[i]);
        }
      }
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
            double2 *rj = lu + j * L * 32 + lane, *rp = lu + p * L * 32 + lane;
#pragma unroll
            for (int k = 0; k < j; ++k) {
              const double2 t = rj[k * 32];
              rj[k * 32] = rp[k * 32];
              rp[k * 32] = t;
            }
          }
        }
      }
      const double rd = 1.0 / fma(px, px, py * py), ix = px * rd, iy = -py * rd;
      lu[(j * L + j) * 32 + lane] = make_double2(ix, iy);  // the pivot's inverse
#pragma unroll
      for (int i = j + 1; i < L; ++i)
        lu[(i * L + j) * 32 + lane] =
            make_double2(fma(mx[i], ix, -my[i] * iy), fma(mx[i], iy, my[i] * ix));
    }
    const int ix = A.nf > 1 ? __ldg(A.rep + hc) % A.gx : 0;
    for (int c = 0; c < L; ++c) {  // column c of the inverse, times the point's weight
      double x[2 * L];
#pragma unroll
      for (int i = 0; i < L; ++i) {
        x[2 * i] = ((int)(perm >> (4 * i)) & 15) == c ? wgt : 0.0;
        x[2 * i + 1] = 0.0;
      }
#pragma unroll
      for (int k = 0; k < L; ++k)
#pragma unroll
        for (int i = k + 1; i < L; ++i) {
          const double2 l = lu[(i * L + k) * 32 + lane];
          x[2 * i] = fma(l.y, x[2 * k + 1], fma(-l.x, x[2 * k], x[2 * i]));
          x[2 * i + 1] = fma(-l.y, x[2 * k], fma(-l.x, x[2 * k + 1], x[2 * i + 1]));
        }
#pragma unroll
      for (int i = L - 1; i >= 0; --i) {
#pragma unroll
        for (int k = i + 1; k < L; ++k) {
          const double2 u = lu[(i * L + k) * 32 + lane];
          x[2 * i] = fma(u.y, x[2 * k + 1], fma(-u.x, x[2 * k], x[2 * i]));
          x[2 * i + 1] = fma(-u.y, x[2 * k], fma(-u.x, x[2 * k + 1], x[2 * i + 1]));
        }
        const double2 d = lu[(i * L + i) * 32 + lane];
        const double re = fma(x[2 * i], d.x, -x[2 * i + 1] * d.y);
        x[2 * i + 1] = fma(x[2 * i], d.y, x[2 * i + 1] * d.x);
        x[2 * i] = re;
      }
      for (int f = 0; f < A.nf; ++f) {
        double a[V];
        const double g = f ? __ldg(A.wx + (size_t)(f - 1) * A.gx + ix) : 1.0;
#pragma unroll
        for (int i = 0; i < V; ++i) a[i] = i < 2 * L ? (f ? x[i] * g : x[i]) : 0.0;
        const double s = warp_sums<V>(a, lane);
        constexpr int per = 32 / V;
        if (lane % per == 0 && lane / per < 2 * L) acc[(f * L + c) * 2 * L + lane / per] += s;
      }
    }
  }
  __syncwarp();
  // part[((w nrow + row) nf + f) L L + c L + i], the inverse's (i, c)
  double* out = (double*)(A.part + ((size_t)blockIdx.x * A.nf) * (L * L));
  for (int i = lane; i < A.nf * L * 2 * L; i += 32) out[i] = acc[i];
}

// out[w][m](a, b) = (1/nk) [S+(a, b) + S-(b, a)], S+- the row sums with the
// phases e^{+-2 pi i K.R_m} (S- for paired points only): per row, the x part
// S_0 or S_cos +- i S_sin times the row's phase yz[m][row].
__global__ void k_inv_final(InvArgs A, int L, int nm, const int* __restrict__ fx,
                            const double2* __restrict__ yz, int paired, double inv_nk,
                            double2* __restrict__ out) {
  const size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const int LL = L * L;
  if (idx >= (size_t)A.nw * nm * LL) return;
  const int e = (int)(idx % LL), m = (int)(idx / LL % nm), w = (int)(idx / LL / nm);
  const int a = e / L, b = e - a * L;
  const int f = fx ? fx[m] : 0;  // 0: no x phase; +-(2u + 1): cosine in function 2u + 1, sine after it
  double sx = 0.0, sy = 0.0;
  for (int side = 0; side < (paired ? 2 : 1); ++side) {
    const double sg = side ? -1.0 : 1.0;
    const int at = side ? a * L + b : b * L + a;  // (i, c) is stored at c L + i
    for (int r = 0; r < A.nrow; ++r) {
      const double2* p = A.part + ((size_t)w * A.nrow + r) * A.nf * LL + at;
      double2 v = p[(size_t)(f < 0 ? -f : f) * LL];
      if (f) {
        const double2 t = p[(size_t)((f < 0 ? -f : f) + 1) * LL];
        const double g = f < 0 ? -sg : sg;  // v + i g t
        v.x -= g * t.y;
        v.y += g * t.x;
      }
      if (yz) {
        const double2 ph = yz[(size_t)m * A.nrow + r];
        const double py = sg * ph.y;
        sx += v.x * ph.x - v.y * py;
        sy += v.x * py + v.y * ph.x;
      } else {
        sx += v.x;
        sy += v.y;
      }
    }
  }
  out[idx] = make_double2(sx * inv_nk, sy * inv_nk);
}

template <int L>
static void launch_rows(int n, const InvArgs& A, cudaStream_t s) {
  if constexpr (L > 0) {
    if (n != L) return launch_rows<L - 1>(n, A, s);
    const size_t smem = (size_t)L * L * 32 * sizeof(double2) + (size_t)A.nf * 2 * L * L * sizeof(double);
    auto kern = k_inv_rows<L>;
    if (smem > 48 * 1024)
      QCMG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const size_t grid = (size_t)A.nw * A.nrow;
    QCMG_CHECK_ARG(grid <= 0x7fffffffu, "too many points for one launch");
    kern<<<(unsigned)grid, 32, smem, s>>>(A);
    QCMG_CUDA(cudaGetLastError());
  }
}

void launch_inverse_means(int L, const InvArgs& A, int nm, const int* fx, const double2* yz,
                          bool paired, double inv_nk, double2* out, cudaStream_t s) {
  launch_rows<kMaxPointL>(L, A, s);
  const size_t n = (size_t)A.nw * nm * L * L;
  k_inv_final<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(A, L, nm, fx, yz, paired ? 1 : 0, inv_nk, out);
  QCMG_CUDA(cudaGetLastError());
}

}  // namespace qcmg
