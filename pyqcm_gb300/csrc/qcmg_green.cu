// Lehmann Green function of a Q-matrix, batched over frequencies:
//   G_w(b, a) = sum_i v(a,i) u_w(i) conj(v(b,i)),  u_w(i) = 1 / (z_w - e_i)
// (src_ed/Q_matrix.hpp:133-151 with VDVH_naive, src_util/VDVH_kernel.cpp:28-48).
//
// A thread owns one matrix element of kFreq frequencies, so the product
// v_a conj(v_b) is formed once per pole for all of them; with a real v only
// the elements a <= b are computed (G is symmetric) and a pole costs
// 1 + 2 kFreq FP64 instructions instead of 8 per element and frequency. The
// eight warps of a block take every eighth pole and are added in a fixed
// order, which keeps the chip's FP64 pipes busy at a few hundred frequencies;
// u_w is tabulated in shared memory, one tile of poles at a time.
// L = 12, 1,100 poles, 256 frequencies: 979 us, 205 us now.
#include "qcmg_internal.h"
#include "qcmg_krylov.h"

namespace qcmg {

constexpr int kFreq = 4;   // frequencies per thread
constexpr int kPoles = 32;  // poles per tile of u
constexpr int kGreenWarps = 8;

template <bool REAL>
__global__ void __launch_bounds__(32 * kGreenWarps)
    k_green(int L, int M, int nel, int nz, const double* __restrict__ e,
            const double2* __restrict__ v, const double2* __restrict__ z,
            double2* __restrict__ G) {
  extern __shared__ double2 u[];  // frequencies of the block x kPoles, then the warps' sums
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  // thread = (frequency group, element), elements fastest; nfg groups
  const int nfg = (nz + kFreq - 1) / kFreq;
  const int t0 = blockIdx.x * 32, t = t0 + lane;
  const int g0 = t0 / nel, g1 = min((t0 + 31) / nel, nfg - 1);
  const int f0 = g0 * kFreq, nf = (g1 - g0 + 1) * kFreq;
  const bool live = t < nfg * nel;
  const int fg = live ? t / nel : g0, el = live ? t - fg * nel : 0;
  int a, b;  // element: all (a, b), or a <= b
  if (REAL) {
    b = (int)((sqrtf(8.0f * el + 1.0f) - 1.0f) * 0.5f);
    while (b * (b + 1) / 2 > el) --b;
    while ((b + 1) * (b + 2) / 2 <= el) ++b;
    a = el - b * (b + 1) / 2;
  } else {
    a = el / L;
    b = el - a * L;
  }
  double sr[kFreq], si[kFreq];
#pragma unroll
  for (int f = 0; f < kFreq; ++f) sr[f] = si[f] = 0.0;
  for (int i0 = 0; i0 < M; i0 += kPoles) {
    const int np = min(kPoles, M - i0);
    __syncthreads();
    for (int q = threadIdx.x; q < nf * kPoles; q += blockDim.x) {
      const int f = f0 + q / kPoles, i = q % kPoles;
      if (i < np && f < nz) {
        const double re = z[f].x - e[i0 + i], im = z[f].y, r = 1.0 / (re * re + im * im);
        u[q] = make_double2(re * r, -im * r);
      } else {
        u[q] = make_double2(0.0, 0.0);
      }
    }
    __syncthreads();
    const double2* uf = u + (fg - g0) * kFreq * kPoles;
#pragma unroll
    for (int i = wp; i < kPoles; i += kGreenWarps) {
      if (i >= np) break;
      const double2 va = __ldg(v + a + (size_t)L * (i0 + i)), vb = __ldg(v + b + (size_t)L * (i0 + i));
      if (REAL) {
        const double p = va.x * vb.x;
#pragma unroll
        for (int f = 0; f < kFreq; ++f) {
          const double2 ui = uf[f * kPoles + i];
          sr[f] = fma(p, ui.x, sr[f]);
          si[f] = fma(p, ui.y, si[f]);
        }
      } else {
        const double pr = va.x * vb.x + va.y * vb.y, pi = va.y * vb.x - va.x * vb.y;  // va conj(vb)
#pragma unroll
        for (int f = 0; f < kFreq; ++f) {
          const double2 ui = uf[f * kPoles + i];
          sr[f] = fma(-pi, ui.y, fma(pr, ui.x, sr[f]));
          si[f] = fma(pi, ui.x, fma(pr, ui.y, si[f]));
        }
      }
    }
  }
  __syncthreads();
  double2* red = u;  // kGreenWarps x kFreq x 32
#pragma unroll
  for (int f = 0; f < kFreq; ++f) red[(wp * kFreq + f) * 32 + lane] = make_double2(sr[f], si[f]);
  __syncthreads();
  if (wp < kFreq && live && fg * kFreq + wp < nz) {  // warp f finishes frequency f of the group
    double2 s = red[wp * 32 + lane];
    for (int q = 1; q < kGreenWarps; ++q) {
      const double2 r = red[(q * kFreq + wp) * 32 + lane];
      s.x += r.x;
      s.y += r.y;
    }
    double2* Gw = G + (size_t)(fg * kFreq + wp) * L * L;
    Gw[b + a * L] = s;
    if (REAL && a != b) Gw[a + b * L] = s;
  }
}

void green_function_batch(int L, int M, const double* e, const double* v, bool real, int nz,
                          const double* z, double* G, cudaStream_t s) {
  if (nz <= 0 || L <= 0) return;
  QCMG_CHECK_ARG((size_t)std::max(M, 1) * sizeof(double2) <= 200 * 1024, "too many poles for one shared-memory pass");
  const int nel = real ? L * (L + 1) / 2 : L * L, nfg = (nz + kFreq - 1) / kFreq;
  const size_t threads = (size_t)nfg * nel;
  QCMG_CHECK_ARG(threads < (1u << 31), "too many frequencies for one call");
  // frequency groups that 32 consecutive threads can meet
  const int groups = (int)std::min<size_t>(nfg, 31 / nel + 2);
  const size_t smem = std::max((size_t)groups * kFreq * kPoles, (size_t)kGreenWarps * kFreq * 32) * sizeof(double2);
  auto kern = real ? k_green<true> : k_green<false>;
  if (smem > 48 * 1024)
    QCMG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<(unsigned)((threads + 31) / 32), 32 * kGreenWarps, smem, s>>>(
      L, M, nel, nz, e, (const double2*)v, (const double2*)z, (double2*)G);
  QCMG_CUDA(cudaGetLastError());
}

}  // namespace qcmg
