// Lehmann Green function of a Q-matrix, batched over frequencies:
//   G_w(b, a) = sum_i v(a,i) u_w(i) conj(v(b,i)),  u_w(i) = 1 / (z_w - e_i)
// (src_ed/Q_matrix.hpp:133-151 with VDVH_naive, src_util/VDVH_kernel.cpp:28-48).
//
// A thread owns one matrix element of F frequencies, so the product
// v_a conj(v_b) is formed once per pole for all of them; with a real v only
// the elements a <= b are computed (G is symmetric) and a pole costs
// 1 + 2 F FP64 instructions instead of 8 F per element. The
// eight warps of a block take every eighth pole and are added in a fixed
// order, which keeps the chip's FP64 pipes busy at a few hundred frequencies;
// u_w is tabulated in shared memory, one tile of poles at a time.
// L = 12, 1,100 poles, 256 frequencies: 979 us, 205 us now.
//
// F = 4 where the chip is filled that way. A grid of less than a block per SM
// is bound by the FP64 pipe of the few SMs it has (most of it the table u of
// the block's 32 F / elements frequencies): F = 2 or 1 then, a quarter of the
// work per block. L = 4, 480 poles, 200 frequencies: 79 us with F = 4
// (16 blocks, tiles of 32 poles), 28 us with F = 1 (63 blocks, tiles of 128).
// The sums of an element, and their order, are the same for every F.
#include "qcmg_internal.h"
#include "qcmg_krylov.h"

namespace qcmg {

constexpr int kGreenWarps = 8;

// F: frequencies per thread (F <= kGreenWarps).  A tile of u holds 128 / F
// poles (a multiple of the warps: the order of a warp's poles is the same for
// every F).
template <bool REAL, int F>
__global__ void __launch_bounds__(32 * kGreenWarps)
    k_green(int L, int M, int nel, int nz, const double* __restrict__ e,
            const double2* __restrict__ v, const double2* __restrict__ z,
            double2* __restrict__ G) {
  constexpr int kPoles = 128 / F;
  extern __shared__ double2 u[];  // frequencies of the block x kPoles, then the warps' sums
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  // thread = (frequency group, element), elements fastest; nfg groups
  const int nfg = (nz + F - 1) / F;
  const int t0 = blockIdx.x * 32, t = t0 + lane;
  const int g0 = t0 / nel, g1 = min((t0 + 31) / nel, nfg - 1);
  const int f0 = g0 * F, nf = (g1 - g0 + 1) * F;
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
  double sr[F], si[F];
#pragma unroll
  for (int f = 0; f < F; ++f) sr[f] = si[f] = 0.0;
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
    const double2* uf = u + (fg - g0) * F * kPoles;
#pragma unroll 4
    for (int i = wp; i < np; i += kGreenWarps) {
      const double2 va = __ldg(v + a + (size_t)L * (i0 + i)), vb = __ldg(v + b + (size_t)L * (i0 + i));
      if (REAL) {
        const double p = va.x * vb.x;
#pragma unroll
        for (int f = 0; f < F; ++f) {
          const double2 ui = uf[f * kPoles + i];
          sr[f] = fma(p, ui.x, sr[f]);
          si[f] = fma(p, ui.y, si[f]);
        }
      } else {
        const double pr = va.x * vb.x + va.y * vb.y, pi = va.y * vb.x - va.x * vb.y;  // va conj(vb)
#pragma unroll
        for (int f = 0; f < F; ++f) {
          const double2 ui = uf[f * kPoles + i];
          sr[f] = fma(-pi, ui.y, fma(pr, ui.x, sr[f]));
          si[f] = fma(pi, ui.x, fma(pr, ui.y, si[f]));
        }
      }
    }
  }
  __syncthreads();
  double2* red = u;  // kGreenWarps x F x 32
#pragma unroll
  for (int f = 0; f < F; ++f) red[(wp * F + f) * 32 + lane] = make_double2(sr[f], si[f]);
  __syncthreads();
  if (wp < F && live && fg * F + wp < nz) {  // warp f finishes frequency f of the group
    double2 s = red[wp * 32 + lane];
    for (int q = 1; q < kGreenWarps; ++q) {
      const double2 r = red[(q * F + wp) * 32 + lane];
      s.x += r.x;
      s.y += r.y;
    }
    double2* Gw = G + (size_t)(fg * F + wp) * L * L;
    Gw[b + a * L] = s;
    if (REAL && a != b) Gw[a + b * L] = s;
  }
}

template <int F>
static void launch_green(int L, int M, const double* e, const double* v, bool real, int nz,
                         const double* z, double* G, cudaStream_t s) {
  const int nel = real ? L * (L + 1) / 2 : L * L, nfg = (nz + F - 1) / F;
  // frequency groups that 32 consecutive threads can meet
  const int groups = (int)std::min<size_t>(nfg, 31 / nel + 2);
  const size_t smem = std::max((size_t)groups * 128, (size_t)kGreenWarps * F * 32) * sizeof(double2);
  auto kern = real ? k_green<true, F> : k_green<false, F>;
  if (smem > 48 * 1024)
    QCMG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const size_t threads = (size_t)nfg * nel;
  kern<<<(unsigned)((threads + 31) / 32), 32 * kGreenWarps, smem, s>>>(
      L, M, nel, nz, e, (const double2*)v, (const double2*)z, (double2*)G);
  QCMG_CUDA(cudaGetLastError());
}

void green_function_batch(int L, int M, const double* e, const double* v, bool real, int nz,
                          const double* z, double* G, cudaStream_t s) {
  if (nz <= 0 || L <= 0) return;
  // the interface's limit, which the kernel itself does not need: poles go
  // through shared memory a tile at a time
  QCMG_CHECK_ARG(M <= 12800, "more than 12,800 poles");
  const size_t nel = real ? L * (L + 1) / 2 : L * L;
  int dev = 0, sms = 0;
  QCMG_CUDA(cudaGetDevice(&dev));
  QCMG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  // a launch numbers its threads (elements x frequency groups) in 31 bits
  const int most = (int)std::min<size_t>(nz, std::max<size_t>(1, (((size_t)1 << 31) - 32) / nel / 4 * 4));
  for (int z0 = 0; z0 < nz;) {
    const int n = std::min(most, nz - z0);
    const double* zc = z + 2 * (size_t)z0;
    double* Gc = G + (size_t)2 * L * L * z0;
    auto threads = [&](int F) { return ((size_t)n + F - 1) / F * nel; };
    if (threads(4) >= (size_t)32 * sms)
      launch_green<4>(L, M, e, v, real, n, zc, Gc, s);
    else if (threads(2) >= (size_t)32 * sms)
      launch_green<2>(L, M, e, v, real, n, zc, Gc, s);
    else
      launch_green<1>(L, M, e, v, real, n, zc, Gc, s);
    z0 += n;
  }
}

}  // namespace qcmg
