// Band Lanczos (Freund) on chip: the recurrence of band_lanczos
// (qcmg_krylov.cu; pyqcm src_ed/Hamiltonian/Lanczos.hpp:214-395) for p start
// vectors inside one thread-block cluster, many steps per launch, in the
// manner of qcmg_chip.cu.
//
// On a 3,920-state impurity sector a step was five launches and a host wait,
// ~63 us; here it is two cluster barriers: after the norm and the band dots of
// v_j (one reduction for all of them; v_j goes out to every CTA meanwhile), and
// after the Gram-Schmidt update of the next p - 1 vectors, the product and the
// band recurrence with its closing dot. The 2p + 1 vectors of the band live
// in shared memory, each CTA's part of them; only v_j is held whole (the
// hops gather from it). One impurity of the 2x2 + 4 bath model from its
// parameters to G (two runs of ~111 steps among it): 11.4 ms -> 6.9 ms;
// two barriers instead of three and 32 states a tile 5.49 -> 5.13 ms later.
// (A second buffer for the whole vector, so that v_{j+1} goes out with its
// update, makes no difference: 3,920 states, p = 4, 272 steps 5.68 ms with
// one as with two, 10,584 states, p = 8 18.4 ms.)
// The dots of a tile are added over the lanes together, by a reduction that
// halves the values per lane at each step (2p - 1 additions instead of 5p).
//
// A vector whose norm falls below the deflation threshold ends the on-chip
// run; the caller then takes the general path from the start (sectors whose
// Krylov space is exhausted, or dependent start vectors).
#include <algorithm>
#include <cmath>

#include "qcmg_chip.cuh"
#include "qcmg_pool.h"
#include "qcmg_tridiag.h"
#include "qcmg_vec.cuh"

namespace qcmg {

constexpr int kBandChunk = 16;  // steps per launch

struct ChipBand {
  ChipOp op;
  const double* phi;  // p x D
  double* ring;       // (2p + 1) x D: the band's vectors between launches
  double* coef;       // page-locked: per step z, c_1..c_{p-1}, d, p projections
  int* deflated;      // page-locked: the step at which a vector deflated, or -1
  int j0, steps;
  double acc_defl;
};

constexpr int pow2_of(int n) { return n <= 1 ? 1 : 2 * pow2_of((n + 1) / 2); }

// Step j (u_j: v_j before normalization):
//   u_j to every CTA's x; z = |u_j| and <u_{j+i}, u_j>             one barrier
//   v_j = u_j / z; v_{j+i} -= c_i v_j; w = H v_j - sum_k T(k, j) v_k;
//   d = <w, v_j>                                                  one barrier
//   w -= d v_j
template <int P>
__global__ void __launch_bounds__(kChipThreads, 1) k_chip_band(ChipBand S) {
  constexpr int R = 2 * P + 1;
  extern __shared__ double sm[];
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const ChipOp& A = S.op;
  const uint32_t D = A.D;
  const int nt = (int)((D + kTile - 1) / kTile), per = (nt + C - 1) / C;
  const int t0 = min(nt, rank * per), t1 = min(nt, t0 + per);
  const int seg = per * kTile;
  double* x = sm;                          // D: u_j
  double* v = x + D;                       // R x seg: the band's vectors, this CTA's part
  double* dg = v + R * seg;                // seg
  double* part = dg + seg;                 // (2 P + 1) x nt
  __shared__ double tot[2 * P + 1], zs[2], ds;
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, nw = kChipThreads / 32;
  if (*(volatile int*)S.deflated >= 0) return;  // an earlier launch ended the run
  for (int t = t0 + wp; t < t1; t += nw) {
    const uint32_t i = t * kTile + lane, a = (t - t0) * kTile + lane;
    dg[a] = i < D ? chip_diag(A, i % A.du, i / A.du) : 0.0;
    for (int k = 0; k < R; ++k) {
      double y = 0.0;
      if (i < D) y = S.j0 > 0 ? S.ring[(size_t)k * D + i] : (k < P ? S.phi[(size_t)k * D + i] : 0.0);
      v[k * seg + a] = y;
    }
  }
  // the V sums of tile t to every CTA: value m goes to part[m nt + t]
  auto send = [&](auto& acc, int count, int first, int t) {
    constexpr int V = sizeof(acc) / sizeof(double), sub = 32 / V;
    const double s = lane_sums<V>(acc, lane);
    const int m = lane / sub;
    if (m < count)
      for (int r = lane % sub; r < C; r += sub) cl.map_shared_rank(part, r)[(first + m) * nt + t] = s;
  };
  auto total = [&](int m) {  // one warp: the sum of value m's tiles, fixed order
    double s = 0.0;
    for (int t = lane; t < nt; t += 32) s += part[m * nt + t];
    return warp_total(s);
  };
  cl.sync();
  for (int s = 0; s < S.steps; ++s) {
    const int j = S.j0 + s;
    int slot[R];  // slot[k]: v_{j - P + k}
#pragma unroll
    for (int k = 0; k < R; ++k) slot[k] = ((j + k + P + 1) % R) * seg;  // j - P + k + R, mod R
    const bool proj = j < P;
    // |u_j|^2, <u_{j+i}, u_j>, and while j < p <phi_k, u_j>
    for (int t = t0 + wp; t < t1; t += nw) {
      double acc[pow2_of(P)] = {}, pr[pow2_of(P)] = {};
      const uint32_t i = t * kTile + lane, a = (t - t0) * kTile + lane;
      const double vj = v[slot[P] + a];
#pragma unroll
      for (int k = 0; k < P; ++k) acc[k] = v[slot[P + k] + a] * vj;
      if (proj && i < D)
#pragma unroll
        for (int k = 0; k < P; ++k) pr[k] = S.phi[(size_t)k * D + i] * vj;
      if (i < D)
        for (int r = 0; r < C; ++r) cl.map_shared_rank(x, r)[i] = vj;
      send(acc, P, 0, t);
      if (proj) send(pr, P, P, t);
    }
    cl.sync();
    for (int m = wp; m < (proj ? 2 * P : P); m += nw) {
      const double y = total(m);
      if (lane == 0) {
        tot[m] = y;
        if (m == 0) root_and_inverse(y, zs);
      }
    }
    __syncthreads();
    const double z = zs[0], iz = zs[1];
    if (z < S.acc_defl) {  // the same decision in every CTA
      if (rank == 0 && threadIdx.x == 0) *S.deflated = j;
      return;
    }
    double* co = S.coef + (size_t)s * (2 * P + 1);
    if (rank == 0 && threadIdx.x == 0) {
      co[0] = z;
      for (int k = 1; k < P; ++k) co[k] = tot[k] * iz;
      for (int k = 0; k < P; ++k) co[P + 1 + k] = proj ? tot[P + k] * iz : 0.0;
    }
    double c[P];  // T(j - p + k, j): c_0 = z
#pragma unroll
    for (int k = 0; k < P; ++k) c[k] = k ? tot[k] * iz : z;
    for (int t = t0 + wp; t < t1; t += nw) {
      const uint32_t i = t * kTile + lane, a = (t - t0) * kTile + lane;
      double acc[1] = {0.0}, w = 0.0;
      const double y = v[slot[P] + a] * iz;
      v[slot[P] + a] = y;
#pragma unroll
      for (int k = 1; k < P; ++k) v[slot[P + k] + a] = fma(-c[k], y, v[slot[P + k] + a]);
      if (i < D) {
        const uint32_t id = i / A.du, iu = i - id * A.du;
        w = fma(dg[a], y, chip_hops(A, x, iu, id, 0.0) * iz);
#pragma unroll
        for (int k = 0; k < P; ++k)
          if (j - P + k >= 0) w = fma(-c[k], v[slot[k] + a], w);
        acc[0] = w * y;
      }
      v[slot[2 * P] + a] = w;
      send(acc, 1, 2 * P, t);
    }
    cl.sync();  // all gathers from x are over, too
    if (wp == 0) {
      const double y = total(2 * P);
      if (lane == 0) ds = y;
    }
    __syncthreads();
    const double d = ds;
    if (rank == 0 && threadIdx.x == 0) co[P] = d;
    for (int t = t0 + wp; t < t1; t += nw) {
      const uint32_t a = (t - t0) * kTile + lane;
      v[slot[2 * P] + a] = fma(-d, v[slot[P] + a], v[slot[2 * P] + a]);
    }
    // a thread reads and writes its own elements only, so the next step needs
    // no barrier here
  }
  for (int t = t0 + wp; t < t1; t += nw) {
    const uint32_t i = t * kTile + lane, a = (t - t0) * kTile + lane;
    if (i < D)
      for (int k = 0; k < R; ++k) S.ring[(size_t)k * D + i] = v[k * seg + a];
  }
}

static size_t band_smem(uint32_t D, int p, int C) {
  const size_t nt = (D + kTile - 1) / kTile, per = (nt + C - 1) / C;
  return (D + (2 * p + 2) * per * kTile + (2 * p + 1) * nt) * sizeof(double);
}

constexpr int kBandMaxP = 12;

template <int P, class F>
static void with_band_kernel(int p, F&& f) {
  if constexpr (P > 0) {
    if (p != P) return with_band_kernel<P - 1>(p, f);
    f(k_chip_band<P>);
  }
}

bool chip_band_fits(const qcmg_hamiltonian* H, int p) {
  int optin = 0;
  QCMG_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, H->device));
  return chip_fits(H) && p <= kBandMaxP && band_smem((uint32_t)H->dim, p, 8) <= (size_t)optin - 1024;
}

bool chip_band(qcmg_hamiltonian* H, int p, const double* phi, int M0, double acc_defl,
               double acc_band, std::vector<double>& t, std::vector<double>& P, int* M) {
  const uint32_t D = (uint32_t)H->dim;
  int optin = 0;
  QCMG_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, H->device));
  const int per_step = 2 * p + 1, chunk_len = kBandChunk * per_step;
  PoolBuf<double> ring;
  ring.alloc((size_t)(2 * p + 1) * D);
  PinnedBuf<double> coef;  // two chunks, then the flag
  coef.alloc(2 * (size_t)chunk_len + 1);
  volatile int* deflated = reinterpret_cast<int*>(coef.p + 2 * chunk_len);
  *deflated = -1;
  // a lane of its own, after what the handle's stream holds (the start
  // vectors); closed (waited for) before the buffers above go
  PoolStream lane;
  lane.open();
  QCMG_CUDA(cudaEventRecord(lane.e[0], H->stream));
  QCMG_CUDA(cudaStreamWaitEvent(lane.s, lane.e[0], 0));
  cudaStream_t s = lane.s;
  ChipBand S;
  S.op = chip_op(H);
  S.phi = phi;
  S.ring = ring.p;
  S.deflated = const_cast<int*>(deflated);
  S.acc_defl = acc_defl;
  int C = 8;
  auto launch = [&](int c) {
    S.j0 = c * kBandChunk;
    S.steps = std::min(kBandChunk, M0 - S.j0);
    if (S.steps <= 0) return;
    S.coef = coef.p + (size_t)(c & 1) * chunk_len;
    with_band_kernel<kBandMaxP>(p, [&](auto kern) {
      if (c == 0) {
        QCMG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - 1024));
        if (clusters_run(kern, 16, band_smem(D, p, 16))) C = 16;
      }
      launch_clusters(kern, 1, C, band_smem(D, p, C), s, S);
    });
    QCMG_CUDA(cudaEventRecord(lane.e[c & 1], s));
  };
  t.assign((size_t)M0 * M0, 0.0);
  P.assign((size_t)p * M0, 0.0);
  auto T = [&](int r, int c) -> double& { return t[(size_t)r + (size_t)M0 * c]; };
  double ev_old = 1e12, last_change = INFINITY;
  launch(0);
  for (int c = 0;; ++c) {
    launch(c + 1);  // computed in vain if this chunk converges
    const int j0 = c * kBandChunk, n = std::min(kBandChunk, M0 - j0);
    if (n <= 0) break;
    QCMG_CUDA(cudaEventSynchronize(lane.e[c & 1]));
    const double* co = coef.p + (size_t)(c & 1) * chunk_len;
    const int stop = *deflated;
    for (int q = 0; q < n; ++q, co += per_step) {
      const int j = j0 + q;
      if (stop >= 0 && j >= stop) return false;
      if (j >= p) T(j, j - p) = co[0];
      for (int i = 1; i < p; ++i)
        if (j + i >= p) T(j, j + i - p) = co[i];
      for (int k = std::max(0, j - p); k < j; ++k) T(k, j) = T(j, k);
      T(j, j) = co[p];
      if (j < p)
        for (int k = 0; k < p; ++k) P[k + (size_t)p * j] = co[p + 1 + k];
      if (!std::isfinite(co[0]) || !std::isfinite(co[p])) return false;
      if (j >= 4 * p && j % p == 0) {
        const bool warm = ev_old < 1e12;
        const double width =
            std::isfinite(last_change) && warm
                ? std::max(4.0 * last_change, 1e-12 * std::max(1.0, std::fabs(ev_old)))
                : 1e-3 * std::max(1.0, std::fabs(ev_old));
        const double e0 = warm ? band_lowest(t, M0, j, p, ev_old, width) : band_lowest(t, M0, j, p);
        const double test = std::fabs(e0 - ev_old);
        if (ev_old < 1e12) last_change = test;
        ev_old = e0;
        if (test < acc_band) {
          *M = j;
          return true;
        }
      }
    }
  }
  *M = M0;
  return true;
}

}  // namespace qcmg
