// Band Lanczos steps on sectors larger than a cluster's shared memory, three
// launches per step and no host round trip: the step's coefficients (the norm
// of v_j, the band dots, the closing dot) stay in device memory, and the
// host reads them p steps at a time for its convergence probe while the next
// p steps run.
//   k_band_dots   applies the last step's coefficients (v_{j-1} /= z,
//                 v_{j-1+k} -= c_k v_{j-1}, the closing dot on v_{j+p-1}), then
//                 |v_j|^2 and <v_{j+i}, v_j>; the last block forms z and c_i
//   (product)     w = H u, u = z v_j as it stands
//   k_band_recur  w = w / z - sum_k T(k, j) v_k and <w, v_j>; the last block
//                 adds it up
// Each is one pass with the loads of all its vectors in flight together; the
// FP64 pipe (12 + 12 + 14 FMAs per element at p = 12, and ~37 of the product)
// is the floor: 87 us per step at 731,808 states. Five launches with a host
// wait and a host-side sum per step took ~190 us, four (the scaling and the
// updates in a pass of their own) ~140 us, these ~115 us (600 steps and
// G: 146 -> 117 -> 103 ms, 35 of them the host's eigenproblem of the
// 600 x 600 band).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "qcmg_band.h"
#include "qcmg_pool.h"
#include "qcmg_tridiag.h"
#include "qcmg_vec.cuh"

namespace qcmg {

// Coefficients of one step: z, c_1 .. c_{p-1}, d, 1/z.
__host__ __device__ inline int row_len(int p) { return p + 2; }

// True in every thread of the block that finishes last (its partials and all
// others' are then visible); the counter is left at zero.
__device__ __forceinline__ bool last_block(unsigned* ticket) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    if (last) *ticket = 0;
  }
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// Fixed-order sum of value k's nb partials, by one warp.
__device__ __forceinline__ double sum_partials(const double* part, int nb, int m, int k) {
  double s = 0.0;
  for (int b = threadIdx.x & 31; b < nb; b += 32) s += __ldcg(part + (size_t)b * m + k);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// V: v_{j+p-1} first, then v_j .. v_{j+p-2} (the vector with the closing dot
// at a fixed place keeps the packs in registers); u = v_{j-1} (null at j = 0)
// and prev its row: c_k is the coefficient of v_{j-1+k}, prev[p] the closing
// dot's.
template <int MAXM, int VEC>
__global__ void __launch_bounds__(kDotThreads, 2)
    k_band_dots(MutVecList V, int p, double* u, const double* __restrict__ prev, size_t nv,
                double* __restrict__ part, unsigned* ticket, double* __restrict__ row, int j,
                double acc_defl, int* flag) {
  if (*(volatile int*)flag >= 0) return;
  __shared__ double cs[MAXM + 1];  // of V's vectors, in V's order; then 1/z
  if (u && threadIdx.x <= p) cs[threadIdx.x] = prev[threadIdx.x == 0 ? p : threadIdx.x == p ? p + 1 : threadIdx.x];
  __syncthreads();
  double acc[MAXM];
#pragma unroll
  for (int k = 0; k < MAXM; ++k) acc[k] = 0.0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nv;
       i += (size_t)gridDim.x * blockDim.x) {
    Pack<VEC> v[MAXM];
#pragma unroll
    for (int k = 0; k < MAXM; ++k)
      if (k < p) v[k] = load_pack<VEC>(V[k], i);
    if (u) {
      Pack<VEC> y = load_pack<VEC>(u, i);
#pragma unroll
      for (int e = 0; e < VEC; ++e) y.e[e] *= cs[p];
      store_pack<VEC>(u, i, y);
#pragma unroll
      for (int k = 0; k < MAXM; ++k)
        if (k < p) {
#pragma unroll
          for (int e = 0; e < VEC; ++e) v[k].e[e] = fma(-cs[k], y.e[e], v[k].e[e]);
          store_pack<VEC>(V[k], i, v[k]);
        }
    }
    Pack<VEC> x = v[0];
    if (p > 1) x = v[1];
#pragma unroll
    for (int k = 0; k < MAXM; ++k)
      if (k < p)
#pragma unroll
        for (int e = 0; e < VEC; ++e) acc[k] = fma(v[k].e[e], x.e[e], acc[k]);
  }
  block_sums<MAXM>(acc, p, part + (size_t)blockIdx.x * p);
  if (!last_block(ticket)) return;
  __shared__ double tot[MAXM];
  for (int k = threadIdx.x >> 5; k < p; k += kDotThreads / 32) {
    const double s = sum_partials(part, (int)gridDim.x, p, k);
    if ((threadIdx.x & 31) == 0) tot[k ? k - 1 : p - 1] = s;  // back to v_j, v_{j+1}, ...
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const double z = sqrt(tot[0]), iz = 1.0 / z;
    row[0] = z;
    for (int k = 1; k < p; ++k) row[k] = tot[k] * iz;
    row[p + 1] = iz;
    if (z < acc_defl) *flag = j;
  }
}

// V: the m = min(p, j) vectors v_{j-m} .. v_{j-1}; u = z v_j, w = H u
template <int MAXM, int VEC>
__global__ void __launch_bounds__(kDotThreads, 2)
    k_band_recur(VecList V, int m, int p, double* __restrict__ w, const double* __restrict__ u,
                 size_t nv, double* __restrict__ part, unsigned* ticket, double* __restrict__ row,
                 const int* flag) {
  if (*(volatile const int*)flag >= 0) return;
  __shared__ double cs[MAXM + 1];
  if (threadIdx.x < m) cs[threadIdx.x] = row[p - m + threadIdx.x];
  if (threadIdx.x == 0) cs[MAXM] = row[p + 1];
  __syncthreads();
  const double iz = cs[MAXM];
  double acc[1] = {0.0};
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nv;
       i += (size_t)gridDim.x * blockDim.x) {
    Pack<VEC> v[MAXM];
#pragma unroll
    for (int k = 0; k < MAXM; ++k)
      if (k < m) v[k] = load_pack<VEC>(V[k], i);
    Pack<VEC> s = load_pack<VEC>(w, i);
    Pack<VEC> y = load_pack<VEC>(u, i);
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
      s.e[e] *= iz;
      y.e[e] *= iz;
    }
#pragma unroll
    for (int k = 0; k < MAXM; ++k)
      if (k < m)
#pragma unroll
        for (int e = 0; e < VEC; ++e) s.e[e] = fma(-cs[k], v[k].e[e], s.e[e]);
    store_pack<VEC>(w, i, s);
#pragma unroll
    for (int e = 0; e < VEC; ++e) acc[0] = fma(s.e[e], y.e[e], acc[0]);
  }
  block_sums<1>(acc, 1, part + blockIdx.x);
  if (!last_block(ticket)) return;
  if (threadIdx.x < 32) {
    const double s = sum_partials(part, (int)gridDim.x, 1, 0);
    if (threadIdx.x == 0) row[p] = s;
  }
}

// <phi_k, v_j> of an unnormalized v_j for k < p (the first p steps only):
// block (k, b)'s share, which the host adds up.  With a block per k, 731,808
// states took 677 us a step, 27 us this way.
constexpr int kProjBlocks = 32;
__global__ void __launch_bounds__(256) k_band_project(const double* __restrict__ phi, size_t n,
                                                      const double* __restrict__ v,
                                                      double* __restrict__ out) {
  const double* f = phi + (size_t)blockIdx.x * n;
  double acc[1] = {0.0};
#pragma unroll 4
  for (size_t i = blockIdx.y * 256u + threadIdx.x; i < n; i += 256u * kProjBlocks)
    acc[0] = fma(f[i], v[i], acc[0]);
  block_sums<1>(acc, 1, out + blockIdx.x * kProjBlocks + blockIdx.y);
}

namespace {

// f(integral constant) with the smallest list size of the kernels >= p
template <class F>
void with_size(int p, F&& f) {
  if (p <= 4)
    f(std::integral_constant<int, 4>{});
  else if (p <= 8)
    f(std::integral_constant<int, 8>{});
  else if (p <= 12)
    f(std::integral_constant<int, 12>{});
  else
    f(std::integral_constant<int, 16>{});
}

// The events of two chunks of steps; the stream is waited for before they, and
// the buffers declared ahead of them, go.
struct Wait {
  cudaEvent_t e[2] = {nullptr, nullptr};
  Drain drain;
  explicit Wait(cudaStream_t st) : drain(st) {
    for (auto& x : e) QCMG_CUDA(cudaEventCreateWithFlags(&x, cudaEventDisableTiming));
  }
  ~Wait() {
    cudaStreamSynchronize(drain.s);
    for (auto x : e)
      if (x) cudaEventDestroy(x);
  }
};

}  // namespace

bool band_steps(qcmg_hamiltonian* H, int p, const double* phi, int M0, double acc_defl,
                double acc_band, const std::vector<double*>& ring, std::vector<double>& t,
                std::vector<double>& P, BandRun& run) {
  const size_t n = H->dim;
  cudaStream_t s = H->stream;
  const int R = 2 * p + 1, rl = row_len(p);
  uintptr_t low = 0;
  for (double* r : ring) low |= (uintptr_t)r;
  const bool two = (n & 1u) == 0 && (low & 15u) == 0;
  const size_t nv = two ? n / 2 : n;
  // two blocks per SM, at p = 12 those that the registers leave resident: one
  // round of equal shares; three took the recurrence 1.5 rounds (green run
  // 106.8 ms, 102.5). Smaller bands could hold three or four; with two,
  // 731,808 states take 112 to 118 us a step at p = 1 to 4 and 144 at p = 8
  // (168 to 172 and 223 by the host-driven loop)
  const unsigned grid = (unsigned)std::max<size_t>(1, std::min<size_t>((nv + kDotThreads - 1) / kDotThreads, 2 * 152));
  PoolBuf<double> rows, proj, part;
  PinnedBuf<double> landed;  // p steps' rows and the flag, twice; the projections
  PoolBuf<int> flags;  // the deflated step, then the block counter
  rows.alloc((size_t)(M0 + 1) * rl);
  proj.alloc((size_t)p * p * kProjBlocks);
  part.alloc((size_t)grid * p);
  flags.alloc(2);
  const size_t slot = (size_t)p * rl + 1, pp = (size_t)p * p * kProjBlocks;
  landed.alloc(2 * slot + pp);
  Wait wait(s);
  const int init[2] = {-1, 0};
  QCMG_CUDA(cudaMemcpyAsync(flags.p, init, sizeof init, cudaMemcpyHostToDevice, s));
  int* flag = flags.p;
  unsigned* ticket = reinterpret_cast<unsigned*>(flags.p + 1);
  for (int k = 0; k < p; ++k)
    QCMG_CUDA(cudaMemcpyAsync(ring[k], phi + (size_t)k * n, n * 8, cudaMemcpyDeviceToDevice, s));
  auto at = [&](int k) { return ring[k % R]; };
  auto step = [&](int j) {
    double* row = rows.p + (size_t)j * rl;
    VecList B;
    MutVecList L;
    for (int k = 0; k < p; ++k) L.v[k] = at(k ? j + k - 1 : j + p - 1);
    const int m = std::min(p, j);
    for (int k = 0; k < m; ++k) B.v[k] = at(j - m + k);
    double* u = j > 0 ? at(j - 1) : nullptr;
    const double* prev = j > 0 ? row - rl : nullptr;
    double *vj = at(j), *w = at(j + p);
    with_size(p, [&](auto size) {
      constexpr int MX = decltype(size)::value;
      auto go = [&](auto vec) {
        constexpr int VC = decltype(vec)::value;
        k_band_dots<MX, VC><<<grid, kDotThreads, 0, s>>>(L, p, u, prev, nv, part.p, ticket, row, j,
                                                       acc_defl, flag);
        if (j < p)
          k_band_project<<<dim3(p, kProjBlocks), 256, 0, s>>>(phi, n, vj, proj.p + (size_t)j * p * kProjBlocks);
        matvec(H, vj, w, false, flag);
        k_band_recur<MX, VC><<<grid, kDotThreads, 0, s>>>(B, m, p, w, vj, nv, part.p, ticket, row, flag);
      };
      if (two)
        go(std::integral_constant<int, 2>{});
      else
        go(std::integral_constant<int, 1>{});
    });
    QCMG_CUDA(cudaGetLastError());
  };
  // p steps at a time, their rows and the flag copied back
  auto queue = [&](int c) {
    const int j0 = c * p, j1 = std::min(M0, j0 + p);
    if (j0 >= j1) return;
    for (int j = j0; j < j1; ++j) step(j);
    double* h = landed.p + (size_t)(c & 1) * slot;
    QCMG_CUDA(cudaMemcpyAsync(h, rows.p + (size_t)j0 * rl, (size_t)(j1 - j0) * rl * 8, cudaMemcpyDeviceToHost, s));
    QCMG_CUDA(cudaMemcpyAsync(h + (size_t)p * rl, flag, sizeof(int), cudaMemcpyDeviceToHost, s));
    if (c == 0)
      QCMG_CUDA(cudaMemcpyAsync(landed.p + 2 * slot, proj.p, pp * 8, cudaMemcpyDeviceToHost, s));
    QCMG_CUDA(cudaEventRecord(wait.e[c & 1], s));
  };
  auto T = [&](int r, int c) -> double& { return t[(size_t)r + (size_t)M0 * c]; };
  queue(0);
  for (int c = 0; c * p < M0; ++c) {
    queue(c + 1);  // runs during the probe; computed in vain if that ends the run
    QCMG_CUDA(cudaEventSynchronize(wait.e[c & 1]));
    const double* h = landed.p + (size_t)(c & 1) * slot;
    int stop;
    std::memcpy(&stop, h + (size_t)p * rl, sizeof stop);
    for (int j = c * p; j < std::min(M0, (c + 1) * p); ++j) {
      if (stop >= 0 && j >= stop) {
        run.M = stop;
        return false;
      }
      const double* row = h + (size_t)(j - c * p) * rl;
      if (j >= p) T(j, j - p) = row[0];
      for (int i = 1; i < p; ++i)
        if (j + i >= p) T(j, j + i - p) = row[i];
      for (int k = std::max(0, j - p); k < j; ++k) T(k, j) = T(j, k);
      T(j, j) = row[p];
      if (j < p)
        for (int k = 0; k < p; ++k) {
          double part[kProjBlocks];
          std::memcpy(part, landed.p + 2 * slot + ((size_t)j * p + k) * kProjBlocks, sizeof part);
          for (int w = kProjBlocks / 2; w > 0; w /= 2)  // pairwise
            for (int b = 0; b < w; ++b) part[b] += part[b + w];
          P[k + (size_t)p * j] = part[0] * row[p + 1];
        }
      if (j >= 4 * p && j % p == 0) {
        const bool warm = run.ev_old < 1e12;
        const double width = std::isfinite(run.last_change) && warm
                                 ? std::max(4.0 * run.last_change, 1e-12 * std::max(1.0, std::fabs(run.ev_old)))
                                 : 1e-3 * std::max(1.0, std::fabs(run.ev_old));
        const double e0 = warm ? band_lowest(t, M0, j, p, run.ev_old, width) : band_lowest(t, M0, j, p);
        const double test = std::fabs(e0 - run.ev_old);
        if (run.ev_old < 1e12) run.last_change = test;
        run.ev_old = e0;
        if (test < acc_band) {
          run.M = j;
          return true;
        }
      }
    }
  }
  run.M = M0;
  return true;
}

}  // namespace qcmg
