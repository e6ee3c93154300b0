// Lanczos on chip: one thread-block cluster per sector, many steps per launch.
//
// A sector of a few thousand states is bound by latency when every step is a
// chain of six launches (3 to 7 us each on the device, and the host's share
// of launching them): 48 impurity sectors of 3,920 and 4,900 states took
// 146 ms for their ground states (104 ms of it not the host's convergence
// test), here 4.6 ms.
// The whole recurrence stays inside a cluster of up to sixteen CTAs:
//  - every CTA holds the full basis vector x in shared memory (8 D bytes), so
//    all hops are local gathers, and its own part of the second vector and of
//    the diagonal;
//  - dot products leave one partial per tile of 32 states in every CTA's
//    shared memory (distributed shared memory stores) and each CTA adds them
//    in the same order, so the result depends on neither the cluster's size
//    nor the tile's owner, and a batch gives the same bits as a single solve;
//  - the new basis vector is stored to all CTAs by its owners.
// Two cluster barriers per step and the FP64 pipe (two FMAs per SM and
// cycle, ~25 instructions per state and step) are what a step costs: 10.3 us
// for one sector of 4,900 states on sixteen CTAs with the host's test after
// every step, 22 us for 15,876 states. (With three barriers and 64 states a
// tile the batch took 4.73 ms; 33.5 us a step at 15,876 states on eight CTAs.)
// Up to 16,384 states: x then takes 128 KB of a CTA's 227 KB. Above, the
// grid-wide kernels have enough work per launch.
//
// Host side: chunks of kChunk steps; the next chunk is launched before the
// last one's coefficients are tested (one chunk is computed in vain), the
// coefficients land in page-locked memory. The basis vectors are kept for
// the ground-state vector, psi = sum_j z_j v_j, or, when they would take more
// than a quarter of the free memory, recomputed by a second run.
#include <algorithm>
#include <cmath>
#include <memory>
#include <thread>

#include "qcmg_chip.cuh"
#include "qcmg_memo.h"
#include "qcmg_pool.h"
#include "qcmg_shares.h"
#include "qcmg_tridiag.h"

namespace qcmg {

constexpr int kChunk = 16;       // steps per launch
constexpr int kKeepSteps = 320;  // basis vectors kept at most

struct ChipSector {
  ChipOp op;
  double *x, *q;     // raw and v_{j-1} between launches
  double* scale;     // beta, 1/beta between launches
  double* V;         // basis vectors of this chunk (kChunk x D), or null
  double* coef;      // page-locked: alpha then beta of this chunk
  const double* z;   // replay: coefficients of the ground state, from this chunk's first step on
  double* gs;        // replay: the ground state
  int steps;         // steps of this launch
  int first;         // the first launch of the run: q is zero
};

// Step j, with v_j = inv raw (raw in every CTA):
//   w = H v_j - beta v_{j-1};  alpha = <v_j, w>           one barrier
//   raw' = w - alpha v_j, stored to every CTA; beta' = |raw'|, inv' = 1/beta'
//                                                         one barrier
// The basis vector goes out before its norm is known and the product is
// scaled instead, so normalizing and sending it needs no barrier of its own.
__global__ void __launch_bounds__(kChipThreads, 1) k_chip_lanczos(const ChipSector* __restrict__ secs) {
  extern __shared__ double sm[];
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const ChipSector S = secs[blockIdx.x / C];
  const ChipOp& A = S.op;
  const uint32_t D = A.D;
  const int nt = (int)((D + kTile - 1) / kTile), per = (nt + C - 1) / C;
  const int t0 = min(nt, rank * per), t1 = min(nt, t0 + per);
  double* x = sm;                      // D: raw
  double* v = x + D;                   // per x kTile: v_{j-1}, then v_j
  double* q = v + per * kTile;         // per x kTile: w
  double* dg = q + per * kTile;        // per x kTile
  double* part = dg + per * kTile;     // 2 x nt
  __shared__ double slot[3];
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, nw = kChipThreads / 32;
  for (uint32_t i = threadIdx.x; i < D; i += kChipThreads) x[i] = S.x[i];
  for (int t = t0 + wp; t < t1; t += nw) {
    const uint32_t i = t * kTile + lane, a = (t - t0) * kTile + lane;
    v[a] = (i < D && !S.first) ? S.q[i] : 0.0;
    dg[a] = i < D ? chip_diag(A, i % A.du, i / A.du) : 0.0;
  }
  double beta = S.first ? 0.0 : S.scale[0], inv = S.first ? 1.0 : S.scale[1];
  // lane r of a warp stores a tile's partial to CTA r
  double* peer_part = lane < C ? cl.map_shared_rank(part, lane) : part;
  cl.sync();
  for (int s = 0; s < S.steps; ++s) {
    for (int t = t0 + wp; t < t1; t += nw) {
      const uint32_t i = t * kTile + lane, a = (t - t0) * kTile + lane;
      double d = 0.0;
      if (i < D) {
        const uint32_t id = i / A.du, iu = i - id * A.du;
        const double xi = x[i], vi = xi * inv;
        const double h = fma(dg[a], xi, chip_hops(A, x, iu, id, 0.0));
        const double w = fma(-beta, v[a], h * inv);
        v[a] = vi;
        q[a] = w;
        d = vi * w;
        if (S.V) S.V[(size_t)s * D + i] = vi;
        if (S.gs) S.gs[i] = fma(S.z[s], vi, S.gs[i]);
      }
      d = warp_total(d);
      if (lane < C) peer_part[t] = d;
    }
    cl.sync();  // all gathers from x are over, too
    tile_total<false>(part, nt, slot);
    const double alpha = slot[0];
    for (int t = t0 + wp; t < t1; t += nw) {
      const uint32_t i = t * kTile + lane, a = (t - t0) * kTile + lane;
      double d = 0.0;
      if (i < D) {
        const double w = fma(-alpha, v[a], q[a]);
        d = w * w;
        for (int r = 0; r < C; ++r) cl.map_shared_rank(x, r)[i] = w;
      }
      d = warp_total(d);
      if (lane < C) peer_part[nt + t] = d;
    }
    cl.sync();
    tile_total<true>(part + nt, nt, slot + 1);
    beta = slot[1];
    inv = slot[2];
    if (rank == 0 && threadIdx.x == 0 && S.coef) {
      S.coef[s] = alpha;
      S.coef[kChunk + s] = beta;
    }
  }
  for (int t = t0 + wp; t < t1; t += nw) {
    const uint32_t i = t * kTile + lane, a = (t - t0) * kTile + lane;
    if (i < D) {
      S.x[i] = x[i];
      S.q[i] = v[a];
    }
  }
  if (rank == 0 && threadIdx.x == 0) {
    S.scale[0] = beta;
    S.scale[1] = inv;
  }
}

// psi_i (+)= sum_j z_j v_j,i over a span of a sector's kept vectors.
struct ChipSum {
  const double* V;  // nz x D
  const double* z;
  double* psi;
  uint32_t D;
  int nz;
};
__global__ void __launch_bounds__(256) k_chip_combine(const ChipSum* __restrict__ sums, bool add) {
  const ChipSum S = sums[blockIdx.y];
  const uint32_t i = blockIdx.x * 256u + threadIdx.x;
  if (i >= S.D) return;
  double g = add ? S.psi[i] : 0.0;
#pragma unroll 4
  for (int j = 0; j < S.nz; ++j) g = fma(__ldg(S.z + j), __ldg(S.V + (size_t)j * S.D + i), g);
  S.psi[i] = g;
}

static size_t chip_smem(uint32_t D, int C) {
  const size_t nt = (D + kTile - 1) / kTile, per = (nt + C - 1) / C;
  return (D + 3 * per * kTile + 2 * nt) * sizeof(double);
}

bool chip_fits(const qcmg_hamiltonian* H) { return H->dim > 0 && H->dim <= kChipStates && H->up.nval > 0; }

namespace {

// One host thread's share of the sectors.
struct ChipGroup {
  std::vector<int> ids;  // into the caller's arrays
  int C = 1;
  size_t smem = 0;
};

}  // namespace

static void chip_group(ChipGroup& g, qcmg_hamiltonian* const* Hs, const double* const* x0, double tol,
                       int max_iter, bool keep, double* const* psi, ChipResult* res) {
  const int n = (int)g.ids.size();
  std::vector<size_t> at(n + 1, 0);  // offsets of the sectors' vectors
  for (int k = 0; k < n; ++k) at[k + 1] = at[k] + Hs[g.ids[k]]->dim;
  const size_t total = at[n];
  PoolBuf<double> xq, zbuf, gsbuf;
  std::vector<std::unique_ptr<PoolBuf<double>>> V;  // kSpan chunks of every sector each
  constexpr int kSpan = 8;
  xq.alloc(2 * total + 2 * (size_t)n);
  PoolBuf<ChipSector> secs;
  secs.alloc((size_t)2 * n);
  PoolBuf<ChipSum> sums;
  PinnedBuf<double> coef;  // [parity][sector][2 kChunk]
  coef.alloc((size_t)n * 4 * kChunk);
  std::vector<ChipSector> hs[2];  // by chunk parity: a launch still reads the other one
  PoolStream lane;  // closed (waited for) before the buffers above go
  lane.open();
  cudaStream_t s = lane.s;
  std::vector<TridiagLowest> lowest(n);
  std::vector<size_t> zat(n, 0);  // replay: offsets of the sectors' coefficients
  auto chunk_vectors = [&](int c, int k) -> double* {
    if (keep && c * kChunk >= kKeepSteps) {  // a long run: it will be repeated instead
      QCMG_CUDA(cudaStreamSynchronize(s));
      V.clear();
      keep = false;
    }
    if (!keep) return nullptr;
    while ((int)V.size() <= c / kSpan) {
      V.emplace_back(new PoolBuf<double>);
      V.back()->alloc(total * kChunk * kSpan);
    }
    // sector k's vectors of the span are contiguous: (step in span) x D
    return V[c / kSpan]->p + at[k] * kChunk * kSpan + (size_t)(c % kSpan) * kChunk * (at[k + 1] - at[k]);
  };
  auto start = [&] {
    for (int k = 0; k < n; ++k)
      QCMG_CUDA(cudaMemcpyAsync(xq.p + at[k], x0[g.ids[k]], (at[k + 1] - at[k]) * 8,
                                cudaMemcpyDeviceToDevice, s));
  };
  // chunk c of the sectors still running; which[]: their places in the launch
  auto launch = [&](int c, const std::vector<int>& which, bool replay) {
    std::vector<ChipSector>& h = hs[c & 1];
    h.resize(which.size());
    for (size_t m = 0; m < which.size(); ++m) {
      const int k = which[m];
      ChipSector& S = h[m];
      S.op = chip_op(Hs[g.ids[k]]);
      S.x = xq.p + at[k];
      S.q = xq.p + total + at[k];
      S.scale = xq.p + 2 * total + 2 * k;
      S.V = replay ? nullptr : chunk_vectors(c, k);
      S.coef = replay ? nullptr : coef.p + ((size_t)(c & 1) * n + k) * 2 * kChunk;
      S.z = nullptr;
      S.gs = nullptr;
      S.steps = kChunk;
      S.first = c == 0;
      if (replay) {
        S.z = zbuf.p + zat[k] + (size_t)c * kChunk;
        S.gs = gsbuf.p + at[k];
        S.steps = std::min(kChunk, res[g.ids[k]].niter - c * kChunk);
      }
    }
    ChipSector* d = secs.p + (size_t)(c & 1) * n;
    QCMG_CUDA(cudaMemcpyAsync(d, h.data(), h.size() * sizeof(ChipSector), cudaMemcpyHostToDevice, s));
    launch_clusters(k_chip_lanczos, (int)which.size(), g.C, g.smem, s, (const ChipSector*)d);
  };
  start();
  std::vector<int> now, next;
  for (int k = 0; k < n; ++k) now.push_back(k);
  launch(0, now, false);
  QCMG_CUDA(cudaEventRecord(lane.e[0], s));
  for (int c = 0; !now.empty(); ++c) {
    // the next chunk of every sector that may need one, before the test
    launch(c + 1, now, false);
    QCMG_CUDA(cudaEventRecord(lane.e[(c + 1) & 1], s));
    QCMG_CUDA(cudaEventSynchronize(lane.e[c & 1]));
    next.clear();
    for (int k : now) {
      ChipResult& r = res[g.ids[k]];
      const double* co = coef.p + ((size_t)(c & 1) * n + k) * 2 * kChunk;
      bool stop = false;
      for (int t = 0; t < kChunk && !stop; ++t) {
        r.alpha.push_back(co[t]);
        r.beta.push_back(co[kChunk + t]);
        r.energy = lowest[k](r.alpha, r.beta, r.z);
        const double ritz = std::fabs(r.z.back() * r.beta.back());
        stop = true;
        if (!std::isfinite(r.energy) || !std::isfinite(ritz))
          r.status = QCMG_ERR_NUMERIC;
        else if (ritz <= tol)
          r.status = QCMG_OK;
        else if ((int)r.alpha.size() > max_iter)
          r.status = QCMG_ERR_NOCONV;
        else
          stop = false;
      }
      r.niter = (int)r.alpha.size();
      if (!stop) next.push_back(k);
    }
    now.swap(next);
  }
  if (!psi) return;
  std::vector<int> want;
  for (int k = 0; k < n; ++k)
    if (psi[g.ids[k]] && res[g.ids[k]].status == QCMG_OK) want.push_back(k);
  if (want.empty()) return;
  gsbuf.alloc(total);
  std::vector<double> hz;
  std::vector<ChipSum> hsum;
  if (!keep) {  // a second run, accumulating z_j v_j
    for (int k : want) {
      zat[k] = hz.size();
      hz.insert(hz.end(), res[g.ids[k]].z.begin(), res[g.ids[k]].z.end());
    }
    zbuf.upload(hz.data(), hz.size(), s);
    QCMG_CUDA(cudaMemsetAsync(gsbuf.p, 0, total * 8, s));
    start();
    for (int c = 0;; ++c) {
      std::vector<int> which;
      for (int k : want)
        if (res[g.ids[k]].niter > c * kChunk) which.push_back(k);
      if (which.empty()) break;
      launch(c, which, true);
      QCMG_CUDA(cudaStreamSynchronize(s));
    }
  } else {
    // spans of kSpan kChunk vectors are contiguous per sector
    const int span = kSpan * kChunk;
    for (size_t v = 0; v < V.size(); ++v) {
      hsum.clear();
      hz.clear();
      uint32_t most = 0;
      for (int k : want) {
        const ChipResult& r = res[g.ids[k]];
        const int j0 = (int)v * span, m = std::min(span, (int)r.z.size() - j0);
        if (m <= 0) continue;
        hsum.push_back({V[v]->p + at[k] * span, nullptr, gsbuf.p + at[k], (uint32_t)(at[k + 1] - at[k]), m});
        hz.insert(hz.end(), r.z.begin() + j0, r.z.begin() + j0 + m);
        most = std::max(most, hsum.back().D);
      }
      if (hsum.empty()) break;
      zbuf.upload(hz.data(), hz.size(), s);
      size_t o = 0;
      for (ChipSum& c : hsum) {
        c.z = zbuf.p + o;
        o += c.nz;
      }
      sums.upload(hsum.data(), hsum.size(), s);
      k_chip_combine<<<dim3((most + 255) / 256, (unsigned)hsum.size()), 256, 0, s>>>(sums.p, v > 0);
      QCMG_CUDA(cudaGetLastError());
      QCMG_CUDA(cudaStreamSynchronize(s));  // the host lists are rebuilt
    }
  }
  for (int k : want)
    QCMG_CUDA(cudaMemcpyAsync(psi[g.ids[k]], gsbuf.p + at[k], (at[k + 1] - at[k]) * 8,
                              cudaMemcpyDeviceToHost, s));
  QCMG_CUDA(cudaStreamSynchronize(s));
}

void chip_lanczos(int n, qcmg_hamiltonian* const* Hs, const double* const* x0, double tol,
                  int max_iter, double* const* psi, ChipResult* res) {
  if (n == 0) return;
  int dev = 0, sms = 0, optin = 0;
  QCMG_CUDA(cudaGetDevice(&dev));
  QCMG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  QCMG_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  QCMG_CUDA(cudaFuncSetAttribute(k_chip_lanczos, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 optin - 64));
  uint32_t most = 0;
  size_t states = 0;
  for (int k = 0; k < n; ++k) {
    most = std::max(most, (uint32_t)Hs[k]->dim);
    states += Hs[k]->dim;
  }
  // The portable 8, halved while the sectors ask for more than two CTAs per SM
  // and a smaller cluster's share of the vectors fits. One CTA is resident per
  // SM (103 registers and 512 threads), so some clusters of a launch may wait
  // for others to finish: 48 sectors take C = 4, 192 CTAs on 152 SMs, 4.5 ms.
  // For one sector alone sixteen, where the chip allows it
  int C = 8;
  if (n == 1) {
    // (the kernel's consent to more than eight holds for one device's context)
    static DeviceMemo<bool> wide;
    if (wide.get(dev, context_id(), [] { return clusters_run(k_chip_lanczos, 16, chip_smem(kChipStates, 16)); }))
      C = 16;
  }
  while (C > 1 && n * C > 2 * sms && chip_smem(most, C / 2) <= (size_t)optin - 64) C /= 2;
  size_t fr = 0, total = 0;
  const bool want = psi != nullptr;
  if (want) QCMG_CUDA(cudaMemGetInfo(&fr, &total));
  const bool keep = want && states * 8 * std::min<size_t>((size_t)max_iter + 2 * kChunk, kKeepSteps) <= fr / 4;
  // the test after every step is host work: share it out
  const int threads = std::max(1, std::min({8, n, (int)std::thread::hardware_concurrency() / 2}));
  std::vector<std::unique_ptr<ChipGroup>> groups;
  for (int t = 0; t < threads; ++t) {
    groups.emplace_back(new ChipGroup);
    ChipGroup& g = *groups.back();
    for (int k = t; k < n; k += threads) g.ids.push_back(k);
    g.C = C;
    for (int k : g.ids) g.smem = std::max(g.smem, chip_smem((uint32_t)Hs[k]->dim, C));
  }
  if (threads == 1) {
    chip_group(*groups[0], Hs, x0, tol, max_iter, keep, psi, res);
    return;
  }
  run_shares(threads, [&](int t) {
    QCMG_CUDA(cudaSetDevice(dev));
    chip_group(*groups[t], Hs, x0, tol, max_iter, keep, psi, res);
  });
}

}  // namespace qcmg
