// k x omega lattice integrals over the Lehmann cluster Green function
// (CPT / VCA / CDMFT), batched on the GPU in FP64.
//
// Inputs (one spin block): the cluster Green function G(z) from its
// Q-matrix (e, v), the bath hybridization Gamma(z) = tcb diag(1/(z-eb)) tcb^+,
// and the lattice hopping in Fourier form
//   t(K) - t_c = Hdiff + sum_e v_e exp(2 pi i K.R_{n_e}) |r_e><c_e|
// with K in the reduced (superlattice-dual) basis, as the reference builds it
// (lattice_model_instance::set_V, src_qcm/CPT.cpp:22-64).  Then
//   V(K,z) = t(K) - t_c - Gamma(z),
// and every per-(K,z) quantity goes through M(K,z) = G(z)^-1 - V(K,z):
//   SEF   log|det(V G - 1)| = log|det M| + log|det G|        (lattice_model_instance.cpp:624-643)
//   CPT   Gcpt = G (1 - V G)^-1 = M^-1                       (CPT.cpp:76-86)
//         g(K) = (1/L) sum_ab Gcpt_ab e^{2 pi i K.(x_b - x_a)} (lattice_model.cpp:724-740)
//   CDMFT PGF(z) = mean_K Gcpt(K, z)                          (CPT.cpp:283-345)
// G^-1 and |det G| are computed once per frequency; each (K, z) point then
// costs one LU factorization of an L x L complex matrix, done by one thread:
// up to L = 16 by the kernels of qcmg_points.cuh and qcmg_points_inv.cu, else
// with its matrix in shared memory, interleaved across threads.  Sums over a
// K grid take one point of each pair (K, -K) where V(-K) = V(K)^T.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "qcmg_internal.h"
#include "qcmg_krylov.h"
#include "qcmg_lattice.h"
#include "qcmg_points.h"
#include "qcmg_pool.h"

namespace qcmg {

struct cdbl {
  double x, y;
};
__device__ __forceinline__ cdbl cmul(cdbl a, cdbl b) { return {a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x}; }
__device__ __forceinline__ cdbl cfma_sub(cdbl acc, cdbl a, cdbl b) {  // acc - a*b, four FMAs
  return {fma(a.y, b.y, fma(-a.x, b.x, acc.x)), fma(-a.y, b.x, fma(-a.x, b.y, acc.y))};
}
__device__ __forceinline__ cdbl cinv(cdbl a) {
  double d = a.x * a.x + a.y * a.y;
  return {a.x / d, -a.y / d};
}

// ---------------------------------------------------------------------------
// Per-frequency preparation: Base(z) = G(z)^-1 + Gamma(z) - Hdiff and
// |det G(z)|, one block per frequency: in-place Gauss-Jordan elimination with
// row pivoting in shared memory. Two copies of the matrix take turns, so a
// pivot costs one barrier: every warp finds the pivot row by itself, and the
// row exchange, the scaling and the elimination are one expression per
// element (a latency-bound chain of L steps; an augmented matrix with a
// serial pivot search and seven barriers a step took 62 us for 256
// frequencies at L = 12, 26 us now).

__global__ void k_freq_prep(int L, int nw, const double2* __restrict__ G,  // nw x L x L (G[b + a L] = G(b,a))
                            const double2* __restrict__ z, int nb, const double2* __restrict__ tcb,
                            const double* __restrict__ eb, const double2* __restrict__ Hdiff,
                            double2* __restrict__ base, double* __restrict__ logdetG,
                            double* __restrict__ det2, int* __restrict__ dexp) {
  extern __shared__ double2 sm[];
  __shared__ int row_of[32];  // matrix row in each place
  const int LL = L * L, lane = threadIdx.x & 31;
  double2 *A = sm, *B1 = sm + LL;
  double dm = 1.0;  // thread 0: |det G|^2 = dm 2^de
  int de = 0;
  const int w = blockIdx.x;
  // G(r, c) with numpy orientation: G stored as G[b + a L] = G(b, a)  ->  G(r,c) = Gw[r + c L]
  const double2* Gw = G + (size_t)w * LL;
  for (int idx = threadIdx.x; idx < LL; idx += blockDim.x) A[idx] = Gw[idx / L + (idx % L) * L];
  if (threadIdx.x < 32) row_of[threadIdx.x] = threadIdx.x;
  __syncthreads();
  for (int p = 0; p < L; ++p) {
    const bool in = lane >= p && lane < L;
    const double2 mine = in ? A[lane * L + p] : make_double2(0.0, 0.0);
    const unsigned key = in ? pivot_key(mine.x, mine.y) : 0u;
    const unsigned most = __reduce_max_sync(0xffffffffu, key);
    const int piv = __ffs(__ballot_sync(0xffffffffu, in && key == most)) - 1;
    const double2 pp = A[piv * L + p];
    const double d2 = fma(pp.x, pp.x, pp.y * pp.y), rd = 1.0 / d2;
    const cdbl ip = {pp.x * rd, -pp.y * rd};
    for (int idx = threadIdx.x; idx < LL; idx += blockDim.x) {
      const int r = idx / L, c = idx - r * L;
      const double2 pc = A[piv * L + c];
      const cdbl t = c == p ? ip : cmul({pc.x, pc.y}, ip);  // the pivot row of the result
      cdbl v = t;
      if (r != p) {
        const int src = r == piv ? p : r;
        const double2 f = A[src * L + p];
        const double2 a = A[src * L + c];
        v = cfma_sub(c == p ? cdbl{0.0, 0.0} : cdbl{a.x, a.y}, {f.x, f.y}, t);
      }
      B1[idx] = make_double2(v.x, v.y);
    }
    if (threadIdx.x == 0) {
      det_mul(dm, de, d2);
      const int t = row_of[p];
      row_of[p] = row_of[piv];
      row_of[piv] = t;
    }
    __syncthreads();
    double2* t = A;
    A = B1;
    B1 = t;
  }
  // A is (P G)^-1 = G^-1 P^T: its column k is column row_of[k] of G^-1
  // Base = G^-1 + Gamma - Hdiff, row-major base[r*L + c]
  const double2 zw = z[w];
  double2* B = base + (size_t)w * L * L;
  for (int at = threadIdx.x; at < LL; at += blockDim.x) {
    const int r = at / L, c = row_of[at % L], idx = r * L + c;
    double2 gi = A[at];
    double gx = gi.x - Hdiff[idx].x, gy = gi.y - Hdiff[idx].y;
    for (int i = 0; i < nb; ++i) {
      // Gamma(r,c) += tcb(r,i) conj(tcb(c,i)) / (z - eb_i)
      double2 a = tcb[r + (size_t)L * i], b = tcb[c + (size_t)L * i];
      double re = zw.x - eb[i], im = zw.y, den = re * re + im * im;
      double ur = re / den, ui = -im / den;
      double pr = a.x * b.x + a.y * b.y, pi = a.y * b.x - a.x * b.y;  // a conj(b)
      gx += pr * ur - pi * ui;
      gy += pr * ui + pi * ur;
    }
    B[idx] = make_double2(gx, gy);
  }
  if (threadIdx.x == 0) {  // the pivots are those of G itself
    logdetG[w] = 0.5 * (log(dm) + (double)de * 0.6931471805599453094);
    if (det2) {
      det2[w] = dm;
      dexp[w] = de;
    }
  }
}

// Sigma(z) = z - base with base = G^-1 + Gamma + t_c (k_freq_prep with the
// constant block -t_c); Gamma(z) alone for the hybridization function.
__global__ void k_sigma_from_base(int L, int nw, const double2* __restrict__ z,
                                  double2* __restrict__ base) {
  const int w = blockIdx.x;
  double2* B = base + (size_t)w * L * L;
  for (int idx = threadIdx.x; idx < L * L; idx += blockDim.x) {
    const int r = idx / L, c = idx % L;
    const double2 b = B[idx];
    B[idx] = make_double2((r == c ? z[w].x : 0.0) - b.x, (r == c ? z[w].y : 0.0) - b.y);
  }
}

__global__ void k_gamma(int L, int nw, const double2* __restrict__ z, int nb,
                        const double2* __restrict__ tcb, const double* __restrict__ eb,
                        double2* __restrict__ out) {
  const int w = blockIdx.x;
  const double2 zw = z[w];
  for (int idx = threadIdx.x; idx < L * L; idx += blockDim.x) {
    const int r = idx / L, c = idx % L;
    double gx = 0.0, gy = 0.0;
    for (int i = 0; i < nb; ++i) {  // the same sum as in k_freq_prep
      double2 a = tcb[r + (size_t)L * i], b = tcb[c + (size_t)L * i];
      double re = zw.x - eb[i], im = zw.y, den = re * re + im * im;
      double ur = re / den, ui = -im / den;
      double pr = a.x * b.x + a.y * b.y, pi = a.y * b.x - a.x * b.y;
      gx += pr * ur - pi * ui;
      gy += pr * ui + pi * ur;
    }
    out[(size_t)w * L * L + idx] = make_double2(gx, gy);
  }
}

void self_energy_batch(int L, int M, const double* e, const double* v, bool v_real, int nb, const double* tcb,
                       const double* eb, const double* tc, int nz, const double* z, double* sigma,
                       double* gamma, cudaStream_t s) {
  QCMG_CHECK_ARG(L > 0 && L <= 32, "Green function dimension must be 1..32");
  PoolBuf<double> G, ldg, mtc;
  Drain drain{s};
  G.alloc((size_t)2 * L * L * nz);
  if (M > 0)
    green_function_batch(L, M, e, v, v_real, nz, z, G.p, s);
  else
    QCMG_CUDA(cudaMemsetAsync(G.p, 0, (size_t)2 * L * L * nz * 8, s));
  // constant block -t_c
  std::vector<double> h((size_t)2 * L * L);
  QCMG_CUDA(cudaMemcpyAsync(h.data(), tc, h.size() * 8, cudaMemcpyDeviceToHost, s));
  QCMG_CUDA(cudaStreamSynchronize(s));
  for (double& x : h) x = -x;
  mtc.upload(h.data(), h.size(), s);
  ldg.alloc(nz);
  const size_t smem = (size_t)2 * L * L * sizeof(double2);
  k_freq_prep<<<nz, 128, smem, s>>>(L, nz, (const double2*)G.p, (const double2*)z, nb,
                                    (const double2*)tcb, eb, (const double2*)mtc.p,
                                    (double2*)sigma, ldg.p, nullptr, nullptr);
  k_sigma_from_base<<<nz, 128, 0, s>>>(L, nz, (const double2*)z, (double2*)sigma);
  if (gamma)
    k_gamma<<<nz, 128, 0, s>>>(L, nz, (const double2*)z, nb, (const double2*)tcb, eb,
                               (double2*)gamma);
  QCMG_CUDA(cudaGetLastError());
  QCMG_CUDA(cudaStreamSynchronize(s));
}

// ---------------------------------------------------------------------------
// Per-point kernel.  MODE 0: SEF (sum of log|det M| weighted), MODE 1: CPT
// periodized g(K,z), MODE 2: mean of M^-1 (CDMFT projected GF).

struct PointArgs {
  int L;
  int nw;
  const double2* base;  // nw x L x L row-major
  int nel;
  const int* el_r;
  const int* el_c;
  const int* el_n;
  const double2* el_v;
  int nR;
  const double* R;  // nR x 3
  // K points: explicit list or a grid
  int nk;
  const double* K;  // nk x 3 (explicit) or null
  int gx, gy, gz;   // grid sizes (K = (i+off)/gx, ...)
  double off;       // 0 for the SEF grid, 0.5 for the CDMFT midpoint grid
  const double* gpos;  // L x 3 (CPT)
  double2* out;        // MODE 1: nw x nk;  MODE 2: partial sums
  double* vals;        // MODE 0: the per-point values, nw x nk
  int bpf;             // MODE 0: > 0: blocks per frequency (block b works on
                       // frequency b / bpf only, so partials never mix
                       // frequencies); 0: one flat range over all points
  const double* ldg;   // MODE 0: log|det G| per frequency, added point by point
  const int* el_start;  // nR + 1 element ranges per translation
  const double2* tab;   // grid phase tables (gx + gy + gz) x nR, or null: sincos per point
};

__device__ __forceinline__ void point_K(const PointArgs& A, int ik, double* K) {
  if (A.K) {
    K[0] = A.K[3 * ik];
    K[1] = A.K[3 * ik + 1];
    K[2] = A.K[3 * ik + 2];
  } else {
    int i = ik % A.gx, j = (ik / A.gx) % A.gy, l = ik / (A.gx * A.gy);
    K[0] = (i + A.off) / A.gx;
    K[1] = A.gy > 1 ? (j + A.off) / A.gy : 0.0;
    K[2] = A.gz > 1 ? (l + A.off) / A.gz : 0.0;
  }
}

template <int MODE>
__global__ void k_points(PointArgs A) {
  extern __shared__ double smem[];
  const int T = blockDim.x, t = threadIdx.x, L = A.L, LL = L * L;
  double* mr = smem;            // LL x T
  double* mi = smem + LL * T;   // LL x T
#define MR(r, c) mr[((r) * L + (c)) * T + t]
#define MI(r, c) mi[((r) * L + (c)) * T + t]
  const size_t npts = (size_t)A.nk * A.nw;
  // points of this block: a flat range, or (bpf > 0) the K points of one
  // frequency, strided by the frequency's blocks
  const bool per_freq = MODE == 0 && A.bpf > 0;
  const size_t w_blk = per_freq ? blockIdx.x / A.bpf : 0;
  const size_t first = per_freq ? w_blk * A.nk + (blockIdx.x % A.bpf) * (size_t)T + t
                                : blockIdx.x * (size_t)T + t;
  const size_t last = per_freq ? (w_blk + 1) * A.nk : npts;
  const size_t step = per_freq ? (size_t)A.bpf * T : (size_t)gridDim.x * T;
  for (size_t pt = first; pt < last; pt += step) {
    const int w = (int)(pt / A.nk), ik = (int)(pt % A.nk);
    double K[3];
    point_K(A, ik, K);
    const double2* B = A.base + (size_t)w * LL;
    for (int e = 0; e < LL; ++e) {
      double2 b = B[e];
      mr[e * T + t] = b.x;
      mi[e * T + t] = b.y;
    }
    // M = Base - sum_e v_e e^{2 pi i K.R_n(e)} at (r_e, c_e), one phase per
    // translation: on a grid the product of the three axes' table entries,
    // else a sincos
    for (int n = 0; n < A.nR; ++n) {
      const int e0 = A.el_start[n], e1 = A.el_start[n + 1];
      if (e0 == e1) continue;
      double s, c;
      if (A.tab) {
        const int ix = ik % A.gx, iy = (ik / A.gx) % A.gy, iz = ik / (A.gx * A.gy);
        const double2 tx = A.tab[(size_t)ix * A.nR + n];
        const double2 ty = A.tab[(size_t)(A.gx + iy) * A.nR + n];
        const double2 tz = A.tab[(size_t)(A.gx + A.gy + iz) * A.nR + n];
        const double xr = tx.x * ty.x - tx.y * ty.y, xi = tx.x * ty.y + tx.y * ty.x;
        c = xr * tz.x - xi * tz.y;
        s = xr * tz.y + xi * tz.x;
      } else {
        const double* Rn = A.R + 3 * n;
        const double ph = 2.0 * M_PI * (K[0] * Rn[0] + K[1] * Rn[1] + K[2] * Rn[2]);
        sincos(ph, &s, &c);
      }
      for (int e = e0; e < e1; ++e) {
        const double2 v = A.el_v[e];
        const int r = A.el_r[e], cc = A.el_c[e];
        MR(r, cc) -= v.x * c - v.y * s;
        MI(r, cc) -= v.x * s + v.y * c;
      }
    }
    // LU with partial pivoting (row interchanges), in place.
    int perm[32];
    for (int i = 0; i < L; ++i) perm[i] = i;
    double logabs = 0.0;
    for (int p = 0; p < L; ++p) {
      int best = p;
      double bv = MR(p, p) * MR(p, p) + MI(p, p) * MI(p, p);
      for (int r = p + 1; r < L; ++r) {
        double m = MR(r, p) * MR(r, p) + MI(r, p) * MI(r, p);
        if (m > bv) {
          bv = m;
          best = r;
        }
      }
      if (best != p) {
        for (int c = 0; c < L; ++c) {
          double a = MR(p, c), b = MI(p, c);
          MR(p, c) = MR(best, c);
          MI(p, c) = MI(best, c);
          MR(best, c) = a;
          MI(best, c) = b;
        }
        int tp = perm[p];
        perm[p] = perm[best];
        perm[best] = tp;
      }
      logabs += 0.5 * log(bv);
      const cdbl ip = cinv({MR(p, p), MI(p, p)});
      for (int r = p + 1; r < L; ++r) {
        cdbl f = cmul({MR(r, p), MI(r, p)}, ip);
        MR(r, p) = f.x;
        MI(r, p) = f.y;
        for (int c = p + 1; c < L; ++c) {
          cdbl v = cfma_sub({MR(r, c), MI(r, c)}, f, {MR(p, c), MI(p, c)});
          MR(r, c) = v.x;
          MI(r, c) = v.y;
        }
      }
    }
    if (MODE == 0) {
      // log|det(VG - 1)| = log|det M| + log|det G|, formed point by point:
      // at high frequencies both terms are ~L log|z| and their sum is tiny,
      // so summing the large terms over K first would leave the result to
      // the rounding of that sum
      A.vals[pt] = logabs + (A.ldg ? A.ldg[w] : 0.0);
      (void)perm;
    } else if (MODE == 1) {
      // y = M^-1 u, u_b = e^{2 pi i K.x_b};  g = (1/L) u^+ y
      cdbl y[32];
      for (int i = 0; i < L; ++i) {
        const double* x = A.gpos + 3 * perm[i];
        double ph = 2.0 * M_PI * (K[0] * x[0] + K[1] * x[1] + K[2] * x[2]);
        double s, c;
        sincos(ph, &s, &c);
        y[i] = {c, s};  // (P u)_i
      }
      for (int i = 0; i < L; ++i)  // forward: unit lower
        for (int j = 0; j < i; ++j) y[i] = cfma_sub(y[i], {MR(i, j), MI(i, j)}, y[j]);
      for (int i = L - 1; i >= 0; --i) {  // backward: upper
        for (int j = i + 1; j < L; ++j) y[i] = cfma_sub(y[i], {MR(i, j), MI(i, j)}, y[j]);
        y[i] = cmul(y[i], cinv({MR(i, i), MI(i, i)}));
      }
      double gr = 0.0, gi = 0.0;
      for (int b = 0; b < L; ++b) {
        const double* x = A.gpos + 3 * b;
        double ph = 2.0 * M_PI * (K[0] * x[0] + K[1] * x[1] + K[2] * x[2]);
        double s, c;
        sincos(ph, &s, &c);
        // conj(u_b) y_b
        gr += c * y[b].x + s * y[b].y;
        gi += c * y[b].y - s * y[b].x;
      }
      A.out[(size_t)w * A.nk + ik] = make_double2(gr / L, gi / L);
    } else {
      // column j of M^-1: solve M x = e_j (P applied), accumulate into out
      double2* O = A.out + ((size_t)blockIdx.x * A.nw + w) * LL;  // unused layout guard
      (void)O;
      for (int j = 0; j < L; ++j) {
        cdbl y[32];
        for (int i = 0; i < L; ++i) y[i] = {perm[i] == j ? 1.0 : 0.0, 0.0};
        for (int i = 0; i < L; ++i)
          for (int q = 0; q < i; ++q) y[i] = cfma_sub(y[i], {MR(i, q), MI(i, q)}, y[q]);
        for (int i = L - 1; i >= 0; --i) {
          for (int q = i + 1; q < L; ++q) y[i] = cfma_sub(y[i], {MR(i, q), MI(i, q)}, y[q]);
          y[i] = cmul(y[i], cinv({MR(i, i), MI(i, i)}));
        }
        // accumulate column j of the inverse: out[(w*nk + ik) ...] reduced later
        for (int i = 0; i < L; ++i)
          A.out[((size_t)w * A.nk + ik) * LL + i * L + j] = make_double2(y[i].x, y[i].y);
      }
    }
  }
#undef MR
#undef MI
}

// Sum of each row of vals (nrow x ncol), one block of kSumThreads per row:
// thread t adds the elements t, t + kSumThreads, ... in order, then a fixed
// tree adds the threads' sums: an order that does not depend on the point
// kernel's grid.
constexpr int kSumThreads = 256;
__global__ void __launch_bounds__(kSumThreads) k_row_sums(const double* __restrict__ vals,
                                                          int ncol, double* __restrict__ sums) {
  __shared__ double sh[kSumThreads];
  const double* row = vals + (size_t)blockIdx.x * ncol;
  double s = 0.0;
  for (int i = threadIdx.x; i < ncol; i += kSumThreads) s += row[i];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int h = kSumThreads / 2; h > 0; h >>= 1) {
    if ((int)threadIdx.x < h) sh[threadIdx.x] += sh[threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) sums[blockIdx.x] = sh[0];
}

// ---------------------------------------------------------------------------
// host side

static int point_threads(int L) {
  // one L x L complex matrix per thread in shared memory, up to 224 KB a block
  const size_t per = (size_t)2 * L * L * 8;  // bytes per point
  int T = (int)((224 * 1024) / per);
  T = (T / 32) * 32;
  if (T > 256) T = 256;
  if (T < 32) T = 32;
  return T;
}

void Lattice::prepare(int nw, const double* z, cudaStream_t s) {
  QCMG_CHECK_ARG(L > 0 && L <= 32, "lattice Green function dimension must be 1..32");
  QCMG_CHECK_ARG(M >= 0, "Q-matrix not set");
  ws_z.upload(z, (size_t)2 * nw, s);
  ws_G.alloc((size_t)2 * L * L * nw);
  if (M > 0) {
    green_function_batch(L, M, e.p, v.p, v_real, nw, ws_z.p, ws_G.p, s);
  } else {
    QCMG_CUDA(cudaMemsetAsync(ws_G.p, 0, (size_t)2 * L * L * nw * 8, s));
  }
  base.alloc((size_t)2 * L * L * nw);
  logdetG.alloc(nw);
  det2.alloc(nw);
  dexp.alloc(nw);
  const size_t smem = (size_t)2 * L * L * sizeof(double2);
  k_freq_prep<<<nw, 128, smem, s>>>(L, nw, (const double2*)ws_G.p, (const double2*)ws_z.p, nb,
                                    (const double2*)tcb.p, eb.p, (const double2*)hdiff.p,
                                    (double2*)base.p, logdetG.p, det2.p, dexp.p);
  QCMG_CUDA(cudaGetLastError());
  prepared_nw = nw;
}

// ---------------------------------------------------------------------------
// tables over the wavevectors

// Rows of V(K) at nk points: vk[q nk + h] = sum of the elements at position q
// times e^{2 pi i K_h.R}; the phases come from the grid's axis tables (rep:
// the points' flat grid indices) or, for explicit wavevectors, a sincos.
__global__ void k_vk(int nk, const int* __restrict__ rep, const double2* __restrict__ tab, int gx,
                     int gy, const double* __restrict__ K, int nR, const double* __restrict__ R,
                     const int* __restrict__ pos_start, const int* __restrict__ pe_n,
                     const double2* __restrict__ pe_v, double2* __restrict__ vk) {
  const int h = blockIdx.x * blockDim.x + threadIdx.x, q = blockIdx.y;
  if (h >= nk) return;
  double sr = 0.0, si = 0.0;
  for (int e = pos_start[q]; e < pos_start[q + 1]; ++e) {
    const int n = pe_n[e];
    double c, s;
    if (rep) {
      const int ik = rep[h];
      const int ix = ik % gx, iy = (ik / gx) % gy, iz = ik / (gx * gy);
      const double2 tx = tab[(size_t)ix * nR + n];
      const double2 ty = tab[(size_t)(gx + iy) * nR + n];
      const double2 tz = tab[(size_t)(gx + gy + iz) * nR + n];
      const double xr = tx.x * ty.x - tx.y * ty.y, xi = tx.x * ty.y + tx.y * ty.x;
      c = xr * tz.x - xi * tz.y;
      s = xr * tz.y + xi * tz.x;
    } else {
      const double* k = K + 3 * (size_t)h;
      sincos(2.0 * M_PI * (k[0] * R[3 * n] + k[1] * R[3 * n + 1] + k[2] * R[3 * n + 2]), &s, &c);
    }
    const double2 v = pe_v[e];
    sr += v.x * c - v.y * s;
    si += v.x * s + v.y * c;
  }
  vk[(size_t)q * nk + h] = make_double2(sr, si);
}

// uk[a nk + h] = e^{2 pi i K_h.x_a}
__global__ void k_uk(int nk, const double* __restrict__ K, const double* __restrict__ gpos,
                     double2* __restrict__ uk) {
  const int h = blockIdx.x * blockDim.x + threadIdx.x, a = blockIdx.y;
  if (h >= nk) return;
  const double* k = K + 3 * (size_t)h;
  const double* x = gpos + 3 * a;
  double s, c;
  sincos(2.0 * M_PI * (k[0] * x[0] + k[1] * x[1] + k[2] * x[2]), &s, &c);
  uk[(size_t)a * nk + h] = make_double2(c, s);
}

int Lattice::grid_points(int gx, int gy, int gz, double off, cudaStream_t s, bool may_pair) {
  // pairing needs -K on the grid: offsets 0 and 1/2 (axes of one point other
  // than the first have K = 0)
  const bool pair = may_pair && paired() && (off == 0.0 || off == 0.5);
  if (rep.p && gx == rep_gx && gy == rep_gy && gz == rep_gz && off == rep_off && pair == rep_paired)
    return nrep;
  auto minus = [&](int i, int g, bool first) {
    if (g == 1 && !first) return 0;
    return off == 0.0 ? (g - i) % g : g - 1 - i;
  };
  std::vector<int> r;
  std::vector<double> w;
  const int nk = gx * gy * gz;
  for (int ik = 0; ik < nk; ++ik) {
    int p = ik;
    if (pair) {
      const int i = ik % gx, j = (ik / gx) % gy, l = ik / (gx * gy);
      p = minus(i, gx, true) + gx * (minus(j, gy, false) + gy * minus(l, gz, false));
    }
    if (ik > p) continue;
    r.push_back(ik);
    w.push_back(ik < p ? 2.0 : 1.0);
  }
  rep_off = -1.0;
  rep.upload(r.data(), r.size(), s);
  wgt.upload(w.data(), w.size(), s);
  QCMG_CUDA(cudaStreamSynchronize(s));  // r and w go out of scope
  nrep = (int)r.size();
  rep_host.swap(r);
  rep_gx = gx;
  rep_gy = gy;
  rep_gz = gz;
  rep_off = off;
  rep_paired = pair;
  return nrep;
}

void Lattice::point_tables(int h0, int nk, const double* K, int gx, int gy, int gz, double off,
                           bool u, cudaStream_t s) {
  const dim3 grid((unsigned)((nk + 127) / 128), (unsigned)std::max(nnz, 1));
  ws_v.alloc((size_t)2 * std::max(nnz, 1) * nk);
  if (nnz) {
    const double2* tb = K ? nullptr : (const double2*)phase_tables(gx, gy, gz, off, s);
    k_vk<<<grid, 128, 0, s>>>(nk, K ? nullptr : rep.p + h0, tb, gx, gy, K ? K + 3 * (size_t)h0 : nullptr,
                              nR, R.p, pos_start.p, pe_n.p, (const double2*)pe_v.p,
                              (double2*)ws_v.p);
  }
  if (u) {
    ws_u.alloc((size_t)2 * L * nk);
    k_uk<<<dim3(grid.x, L), 128, 0, s>>>(nk, K + 3 * (size_t)h0, gpos.p, (double2*)ws_u.p);
  }
  QCMG_CUDA(cudaGetLastError());
}

// Workspaces up to this size stay with the handle.
constexpr size_t kKeepBytes = (size_t)64 << 20;

void Lattice::trim_workspaces() {
  for (DevBuf<double>* b : {&ws_z, &ws_G, &ws_K, &ws_v, &ws_u, &ws_part, &ws_out, &base})
    if (b->n * 8 > kKeepBytes) b->release();
}

// Wavevectors per launch of the point kernels: a multiple of 32, the tables
// (rows of 16 bytes per wavevector) at most 256 MB.
static int points_per_launch(int rows, int nk) {
  const size_t most = ((size_t)256 << 20) / ((size_t)16 * std::max(rows, 1));
  return (int)std::min<size_t>((size_t)nk, std::max<size_t>(most / 32 * 32, 32));
}

static LuArgs lu_args(const Lattice& lat, int nw) {
  LuArgs A;
  A.nw = nw;
  A.base = (const double2*)lat.base.p;
  A.vidx = lat.vidx.p;
  A.vk = (const double2*)lat.ws_v.p;
  A.uk = (const double2*)lat.ws_u.p;
  A.det2 = lat.det2.p;
  A.dexp = lat.dexp.p;
  return A;
}

static PointArgs point_args(const Lattice& lat, int nw) {
  PointArgs A;
  A.L = lat.L;
  A.nw = nw;
  A.base = (const double2*)lat.base.p;
  A.nel = lat.nel;
  A.el_r = lat.el_r.p;
  A.el_c = lat.el_c.p;
  A.el_n = lat.el_n.p;
  A.el_v = (const double2*)lat.el_v.p;
  A.nR = lat.nR;
  A.R = lat.R.p;
  A.K = nullptr;
  A.gx = A.gy = A.gz = 1;
  A.off = 0.0;
  A.gpos = lat.gpos.p;
  A.out = nullptr;
  A.vals = nullptr;
  A.bpf = 0;
  A.ldg = nullptr;
  A.el_start = lat.el_start.p;
  A.tab = nullptr;
  return A;
}

const double* Lattice::phase_tables(int gx, int gy, int gz, double off, cudaStream_t s) {
  if (tab.p && gx == tab_gx && gy == tab_gy && gz == tab_gz && off == tab_off) return tab.p;
  // K = ((i + off)/gx, gy > 1 ? (j + off)/gy : 0, gz > 1 ? (l + off)/gz : 0), as point_K
  std::vector<double> h((size_t)2 * (gx + gy + gz) * nR);
  auto fill = [&](int base, int g, int axis) {
    for (int i = 0; i < g; ++i) {
      const double k = (axis == 0 || g > 1) ? (i + off) / g : 0.0;
      for (int n = 0; n < nR; ++n) {
        const double ph = 2.0 * M_PI * k * R_host[3 * n + axis];
        const size_t at = ((size_t)(base + i) * nR + n) * 2;
        h[at] = std::cos(ph);
        h[at + 1] = std::sin(ph);
      }
    }
  };
  fill(0, gx, 0);
  fill(gx, gy, 1);
  fill(gx + gy, gz, 2);
  tab.upload(h.data(), h.size(), s);
  QCMG_CUDA(cudaStreamSynchronize(s));
  tab_gx = gx;
  tab_gy = gy;
  tab_gz = gz;
  tab_off = off;
  return tab.p;
}

double Lattice::sef_grid(int nw, const double* w, const double* wt, int nkx, int nky, int nkz,
                         cudaStream_t s) {
  std::vector<double> z(2 * nw), hs(nw);
  for (int i = 0; i < nw; ++i) {
    z[2 * i] = 0.0;
    z[2 * i + 1] = w[i];
  }
  const int nk = nkx * nky * nkz;
  prepare(nw, z.data(), s);
  // each frequency's K sum is taken in a fixed order (k_row_sums over the
  // points, or over the warps' sums), so the weights apply to whole
  // per-frequency sums
  auto sums = [&](const double* rows, int ncol, int i0, int nf) {
    ws_out.alloc(nw);
    k_row_sums<<<nf, kSumThreads, 0, s>>>(rows, ncol, ws_out.p + i0);
    QCMG_CUDA(cudaGetLastError());
  };
  if (L <= kMaxPointL) {
    // as many frequencies at a time as leave 128 MB of warps' sums (a launch
    // then stays within a grid's 2^31 blocks)
    const int np = grid_points(nkx, nky, nkz, 0.0, s), nkb = (np + 31) / 32;
    const int fpl = (int)std::max<size_t>(1, std::min<size_t>(nw, ((size_t)16 << 20) / nkb));
    ws_part.alloc((size_t)fpl * nkb);
    const int step = points_per_launch(nnz, np);
    for (int i0 = 0; i0 < nw; i0 += fpl) {
      const int nf = std::min(fpl, nw - i0);
      for (int h0 = 0; h0 < np; h0 += step) {
        const int n = std::min(step, np - h0);
        if (step < np || i0 == 0) point_tables(h0, n, nullptr, nkx, nky, nkz, 0.0, false, s);
        LuArgs A = lu_args(*this, nf);
        A.base += (size_t)i0 * L * L;
        A.det2 += i0;
        A.dexp += i0;
        A.nk = n;
        A.wgt = wgt.p + h0;
        A.part = ws_part.p + h0 / 32;
        A.part_ld = nkb;
        launch_sef_points(L, A, s);
      }
      sums(ws_part.p, nkb, i0, nf);
    }
  } else {
    // a full matrix per thread in shared memory, several frequencies per
    // launch (enough blocks for many waves on every SM)
    const double2* phases = (const double2*)phase_tables(nkx, nky, nkz, 0.0, s);
    const int T = point_threads(L);
    const unsigned bpf = (unsigned)std::max<size_t>(1, std::min<size_t>((nk + T - 1) / T, 152 * 4));
    const int fpl = std::max(1, std::min(nw, (int)((152u * 16u + bpf - 1) / bpf)));
    const size_t smem = (size_t)2 * L * L * T * 8;
    QCMG_CUDA(cudaFuncSetAttribute(k_points<0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)smem));
    ws_part.alloc((size_t)fpl * nk);
    for (int i0 = 0; i0 < nw; i0 += fpl) {
      const int nf = std::min(fpl, nw - i0);
      PointArgs A = point_args(*this, nf);
      A.base = (const double2*)base.p + (size_t)i0 * L * L;
      A.nk = nk;
      A.gx = nkx;
      A.gy = nky;
      A.gz = nkz;
      A.off = 0.0;
      A.vals = ws_part.p;
      A.bpf = (int)bpf;
      A.ldg = logdetG.p + i0;
      A.tab = phases;
      k_points<0><<<bpf * nf, T, smem, s>>>(A);
      QCMG_CUDA(cudaGetLastError());
      sums(ws_part.p, nk, i0, nf);
    }
  }
  QCMG_CUDA(cudaMemcpyAsync(hs.data(), ws_out.p, (size_t)nw * 8, cudaMemcpyDeviceToHost, s));
  QCMG_CUDA(cudaStreamSynchronize(s));
  trim_workspaces();
  double total = 0.0;
  for (int i = 0; i < nw; ++i) total += wt[i] * (hs[i] / nk);
  return total;
}

void Lattice::cpt(int nz, const double* z, int nk, const double* K, double* g, cudaStream_t s) {
  prepare(nz, z, s);
  ws_K.upload(K, (size_t)3 * nk, s);
  ws_out.alloc((size_t)2 * nz * nk);
  if (L <= kMaxPointL) {
    const int step = points_per_launch(nnz + L, nk);
    for (int h0 = 0; h0 < nk; h0 += step) {
      const int n = std::min(step, nk - h0);
      point_tables(h0, n, ws_K.p, 1, 1, 1, 0.0, true, s);
      LuArgs A = lu_args(*this, nz);
      A.nk = n;
      A.out = (double2*)ws_out.p + h0;
      A.out_ld = nk;
      launch_cpt_points(L, A, s);
    }
  } else {
    PointArgs A = point_args(*this, nz);
    A.nk = nk;
    A.K = ws_K.p;
    A.out = (double2*)ws_out.p;
    const int T = point_threads(L);
    const size_t smem = (size_t)2 * L * L * T * 8;
    QCMG_CUDA(cudaFuncSetAttribute(k_points<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const size_t npts = (size_t)nz * nk;
    unsigned gr = (unsigned)std::max<size_t>(1, std::min<size_t>((npts + T - 1) / T, 152 * 8));
    k_points<1><<<gr, T, smem, s>>>(A);
    QCMG_CUDA(cudaGetLastError());
  }
  QCMG_CUDA(cudaMemcpyAsync(g, ws_out.p, (size_t)2 * nz * nk * 8, cudaMemcpyDeviceToHost, s));
  QCMG_CUDA(cudaStreamSynchronize(s));
  trim_workspaces();
}

// K means of the per-point inverses, per frequency and moment:
//   out[(w nmom + m) LL + e] = (1/nk) sum_K ph[m nk + K] inv[w][K][e]
// (ph null: one moment with phase 1).  One block per (frequency, 32
// consecutive elements e): the lanes take consecutive e (coalesced loads of
// each point's block), the warps interleave over K, and every moment's sums
// stay in registers until a fixed-order reduction over the warps in shared
// memory.
constexpr int kMaxMoments = 16;
constexpr int kMomWarps = 8;

__global__ void __launch_bounds__(32 * kMomWarps)
    k_mean_moments(const double2* __restrict__ inv, int nw, int nk, int LL, int nmom,
                   const double2* __restrict__ ph, double2* __restrict__ out) {
  __shared__ double red[2][kMomWarps][32];
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int w = blockIdx.x, e = blockIdx.y * 32 + lane;
  const int nm = ph ? nmom : 1;
  double sr[kMaxMoments], si[kMaxMoments];
#pragma unroll
  for (int m = 0; m < kMaxMoments; ++m) sr[m] = si[m] = 0.0;
  if (e < LL) {
    const double2* col = inv + (size_t)w * nk * LL + e;
    for (int k = wp; k < nk; k += kMomWarps) {
      const double2 v = col[(size_t)k * LL];
      if (!ph) {
        sr[0] += v.x;
        si[0] += v.y;
        continue;
      }
#pragma unroll
      for (int m = 0; m < kMaxMoments; ++m) {
        if (m < nm) {
          const double2 p = ph[(size_t)m * nk + k];
          sr[m] += v.x * p.x - v.y * p.y;
          si[m] += v.x * p.y + v.y * p.x;
        }
      }
    }
  }
#pragma unroll
  for (int m = 0; m < kMaxMoments; ++m) {
    if (m < nm) {  // the same for the whole block
      red[0][wp][lane] = sr[m];
      red[1][wp][lane] = si[m];
      __syncthreads();
      if (wp == 0 && e < LL) {
        double a = 0.0, b = 0.0;
        for (int q = 0; q < kMomWarps; ++q) {
          a += red[0][q][lane];
          b += red[1][q][lane];
        }
        out[((size_t)w * nm + m) * LL + e] = make_double2(a / nk, b / nk);
      }
      __syncthreads();
    }
  }
}

void Lattice::projected(int nw, const double* w, int kside, int dimk, double* pgf, cudaStream_t s) {
  std::vector<double> z(2 * nw);
  for (int i = 0; i < nw; ++i) {
    z[2 * i] = 0.0;
    z[2 * i + 1] = w[i];
  }
  const int g = kside;
  kmean(nw, z.data(), dimk >= 1 ? g : 1, dimk >= 2 ? g : 1, dimk >= 3 ? g : 1,
        dimk >= 1 ? 0.5 : 0.0, pgf, s);
}

void Lattice::kmean(int nz, const double* z, int gx, int gy, int gz, double off, double* out_host,
                    cudaStream_t s) {
  kmoments(nz, z, gx, gy, gz, off, 0, nullptr, out_host, s);
}

// Whether every translation is one of the lattice; pairing takes
// e^{2 pi i (1 - K).R} for e^{-2 pi i K.R}.
static bool integer_translations(int nmom, const double* Rm) {
  for (int k = 0; k < 3 * nmom; ++k)
    if (Rm[k] != std::rint(Rm[k])) return false;
  return true;
}

// Whether the means with phases go row by row (inverse_means).  A warp takes
// points of one (ky, kz), so a row of less than 32 points, or the end of a
// longer one, leaves lanes idle; below, every point's inverse is stored and
// added up afterwards, as for L > 16 (k_points, k_mean_moments).  The row form
// does that work 28 / L times as fast per lane (measured where both cost the
// same, 64 frequencies, 1,024 points: L = 8 complex 8 x 128 x 1 1.8 ms against
// 2.0, 4 x 16 x 16 3.5 against 2.0; L = 12 complex 8 x 128 x 1 11.2 against
// 6.7, 1 x 1024 x 1 88.9 against 6.6), so it is taken where the lanes that its
// batches occupy are at most 28 / L times the grid's points.
bool Lattice::long_rows(int gx, int gy, int gz, double off, bool may_pair, cudaStream_t s) {
  const int np = grid_points(gx, gy, gz, off, s, may_pair);
  size_t lanes = 0;
  for (int h = 0, h0 = 0; h < np; ++h)
    if (h + 1 == np || rep_host[h + 1] / gx != rep_host[h] / gx) {
      lanes += (size_t)(h - h0 + 32) / 32 * 32;
      h0 = h + 1;
    }
  return lanes * L <= (size_t)28 * gx * gy * gz;
}

// The means of the translations `which` of Rm (empty: the plain mean) into
// their places of out_host, nz x max(nmom, 1) x L x L.
void Lattice::inverse_means(int nz, const double* z, int gx, int gy, int gz, double off, int nmom,
                            const std::vector<int>& which, const double* Rm, double* out_host,
                            cudaStream_t s) {
  const int nk = gx * gy * gz, LL = L * L, nm = std::max<int>(1, (int)which.size());
  const int np = grid_points(gx, gy, gz, off, s, integer_translations(which.empty() ? 0 : nmom, Rm));
  const bool pair = rep_paired;
  // rows: with translations, the points of each (ky, kz), in parts of whole
  // batches of 32 that make about 2,048 warps over all frequencies (a 1,024 x
  // 1 x 1 grid in one row per frequency: 13 ms for one frequency at L = 12,
  // 0.5 ms in parts); else equal parts, about 4,096 warps
  std::vector<int> rows{0}, fx(nm, 0);
  std::vector<double> yz, wx, ax;
  if (which.empty()) {
    const int batches = (np + 31) / 32;
    const int per = std::max(1, std::min(batches, (int)((size_t)batches * nz / 4096)));
    for (int b = per; b < batches; b += per) rows.push_back(32 * b);
    rows.push_back(np);
  } else {
    const int per = 32 * (int)std::max<size_t>(1, std::min<size_t>((size_t)(np + 31) / 32, (size_t)np * nz / (32 * 2048)));
    for (int h = 1; h < np; ++h)
      if (rep_host[h] / gx != rep_host[h - 1] / gx || h - rows.back() == per) rows.push_back(h);
    rows.push_back(np);
    for (size_t q = 0; q < which.size(); ++q) {
      const double r = Rm[3 * which[q]];
      if (r == 0.0) continue;
      size_t u = std::find(ax.begin(), ax.end(), std::fabs(r)) - ax.begin();
      if (u == ax.size()) ax.push_back(std::fabs(r));
      fx[q] = (r < 0 ? -1 : 1) * (int)(2 * u + 1);
    }
    for (double r : ax)
      for (int part = 0; part < 2; ++part)
        for (int i = 0; i < gx; ++i) {
          const double a = 2.0 * M_PI * ((i + off) / gx) * r;
          wx.push_back(part ? std::sin(a) : std::cos(a));
        }
    for (int m : which)
      for (size_t r = 0; r + 1 < rows.size(); ++r) {
        const int yzi = rep_host[rows[r]] / gx, j = yzi % gy, l = yzi / gy;
        const double a = 2.0 * M_PI * ((gy > 1 ? (j + off) / gy : 0.0) * Rm[3 * m + 1] +
                                       (gz > 1 ? (l + off) / gz : 0.0) * Rm[3 * m + 2]);
        yz.push_back(std::cos(a));
        yz.push_back(std::sin(a));
      }
  }
  const int nrow = (int)rows.size() - 1, nf = 1 + 2 * (int)ax.size();
  PoolBuf<int> d_rows, d_fx;
  PoolBuf<double> d_yz, d_wx;
  Drain drain{s};
  d_rows.upload(rows.data(), rows.size(), s);
  if (!which.empty()) {
    d_fx.upload(fx.data(), fx.size(), s);
    d_yz.upload(yz.data(), yz.size(), s);
    if (!wx.empty()) d_wx.upload(wx.data(), wx.size(), s);
  }
  point_tables(0, np, nullptr, gx, gy, gz, off, false, s);
  // frequencies in chunks whose row sums fit in ~512 MB
  const size_t per_z = (size_t)nrow * nf * LL * 16;
  const int chunk = (int)std::max<size_t>(1, std::min<size_t>(nz, ((size_t)512 << 20) / per_z));
  ws_part.alloc((size_t)2 * chunk * nrow * nf * LL);
  ws_out.alloc((size_t)2 * chunk * nm * LL);
  std::vector<double> host((size_t)2 * nz * nm * LL);
  for (int z0 = 0; z0 < nz; z0 += chunk) {
    const int nc = std::min(chunk, nz - z0);
    prepare(nc, z + 2 * (size_t)z0, s);
    InvArgs A;
    A.nk = np;
    A.nw = nc;
    A.nrow = nrow;
    A.base = (const double2*)base.p;
    A.vidx = vidx.p;
    A.vk = (const double2*)ws_v.p;
    A.wgt = wgt.p;
    A.scale = pair ? 0.5 : 1.0;  // a pair's weight 2 is shared by the inverse and its transpose
    A.row_start = d_rows.p;
    A.rep = rep.p;
    A.gx = gx;
    A.nf = nf;
    A.wx = d_wx.p;
    A.part = (double2*)ws_part.p;
    launch_inverse_means(L, A, nm, which.empty() ? nullptr : d_fx.p,
                         which.empty() ? nullptr : (const double2*)d_yz.p, pair, 1.0 / nk,
                         (double2*)ws_out.p, s);
    QCMG_CUDA(cudaMemcpyAsync(host.data() + (size_t)2 * z0 * nm * LL, ws_out.p,
                              (size_t)2 * nc * nm * LL * 8, cudaMemcpyDeviceToHost, s));
    QCMG_CUDA(cudaStreamSynchronize(s));
  }
  trim_workspaces();
  const int ld = std::max(nmom, 1);
  for (int w = 0; w < nz; ++w)
    for (int q = 0; q < nm; ++q)
      std::memcpy(out_host + ((size_t)w * ld + (which.empty() ? 0 : which[q])) * 2 * LL,
                  host.data() + ((size_t)w * nm + q) * 2 * LL, (size_t)2 * LL * 8);
}

void Lattice::kmoments(int nz, const double* z, int gx, int gy, int gz, double off, int nmom,
                       const double* Rm, double* out_host, cudaStream_t s) {
  QCMG_CHECK_ARG(nmom >= 0 && nmom <= kMaxMoments, "at most 16 translations per call");
  if (L <= kMaxPointL && (nmom == 0 || long_rows(gx, gy, gz, off, integer_translations(nmom, Rm), s))) {
    // translations in groups of at most (kMaxInvFuncs - 1)/2 distinct |R_x|
    if (nmom == 0) return inverse_means(nz, z, gx, gy, gz, off, 0, {}, nullptr, out_host, s);
    std::vector<int> todo(nmom);
    for (int m = 0; m < nmom; ++m) todo[m] = m;
    while (!todo.empty()) {
      std::vector<int> now, later;
      std::vector<double> ax;
      for (int m : todo) {
        const double a = std::fabs(Rm[3 * m]);
        const bool known = a == 0.0 || std::find(ax.begin(), ax.end(), a) != ax.end();
        if (!known && (int)ax.size() >= (kMaxInvFuncs - 1) / 2) {
          later.push_back(m);
          continue;
        }
        if (!known) ax.push_back(a);
        now.push_back(m);
      }
      inverse_means(nz, z, gx, gy, gz, off, nmom, now, Rm, out_host, s);
      todo.swap(later);
    }
    return;
  }
  const int nk = gx * gy * gz, LL = L * L;
  const int T = point_threads(L);
  const size_t smem = (size_t)2 * L * L * T * 8;
  QCMG_CUDA(cudaFuncSetAttribute(k_points<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  // phase of each translation at each grid point, K as point_K lays it out
  DevBuf<double> ph;
  if (nmom > 0) {
    std::vector<double> h((size_t)2 * nmom * nk);
    for (int m = 0; m < nmom; ++m)
      for (int ik = 0; ik < nk; ++ik) {
        const int i = ik % gx, j = (ik / gx) % gy, l = ik / (gx * gy);
        const double K0 = (i + off) / gx, K1 = gy > 1 ? (j + off) / gy : 0.0,
                     K2 = gz > 1 ? (l + off) / gz : 0.0;
        const double a = 2.0 * M_PI * (K0 * Rm[3 * m] + K1 * Rm[3 * m + 1] + K2 * Rm[3 * m + 2]);
        h[2 * ((size_t)m * nk + ik)] = std::cos(a);
        h[2 * ((size_t)m * nk + ik) + 1] = std::sin(a);
      }
    ph.upload(h.data(), h.size(), s);
  }
  const int nm = nmom > 0 ? nmom : 1;
  // frequencies in chunks whose per-point inverses fit in ~512 MB
  const size_t per_z = (size_t)nk * LL * 16;
  const int chunk = (int)std::max<size_t>(1, std::min<size_t>(nz, ((size_t)512 << 20) / per_z));
  ws_part.alloc((size_t)2 * chunk * nk * LL);
  ws_out.alloc((size_t)2 * chunk * nm * LL);
  for (int z0 = 0; z0 < nz; z0 += chunk) {
    const int nc = std::min(chunk, nz - z0);
    prepare(nc, z + 2 * (size_t)z0, s);
    PointArgs A = point_args(*this, nc);
    A.gx = gx;
    A.gy = gy;
    A.gz = gz;
    A.nk = nk;
    A.off = off;
    A.tab = (const double2*)phase_tables(gx, gy, gz, off, s);
    A.out = (double2*)ws_part.p;
    const size_t npts = (size_t)nc * nk;
    unsigned gr = (unsigned)std::max<size_t>(1, std::min<size_t>((npts + T - 1) / T, 152 * 8));
    k_points<2><<<gr, T, smem, s>>>(A);
    k_mean_moments<<<dim3(nc, (LL + 31) / 32), 32 * kMomWarps, 0, s>>>(
        (const double2*)ws_part.p, nc, nk, LL, nm, nmom > 0 ? (const double2*)ph.p : nullptr,
        (double2*)ws_out.p);
    QCMG_CUDA(cudaGetLastError());
    QCMG_CUDA(cudaMemcpyAsync(out_host + (size_t)2 * z0 * nm * LL, ws_out.p,
                              (size_t)2 * nc * nm * LL * 8, cudaMemcpyDeviceToHost, s));
    QCMG_CUDA(cudaStreamSynchronize(s));
  }
  trim_workspaces();
}

}  // namespace qcmg
