// Half-basis indexing and half-operator construction on the GPU.
//
// A half basis is the increasing list of L-bit integers with N set bits
// (pyqcm src_ed/ED_basis.cpp:115-125).  For a fixed popcount, increasing
// integer order is colexicographic order of the occupied-orbital sets, so
// the rank of a state b with occupied orbitals c_1 < ... < c_N is
//     rank(b) = sum_k C(c_k, k)        (combinatorial number system)
// and a rank is unranked greedily from the top.  This replaces the
// reference's materialized list plus binary search
// (src_ed/ED_basis.cpp:130-135) with exact integer arithmetic: no table
// larger than the 33 x 33 binomials is needed on the device.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>

#include "qcmg_internal.h"
#include "qcmg_pool.h"

namespace qcmg {

__constant__ uint32_t c_binom[kMaxOrbitals + 1][kMaxOrbitals + 1];

uint64_t binomial(int n, int k) {
  if (k < 0 || n < 0 || k > n) return 0;
  uint64_t r = 1;
  for (int i = 1; i <= k; ++i) r = r * (uint64_t)(n - k + i) / (uint64_t)i;
  return r;
}

void ensure_device_tables(int device) {
  static std::mutex m;
  static std::vector<int> done;
  std::lock_guard<std::mutex> lock(m);
  if (std::find(done.begin(), done.end(), device) != done.end()) return;
  uint32_t h[kMaxOrbitals + 1][kMaxOrbitals + 1];
  for (int n = 0; n <= kMaxOrbitals; ++n)
    for (int k = 0; k <= kMaxOrbitals; ++k) h[n][k] = (uint32_t)binomial(n, k);
  QCMG_CUDA(cudaMemcpyToSymbol(c_binom, h, sizeof(h)));
  done.push_back(device);
}

__device__ __forceinline__ uint32_t dev_rank(uint32_t b) {
  uint32_t r = 0;
  int k = 1;
  while (b) {
    int c = __ffs(b) - 1;
    r += c_binom[c][k];
    ++k;
    b &= b - 1;
  }
  return r;
}

__device__ __forceinline__ uint32_t dev_unrank(uint32_t r, int L, int N) {
  uint32_t b = 0;
  int c = L - 1;
  for (int k = N; k >= 1; --k) {
    while (c_binom[c][k] > r) --c;
    b |= 1u << c;
    r -= c_binom[c][k];
    --c;
  }
  return b;
}

__global__ void k_halfbasis(int L, int N, uint32_t dim, uint32_t* out) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < dim; i += gridDim.x * blockDim.x)
    out[i] = dev_unrank(i, L, N);
}

__global__ void k_rank(int L, const uint32_t* __restrict__ st, size_t n, uint32_t dim,
                       uint32_t* __restrict__ ranks) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    uint32_t b = st[i];
    bool ok = (L >= 32) || (b >> L) == 0;
    uint32_t r = ok ? dev_rank(b) : dim;
    ranks[i] = (r < dim) ? r : dim;
  }
}

static unsigned grid_for(size_t n, unsigned block) {
  size_t g = (n + block - 1) / block;
  if (g < 1) g = 1;
  if (g > 65535u * 8) g = 65535u * 8;
  return (unsigned)g;
}

void launch_halfbasis(int L, int N, uint32_t dim, uint32_t* out, cudaStream_t s) {
  if (!dim) return;
  k_halfbasis<<<grid_for(dim, 256), 256, 0, s>>>(L, N, dim, out);
  QCMG_CUDA(cudaGetLastError());
}

void launch_rank(int L, const uint32_t* states, size_t n, uint32_t dim, uint32_t* ranks,
                 cudaStream_t s) {
  if (!n) return;
  k_rank<<<grid_for(n, 256), 256, 0, s>>>(L, states, n, dim, ranks);
  QCMG_CUDA(cudaGetLastError());
}

// Fermion sign of moving the electron at bit c to bit r: parity of the
// occupied orbitals strictly between (binary_state::interphase,
// src_ed/binary_state.hpp:42-49).
__device__ __forceinline__ int hop_parity(uint32_t b, int r, int c) {
  int lo = min(r, c), hi = max(r, c);
  uint32_t between = (hi >= 32 ? 0xffffffffu : ((1u << hi) - 1u)) & ~((2u << lo) - 1u);
  return __popc(b & between) & 1;
}

// Pass 1: entries per row (hops allowed from each state).
__global__ void k_halfop_count(uint32_t dim, const uint32_t* __restrict__ bin,
                               const HopElement* __restrict__ el, int nel,
                               uint32_t* __restrict__ cnt) {
  for (uint32_t I = blockIdx.x * blockDim.x + threadIdx.x; I < dim; I += gridDim.x * blockDim.x) {
    uint32_t b = bin[I], n = 0;
    for (int k = 0; k < nel; ++k) {
      int r = el[k].r, c = el[k].c;
      if (r == c || el[k].v == 0.0) continue;
      if (((b >> c) & 1u) && !((b >> r) & 1u)) ++n;
    }
    cnt[I] = n;
  }
}

// Pass 2: fill (J, sign * v) in element order and the diagonal.
__global__ void k_halfop_fill(uint32_t dim, const uint32_t* __restrict__ bin,
                              const HopElement* __restrict__ el, int nel,
                              const uint32_t* __restrict__ rowptr, uint32_t* __restrict__ col,
                              double* __restrict__ val, double* __restrict__ diag,
                              uint32_t* __restrict__ ell, uint16_t* __restrict__ len) {
  for (uint32_t I = blockIdx.x * blockDim.x + threadIdx.x; I < dim; I += gridDim.x * blockDim.x) {
    uint32_t b = bin[I];
    uint32_t pos = rowptr[I];
    double d = 0.0;
    for (int k = 0; k < nel; ++k) {
      int r = el[k].r, c = el[k].c;
      double v = el[k].v;
      if (r == c) {
        if ((b >> r) & 1u) d += v;
        continue;
      }
      if (v == 0.0) continue;
      if (((b >> c) & 1u) && !((b >> r) & 1u)) {
        uint32_t bp = b ^ (1u << c) ^ (1u << r);
        const uint32_t J = dev_rank(bp);
        const int neg = hop_parity(b, r, c);
        col[pos] = J;
        val[pos] = neg ? -v : v;
        if (ell) ell[(size_t)(pos - rowptr[I]) * dim + I] = J | ((uint32_t)(2 * k + neg) << 16);
        ++pos;
      }
    }
    if (ell) len[I] = (uint16_t)(pos - rowptr[I]);
    diag[I] = d;
  }
}

// rowptr from the row counts (one block; rows taken 1,024 at a time).
__global__ void __launch_bounds__(1024) k_rowptr(uint32_t dim, uint32_t* __restrict__ rp) {
  // on entry rp[i + 1] is row i's count
  __shared__ uint32_t ws[32];
  __shared__ uint32_t base;
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    base = 0;
    rp[0] = 0;
  }
  __syncthreads();
  for (uint32_t i0 = 0; i0 < dim; i0 += 1024) {
    const uint32_t i = i0 + threadIdx.x;
    uint32_t v = i < dim ? rp[i + 1] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += t;
    }
    if (lane == 31) ws[wp] = v;
    __syncthreads();
    if (wp == 0) {
      uint32_t t = ws[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t q = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= o) t += q;
      }
      ws[lane] = t;
    }
    __syncthreads();
    const uint32_t out = base + v + (wp ? ws[wp - 1] : 0);
    if (i < dim) rp[i + 1] = out;
    __syncthreads();
    if (threadIdx.x == 1023) base = out;
    __syncthreads();
  }
}

// No host round trip: a hop c -> r is allowed from the C(L-2, N-1) states
// with c occupied and r empty, so the number of entries is known beforehand.
// `staging` receives the host copies that the queued uploads read; the
// caller keeps it until the stream is idle.
void build_halfop(HalfOp& op, int L, int N, const std::vector<HopElement>& el, bool slots,
                  std::vector<std::vector<double>>& staging, cudaStream_t s) {
  op.L = L;
  op.N = N;
  uint64_t dim64 = binomial(L, N);
  QCMG_CHECK_ARG(dim64 < (1ull << 31), "half basis too large");
  op.dim = (uint32_t)dim64;
  size_t hops = 0;
  for (auto& e : el) {
    QCMG_CHECK_ARG(e.r >= 0 && e.r < L && e.c >= 0 && e.c < L, "hop element orbital out of range");
    if (e.r != e.c && e.v != 0.0) ++hops;
  }
  const uint64_t per = L >= 2 && N >= 1 ? binomial(L - 2, N - 1) : 0;
  const uint64_t nnz = per * hops;
  QCMG_CHECK_ARG(nnz < (1ull << 32), "half operator too large");
  op.nnz = nnz;
  // slot form: value table +-v per element, at most one hop of a row per element
  const bool slot = slots && op.dim > 0 && op.dim <= 65536u && el.size() <= 1024;
  op.nval = slot ? (int)std::max<size_t>(1, 2 * el.size()) : 0;
  const size_t width = slot ? std::max<size_t>(1, hops) : 0;
  // the tables' places, in doubles
  size_t at = 0;
  auto place = [&](size_t bytes) {
    const size_t here = at;
    at += (bytes + 7) / 8;
    return here;
  };
  const size_t o_val = place(nnz * 8), o_diag = place((size_t)op.dim * 8), o_vtab = place((size_t)op.nval * 8),
               o_el = place(el.size() * sizeof(HopElement)), o_bin = place((size_t)op.dim * 4),
               o_rp = place(((size_t)op.dim + 1) * 4), o_col = place(nnz * 4),
               o_ell = place(width * op.dim * 4), o_len = place(slot ? (size_t)op.dim * 2 : 0);
  op.mem = pool_get(at * 8, &op.mem_got);
  double* m = static_cast<double*>(op.mem);
  op.val.borrow(m + o_val, nnz);
  op.diag.borrow(m + o_diag, op.dim);
  op.bin.borrow(reinterpret_cast<uint32_t*>(m + o_bin), op.dim);
  op.rowptr.borrow(reinterpret_cast<uint32_t*>(m + o_rp), (size_t)op.dim + 1);
  op.col.borrow(reinterpret_cast<uint32_t*>(m + o_col), nnz);
  if (slot) {
    op.vtab = m + o_vtab;
    op.ell = reinterpret_cast<uint32_t*>(m + o_ell);
    op.len = reinterpret_cast<uint16_t*>(m + o_len);
  }
  // value table and elements in one upload (they are neighbours)
  staging.emplace_back(o_bin - o_vtab, 0.0);
  std::vector<double>& h = staging.back();
  if (slot)
    for (size_t k = 0; k < el.size(); ++k) {
      h[2 * k] = el[k].v;
      h[2 * k + 1] = -el[k].v;
    }
  if (!el.empty()) std::memcpy(h.data() + (o_el - o_vtab), el.data(), el.size() * sizeof(HopElement));
  if (!h.empty()) QCMG_CUDA(cudaMemcpyAsync(m + o_vtab, h.data(), h.size() * 8, cudaMemcpyHostToDevice, s));
  const HopElement* d_el = reinterpret_cast<const HopElement*>(m + o_el);
  launch_halfbasis(L, N, op.dim, op.bin.p, s);
  if (op.dim) {
    const unsigned g = grid_for(op.dim, 256);
    k_halfop_count<<<g, 256, 0, s>>>(op.dim, op.bin.p, d_el, (int)el.size(), op.rowptr.p + 1);
    k_rowptr<<<1, 1024, 0, s>>>(op.dim, op.rowptr.p);
    k_halfop_fill<<<g, 256, 0, s>>>(op.dim, op.bin.p, d_el, (int)el.size(), op.rowptr.p, op.col.p,
                                    op.val.p, op.diag.p, op.ell, op.len);
    QCMG_CUDA(cudaGetLastError());
  } else {
    QCMG_CUDA(cudaMemsetAsync(op.rowptr.p, 0, 4, s));
  }
}

// ---------------------------------------------------------------------------
// c / c^dagger on a factorized state (model::create_or_destroy, factorized
// branch, src_ed/model.cpp:160-180; sign from Destroy, src_ed/ED_basis.cpp:79-110).
// One thread per SOURCE state for destruction and per TARGET state for
// creation, so every output element is written by exactly one thread.

__global__ void k_apply_c(int L, int orb, int spin, int pm, int nup, int ndn, uint32_t du,
                          uint32_t dd, uint32_t du2, uint32_t dd2, const double* __restrict__ x,
                          double* __restrict__ y, double z, int accumulate) {
  // Iterate over the TARGET sector: y[t] = z * sign * x[s], where s is the
  // state obtained by removing (creation) or adding (destruction) the electron.
  size_t n2 = (size_t)du2 * dd2;
  uint32_t m = 1u << orb;
  int nup2 = nup + (spin ? 0 : pm), ndn2 = ndn + (spin ? pm : 0);
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n2;
       t += (size_t)gridDim.x * blockDim.x) {
    uint32_t iu2 = (uint32_t)(t % du2), id2 = (uint32_t)(t / du2);
    uint32_t u2 = dev_unrank(iu2, L, nup2), d2 = dev_unrank(id2, L, ndn2);
    double out = 0.0;
    uint32_t occ = spin ? d2 : u2;
    // creation: target must hold the electron; destruction: must not.
    bool ok = (pm > 0) ? ((occ & m) != 0) : ((occ & m) == 0);
    if (ok) {
      uint32_t u = u2, d = d2;
      int par;
      if (!spin) {
        u = u2 ^ m;
        par = __popc(u2 & (m - 1u));
      } else {
        d = d2 ^ m;
        par = __popc(d2 & (m - 1u)) + __popc(u2);
      }
      size_t s = (size_t)dev_rank(u) + (size_t)du * dev_rank(d);
      out = z * ((par & 1) ? -x[s] : x[s]);
    }
    y[t] = accumulate ? y[t] + out : out;
  }
}

void launch_apply_c(int L, int orb, int spin, int pm, int nup, int ndn, const double* x, double* y,
                    double z, bool accumulate, cudaStream_t s) {
  uint32_t du = (uint32_t)binomial(L, nup), dd = (uint32_t)binomial(L, ndn);
  int nup2 = nup + (spin ? 0 : pm), ndn2 = ndn + (spin ? pm : 0);
  uint32_t du2 = (uint32_t)binomial(L, nup2), dd2 = (uint32_t)binomial(L, ndn2);
  size_t n2 = (size_t)du2 * dd2;
  if (!n2) return;
  k_apply_c<<<grid_for(n2, 256), 256, 0, s>>>(L, orb, spin, pm, nup, ndn, du, dd, du2, dd2, x, y,
                                               z, accumulate ? 1 : 0);
  QCMG_CUDA(cudaGetLastError());
}

}  // namespace qcmg
