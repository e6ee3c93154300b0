// FX64 fast path: the factorized product and the Lanczos recurrence on
// fixed-point vectors (see qcmg_fx.cuh for the number format).
//
// Product y (+)= H x in two passes over the sector, stored like the
// reference's vector (up index fastest, one contiguous slab per down state):
//   pass U  one CTA per slab: the slab of x is staged in shared memory and
//           every up-spin hop is an integer gather-add from it; the
//           diagonal (one-body diagonal + density-density terms) and the
//           accumulated input are added; the slab of y is written once.
//   pass D  row bands: the CTAs sweep the down states of one band of rows at
//           a time, so the band of x (~48 MB) stays L2-resident while every
//           down-spin hop adds a neighbour slab segment.
// Both passes read 8 B and write 8 B per state from HBM; the hop gathers hit
// shared memory and L2.  Hop values must share one magnitude per spin
// (the Hubbard form: hops are +-t); other Hamiltonians use the FP64 path.
#include <algorithm>
#include <chrono>
#include <cfloat>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <vector>

#include "qcmg_fx.cuh"
#include "qcmg_tma.cuh"
#include "qcmg_fxpath.h"
#include "qcmg_fxprod.h"
#include "qcmg_internal.h"
#include "qcmg_tridiag.h"

namespace qcmg {

// ---------------------------------------------------------------------------
// host helpers

// x = m * 2^e with |m| < 2^53 (m = 0 for x = 0).
static void split_double(double x, int64_t* m, int* e) {
  if (x == 0.0 || !std::isfinite(x)) {
    *m = 0;
    *e = 0;
    return;
  }
  int ex;
  double f = std::frexp(x, &ex);  // x = f 2^ex, 0.5 <= |f| < 1
  *m = (int64_t)std::llround(std::ldexp(f, 53));
  *e = ex - 53;
}

static int ceil_log2(double x) {
  if (x <= 0.0) return 0;
  int ex;
  double f = std::frexp(x, &ex);  // x = f 2^ex
  return (f == 0.5) ? ex - 1 : ex;
}

static int bitlen(uint64_t v) {
  int n = 0;
  while (v) {
    ++n;
    v >>= 1;
  }
  return n;
}

static unsigned grid_ew(size_t n, int per_sm = 8) {
  size_t g = (n + 255) / 256;
  g = std::max<size_t>(1, std::min<size_t>(g, (size_t)152 * per_sm));
  return (unsigned)g;
}

// ---------------------------------------------------------------------------
// device kernels: conversions and reductions

__global__ void k_absmax_f64(const double* __restrict__ x, size_t n,
                             unsigned long long* __restrict__ out) {
  unsigned long long m = 0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    unsigned long long b = (unsigned long long)__double_as_longlong(x[i]) & 0x7fffffffffffffffull;
    m = max(m, b);
  }
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

__global__ void k_f64_to_fx(const double* __restrict__ x, int64_t* __restrict__ q, size_t n,
                            int E) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    q[i] = f64_to_fx(x[i], E);
}

__global__ void k_fx_to_f64(const int64_t* __restrict__ q, double* __restrict__ x, size_t n,
                            int E, double c) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    x[i] = c * fx_to_f64(q[i], E);
}

// y (+)= c q 2^E straight into the caller's page-locked host vector (zero
// copy).  Elements below m take their old value from ypre, a device copy
// prefetched while the product ran, and are only written (one link
// direction); the others are read and written in host memory (both
// directions at once).  V2: y is 16-byte aligned and m even, two elements
// per access.
template <bool V2>
__global__ void k_fx_to_host(const int64_t* __restrict__ q, double* __restrict__ yh,
                             const double* __restrict__ ypre, size_t m, size_t n, int E, double c,
                             int acc) {
  const size_t step = (size_t)gridDim.x * blockDim.x;
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (V2) {
    double2* y2 = reinterpret_cast<double2*>(yh);
    const double2* p2 = reinterpret_cast<const double2*>(ypre);
    for (; i < n / 2; i += step) {
      double2 v = make_double2(c * fx_to_f64(q[2 * i], E), c * fx_to_f64(q[2 * i + 1], E));
      if (acc) {
        const double2 o = 2 * i < m ? p2[i] : y2[i];
        v.x += o.x;
        v.y += o.y;
      }
      y2[i] = v;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0 && (n & 1)) {
      const double v = c * fx_to_f64(q[n - 1], E);
      yh[n - 1] = acc ? (n - 1 < m ? ypre[n - 1] : yh[n - 1]) + v : v;
    }
  } else {
    for (; i < n; i += step) {
      const double v = c * fx_to_f64(q[i], E);
      yh[i] = acc ? (i < m ? ypre[i] : yh[i]) + v : v;
    }
  }
}

// Fused Lanczos update:
//   q_o = round(q_w * 2^-sw) - round(q_v * ma 2^-sa) - round(q_p * mb 2^-sb)
// written over q_w, with exact |q_o|^2 and max|q_o|.  The block that finishes
// last adds the partials and writes the step's scalars straight into the
// host's page-locked copy, seq after everything else: the host polls it and
// queues the next product while this kernel retires.
template <int MINB>
__global__ void __launch_bounds__(256, MINB) k_fx_update(int64_t* __restrict__ w,
                                                   const int64_t* __restrict__ v,
                                                   const int64_t* __restrict__ p, size_t n,
                                                   FxStep* __restrict__ st,
                                                   I128* __restrict__ part,
                                                   const int* __restrict__ err,
                                                   FxStep* host, unsigned long long seq) {
  const int sw = st->sw, sa = st->sa, sb = st->sb;
  const int64_t ma = st->ma, mb = st->mb;
  I128 s = {0, 0};
  unsigned long long m = 0;
  auto one = [&](int64_t wi, int64_t vi, int64_t pi) {
    int64_t o = shr_round(wi, sw);
    if (ma) o -= mul_fix(vi, ma, sa);
    if (p && mb) o -= mul_fix(pi, mb, sb);
    s = add128(s, shr128(mul_s64(o, o), kDotShift));
    m = max(m, (unsigned long long)(o < 0 ? -o : o));
    return o;
  };
  // two elements per 16-byte load (cudaMalloc'd vectors: even indices are
  // 16-byte aligned); w, v and p are each read once and streamed
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const size_t n2 = n / 2;
  longlong2* w2 = reinterpret_cast<longlong2*>(w);
  const longlong2* v2 = reinterpret_cast<const longlong2*>(v);
  const longlong2* p2 = reinterpret_cast<const longlong2*>(p);
#pragma unroll 2
  for (size_t j = blockIdx.x * (size_t)blockDim.x + threadIdx.x; j < n2; j += stride) {
    const longlong2 wv = __ldcs(w2 + j), vv = __ldcs(v2 + j);
    const longlong2 pv = p ? __ldcs(p2 + j) : make_longlong2(0, 0);
    longlong2 o;
    o.x = one(wv.x, vv.x, pv.x);
    o.y = one(wv.y, vv.y, pv.y);
    __stcs(w2 + j, o);
  }
  if ((n & 1) && blockIdx.x == 0 && threadIdx.x == 0)
    w[n - 1] = one(w[n - 1], v[n - 1], p ? p[n - 1] : 0);
  // one atomic per block (one per warp queue up at the single address)
  __shared__ unsigned long long bmax[8];
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) bmax[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < 8; ++k) m = max(m, bmax[k]);
    atomicMax(&st->qmax, m);
  }
  I128 h;
  if (!last_block_sum128(s, part, &st->ticket, &h) || threadIdx.x != 0) return;
  volatile FxStep* out = host;
  out->alpha = st->alpha;
  out->Eo = st->Eo;
  out->n_hi = h.hi;
  out->n_lo = h.lo;
  out->qmax = __ldcg(&st->qmax);
  out->err = err ? *err : 0;
  __threadfence_system();
  out->seq = seq;
}

// g = round(g * 2^-sg) + round(q * m 2^-s)   (eigenvector accumulation)
__global__ void k_fx_axpy(int64_t* __restrict__ g, const int64_t* __restrict__ q, size_t n, int sg,
                          int64_t m, int s) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    g[i] = shr_round(g[i], sg) + mul_fix(q[i], m, s);
}

// ---------------------------------------------------------------------------
// ---------------------------------------------------------------------------
// tables

static void build_unit_csr(const HalfOp& op, cudaStream_t s, DevBuf<uint32_t>& rp,
                           DevBuf<uint32_t>& rs, DevBuf<uint32_t>& col, double* tmag,
                           int* maxdeg, bool* ok) {
  std::vector<uint32_t> hrp(op.dim + 1), hcol(op.nnz);
  std::vector<double> hval(op.nnz);
  if (op.dim) QCMG_CUDA(cudaMemcpyAsync(hrp.data(), op.rowptr.p, (op.dim + 1) * 4, cudaMemcpyDeviceToHost, s));
  if (op.nnz) {
    QCMG_CUDA(cudaMemcpyAsync(hcol.data(), op.col.p, op.nnz * 4, cudaMemcpyDeviceToHost, s));
    QCMG_CUDA(cudaMemcpyAsync(hval.data(), op.val.p, op.nnz * 8, cudaMemcpyDeviceToHost, s));
  }
  QCMG_CUDA(cudaStreamSynchronize(s));
  double t = 0.0;
  for (double v : hval) {
    if (t == 0.0) t = std::fabs(v);
    if (std::fabs(v) != t) {
      *ok = false;
      return;
    }
  }
  *tmag = t;
  std::vector<uint32_t> nrp(op.dim + 1), nrs(std::max<uint32_t>(op.dim, 1)), ncol(op.nnz);
  int md = 0;
  for (uint32_t i = 0; i < op.dim; ++i) {
    uint32_t pos = hrp[i];
    nrp[i] = pos;
    for (uint32_t k = hrp[i]; k < hrp[i + 1]; ++k)
      if (hval[k] > 0) ncol[pos++] = hcol[k];
    nrs[i] = pos;
    for (uint32_t k = hrp[i]; k < hrp[i + 1]; ++k)
      if (hval[k] < 0) ncol[pos++] = hcol[k];
    md = std::max<int>(md, (int)(hrp[i + 1] - hrp[i]));
  }
  nrp[op.dim] = hrp[op.dim];
  *maxdeg = md;
  rp.upload(nrp.data(), op.dim + 1, s);
  rs.upload(nrs.data(), nrs.size(), s);
  if (op.nnz)
    col.upload(ncol.data(), op.nnz, s);
  else
    col.alloc(1);
  QCMG_CUDA(cudaStreamSynchronize(s));  // host staging vectors go out of scope
}

__global__ void k_diag_to_fx(const double* __restrict__ d, int64_t* __restrict__ out, size_t n,
                             double scale) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    out[i] = (int64_t)llrint(d[i] * scale);  // set-up only
}

bool fx_prepare(qcmg_hamiltonian* H) {
  FxTables& T = H->fx;
  if (T.state != 0) return T.state > 0;
  T.state = -1;
  if (H->dim == 0 || H->du >= (1u << 31) || H->dd >= (1u << 31)) return false;
  int max_optin = 0;
  QCMG_CUDA(cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, H->device));
  if ((size_t)H->du * 8 > (size_t)max_optin) return false;  // slab must fit in shared memory
  cudaStream_t s = H->stream;
  bool ok = true;
  build_unit_csr(H->up, s, T.rp_up, T.rs_up, T.col_up, &T.t_up, &T.maxdeg_up, &ok);
  if (!ok) return false;
  build_unit_csr(H->dn, s, T.rp_dn, T.rs_dn, T.col_dn, &T.t_dn, &T.maxdeg_dn, &ok);
  if (!ok) return false;
  // pass U with bulk-copied slabs: grouped ELL table and slabs per round
  T.ns = choose_slabs_per_pass(H->du, max_optin);
  if (T.ns > 0 && !build_ell4(T.rp_up, T.rs_up, T.col_up, H->du, s, T.ell4, T.cnt4)) T.ns = 0;
  T.err.alloc(1);
  QCMG_CUDA(cudaMemsetAsync(T.err.p, 0, sizeof(int), s));
  // diagonal bound and fixed-point scale 2^-G
  std::vector<double> hdu(H->du), hdd(H->dd), hw;
  QCMG_CUDA(cudaMemcpyAsync(hdu.data(), H->up.diag.p, H->du * 8, cudaMemcpyDeviceToHost, s));
  QCMG_CUDA(cudaMemcpyAsync(hdd.data(), H->dn.diag.p, H->dd * 8, cudaMemcpyDeviceToHost, s));
  if (H->inter_kind == QCMG_INTER_GENERAL) {
    hw.resize((size_t)H->dd * H->L);
    QCMG_CUDA(cudaMemcpyAsync(hw.data(), H->wdn.p, hw.size() * 8, cudaMemcpyDeviceToHost, s));
  }
  QCMG_CUDA(cudaStreamSynchronize(s));
  double mu = 0.0, md = 0.0, mw = 0.0;
  for (double v : hdu) mu = std::max(mu, std::fabs(v));
  for (double v : hdd) md = std::max(md, std::fabs(v));
  if (H->inter_kind == QCMG_INTER_ONSITE) mw = std::fabs(H->U) * H->L;
  if (H->inter_kind == QCMG_INTER_GENERAL)
    for (uint32_t i = 0; i < H->dd; ++i) {
      double s2 = 0.0;
      for (int r = 0; r < H->L; ++r) s2 += std::fabs(hw[(size_t)i * H->L + r]);
      mw = std::max(mw, s2);
    }
  const double dmax = mu + md + mw;
  T.G = 61 - ceil_log2(std::max(dmax, 1.0));
  const double scale = std::ldexp(1.0, T.G);
  T.dup.alloc(H->du);
  T.ddn.alloc(H->dd);
  k_diag_to_fx<<<grid_ew(H->du), 256, 0, s>>>(H->up.diag.p, T.dup.p, H->du, scale);
  k_diag_to_fx<<<grid_ew(H->dd), 256, 0, s>>>(H->dn.diag.p, T.ddn.p, H->dd, scale);
  T.U = (int64_t)std::llrint(H->U * scale);
  if (H->inter_kind == QCMG_INTER_GENERAL) {
    T.wdn.alloc(hw.size());
    k_diag_to_fx<<<grid_ew(hw.size()), 256, 0, s>>>(H->wdn.p, T.wdn.p, hw.size(), scale);
  }
  QCMG_CUDA(cudaGetLastError());
  // Narrow diagonal: when every diagonal entry at scale 2^-G is a multiple of
  // 2^tz and |D| >> tz stays below 2^6 (small-integer energies such as the
  // Hubbard model's), x * (D >> tz) fits in 63 bits and the diagonal term is
  // one 64-bit product and a rounding shift, bit-identical to the 128-bit one.
  {
    int tz = 63;
    auto fold = [&](double v) {
      const long long q = std::llrint(v * scale);  // the value k_diag_to_fx stores
      if (q != 0) tz = std::min(tz, __builtin_ctzll((unsigned long long)q));
    };
    for (double v : hdu) fold(v);
    for (double v : hdd) fold(v);
    for (double v : hw) fold(v);
    if (H->inter_kind == QCMG_INTER_ONSITE) fold(H->U);
    const double dbound = std::ceil(dmax * scale);
    T.dtz = (std::ldexp(dbound, -tz) < 64.0) ? tz : -1;
    if (T.dtz >= 0) {
      auto narrow = [&](const std::vector<double>& src, DevBuf<int32_t>& dst) {
        std::vector<int32_t> h(std::max<size_t>(src.size(), 1), 0);
        for (size_t k = 0; k < src.size(); ++k) h[k] = (int32_t)(std::llrint(src[k] * scale) >> T.dtz);
        dst.upload(h.data(), h.size(), s);
      };
      narrow(hdu, T.dup32);
      narrow(hdd, T.ddn32);
      narrow(hw, T.wdn32);
      T.U32 = (int32_t)(std::llrint(H->U * scale) >> T.dtz);
      QCMG_CUDA(cudaStreamSynchronize(s));  // host staging vectors go out of scope
    }
  }
  T.bound = dmax + T.t_up * T.maxdeg_up + T.t_dn * T.maxdeg_dn;
  T.b = ceil_log2(std::max(T.bound, 1.0));
  // Rows per band of pass D: ~48 MB of x per band (QCMG_FX_BAND_MB
  // overrides).  A band of a down state is one warp's work, and a sector
  // that fits in one such band has too few of them (924 warps for 924 x 924
  // states): small sectors take shorter bands, down to one 64-row sweep, so
  // that the items fill the chip's resident warps (48 per SM) twice.  x is
  // L2-resident there whatever the band.  924 x 924, with the dot product:
  // 49.5 us -> 14.3 us (cold).
  double band_mb = 48.0;
  if (const char* v = std::getenv("QCMG_FX_BAND_MB")) band_mb = std::max(1.0, std::atof(v));
  size_t band = (size_t)(band_mb * 1.0e6 / (8.0 * std::max<uint32_t>(H->dd, 1)));
  band = std::max<size_t>(256, (band / 256) * 256);
  const size_t fill = (size_t)H->du * H->dd / ((size_t)2 * 48 * 152) / 64 * 64;
  band = std::min(band, std::max<size_t>(64, fill));
  T.band = (uint32_t)std::min<size_t>(band, H->du);
  T.state = 1;
  return true;
}

// ---------------------------------------------------------------------------
// FX vectors

void FxVec::alloc(size_t count) {
  buf.alloc(count);
  n = count;
}

void fx_from_f64(const double* x, size_t n, FxVec& v, cudaStream_t s, DevBuf<unsigned long long>& tmp,
                 double mx) {
  v.alloc(n);
  if (!(mx >= 0.0)) {
    tmp.alloc(1);
    QCMG_CUDA(cudaMemsetAsync(tmp.p, 0, 8, s));
    k_absmax_f64<<<grid_ew(n), 256, 0, s>>>(x, n, tmp.p);
    unsigned long long hb = 0;
    QCMG_CUDA(cudaMemcpyAsync(&hb, tmp.p, 8, cudaMemcpyDeviceToHost, s));
    QCMG_CUDA(cudaStreamSynchronize(s));
    std::memcpy(&mx, &hb, 8);
  }
  v.c = 1.0;
  if (mx == 0.0) {
    v.E = 0;
    v.mb = 0;
    QCMG_CUDA(cudaMemsetAsync(v.buf.p, 0, n * 8, s));
    return;
  }
  v.E = ceil_log2(mx) - kFxBits;  // |q| <= 2^56
  k_f64_to_fx<<<grid_ew(n), 256, 0, s>>>(x, v.buf.p, n, v.E);
  QCMG_CUDA(cudaGetLastError());
  v.mb = kFxBits;
}

void fx_to_f64(const FxVec& v, double* x, cudaStream_t s) {
  k_fx_to_f64<<<grid_ew(v.n), 256, 0, s>>>(v.buf.p, x, v.n, v.E, v.c);
  QCMG_CUDA(cudaGetLastError());
}

void FxReducer::init(int sms, cudaStream_t s) {
  update_blocks = 32u * (unsigned)sms;
  part.alloc(std::max(update_blocks, product_dot_partials(sms)));
  step.alloc(1);
  QCMG_CUDA(cudaMemsetAsync(step.p, 0, sizeof(FxStep), s));
  host.alloc(1);
  host.p->seq = seq = 0;
}

// ---------------------------------------------------------------------------
// the product

// y = H x  (or y = H x + gamma * yin with yin != nullptr, yin may be &y).
// The output exponent follows from the bound |H|_inf (T.b) and the input's
// largest component; c_y = c_x.
void fx_matvec(qcmg_hamiltonian* H, const FxVec& x, FxVec& y, const FxVec* yin, double gamma,
               FxReducer* dot, const FxVec* p, double beta) {
  FxTables& T = H->fx;
  cudaStream_t s = H->stream;
  const size_t n = H->dim;
  if (y.n != n) y.alloc(n);
  // bound on the output's real magnitude, in units of c_x
  double bound = std::ldexp(T.bound, x.E + x.mb);
  if (yin && yin->mb > 0) bound += std::fabs(gamma * yin->c / x.c) * std::ldexp(1.0, yin->E + yin->mb);
  int Eo = ceil_log2(bound) - kFxBits;
  FxProdArgs A;
  A.du = H->du;
  A.dd = H->dd;
  A.L = H->L;
  A.rp_up = T.rp_up.p;
  A.rs_up = T.rs_up.p;
  A.col_up = T.col_up.p;
  A.rp_dn = T.rp_dn.p;
  A.rs_dn = T.rs_dn.p;
  A.col_dn = T.col_dn.p;
  A.dup = T.dup.p;
  A.ddn = T.ddn.p;
  A.bin_up = H->up.bin.p;
  A.bin_dn = H->dn.bin.p;
  A.U = T.U;
  A.wdn = T.wdn.p;
  int e;
  split_double(T.t_up, &A.mt_up, &e);
  A.sh_up = Eo - x.E - e;
  split_double(T.t_dn, &A.mt_dn, &e);
  A.sh_dn = Eo - x.E - e;
  A.sh_d = Eo - x.E + T.G;
  A.d_tz = T.dtz;
  A.p2_up = pow2_exponent(A.mt_up);
  A.p2_dn = pow2_exponent(A.mt_dn);
  A.yin = nullptr;
  A.m_in = 0;
  A.sh_in = 0;
  A.p2_in = -1;
  if (yin && yin->mb > 0 && gamma != 0.0) {
    A.yin = yin->buf.p;
    split_double(gamma * yin->c / x.c, &A.m_in, &e);
    A.sh_in = Eo - yin->E - e;
    A.p2_in = pow2_exponent(A.m_in);
  }
  // fixed shifts of the FAST kernels (used only when every multiplier is a
  // power of two and the diagonal is narrow)
  auto fixed = [](int t, int* to, int64_t* ro) {
    t = std::min(t, 63);
    *to = t;
    *ro = t > 0 ? (int64_t)(1ull << (t - 1)) : 0;
  };
  fixed(A.sh_up - A.p2_up, &A.t_up, &A.r_up);
  fixed(A.sh_dn - A.p2_dn, &A.t_dn, &A.r_dn);
  fixed(A.sh_d - T.dtz, &A.t_d, &A.r_d);
  fixed(A.sh_in - A.p2_in, &A.t_in, &A.r_in);
  A.neg_in = A.m_in < 0;
  A.dup32 = T.dup32.p;
  A.ddn32 = T.ddn32.p;
  A.wdn32 = T.wdn32.p;
  A.U32 = T.U32;
  A.x = x.buf.p;
  A.y = y.buf.p;
  A.band = T.band;
  A.nbands = (H->du + T.band - 1) / T.band;
  A.ell4 = T.ell4.p;
  A.cnt4 = T.cnt4.p;
  A.err = T.err.p;
  y.E = Eo;
  y.mb = kFxBits;
  y.c = x.c;
  A.dot_x = nullptr;
  A.dot_part = nullptr;
  if (dot) {
    A.dot_x = x.buf.p;
    A.dot_part = dot->part.p;
    A.dot_step = dot->step.p;
    A.dot_xc = x.c;
    A.dot_xE = x.E;
    A.dot_xmb = x.mb;
    A.dot_yc = y.c;
    A.dot_yE = y.E;
    A.dot_ymb = y.mb;
    A.dot_bp = 0.0;
    A.dot_pE = 0;
    int64_t mb = 0;
    if (p) {
      A.dot_bp = std::fabs(beta * p->c / y.c) * std::ldexp(1.0, p->E + p->mb);
      split_double(beta * p->c / y.c, &mb, &e);
      A.dot_pE = e + p->E;
    }
    A.dot_mb = mb;
  }
  launch_product(H, A, s);
}

void fx_check_error(qcmg_hamiltonian* H) {
  int err = 0;
  if (!H->fx.err.p) return;
  QCMG_CUDA(cudaMemcpyAsync(&err, H->fx.err.p, sizeof(int), cudaMemcpyDeviceToHost, H->stream));
  QCMG_CUDA(cudaStreamSynchronize(H->stream));
  if (err) throw Error(QCMG_ERR_CUDA, "a bulk copy into shared memory did not complete in time");
}

void fx_matvec_f64(qcmg_hamiltonian* H, const double* x, double* y, bool accumulate, double absmax) {
  FxTables& T = H->fx;
  cudaStream_t s = H->stream;
  fx_from_f64(x, H->dim, T.x, s, T.tmp, absmax);
  if (accumulate) {
    fx_from_f64(y, H->dim, T.y, s, T.tmp);
    fx_matvec(H, T.x, T.y, &T.y, 1.0);
  } else {
    fx_matvec(H, T.x, T.y, nullptr, 0.0);
  }
  fx_to_f64(T.y, y, s);
}

// y_host (+)= H x for x on the device and y in page-locked host memory (its
// device-side address yh): H x in fixed point, then one pass that converts
// and accumulates into the host vector, the first m elements' old values
// read from ypre (device) once the event ypre_ready has fired.
void fx_matvec_to_host(qcmg_hamiltonian* H, const double* x, double* yh, bool accumulate,
                       cudaEvent_t product_done, const double* ypre, size_t m,
                       cudaEvent_t ypre_ready) {
  FxTables& T = H->fx;
  cudaStream_t s = H->stream;
  const size_t n = H->dim;
  fx_from_f64(x, n, T.x, s, T.tmp);
  fx_matvec(H, T.x, T.y, nullptr, 0.0);
  if (product_done) QCMG_CUDA(cudaEventRecord(product_done, s));
  if (m && ypre_ready) QCMG_CUDA(cudaStreamWaitEvent(s, ypre_ready, 0));
  const unsigned g = 152u * 8u;
  const int acc = accumulate ? 1 : 0;
  if (((uintptr_t)yh & 15u) == 0 && (m % 2) == 0)
    k_fx_to_host<true><<<g, 256, 0, s>>>(T.y.buf.p, yh, ypre, m, n, T.y.E, T.y.c, acc);
  else
    k_fx_to_host<false><<<g, 256, 0, s>>>(T.y.buf.p, yh, ypre, m, n, T.y.E, T.y.c, acc);
  QCMG_CUDA(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// Lanczos on FX vectors: the reference's recurrence (Lanczos.hpp:64-93)
// written with normalized vectors, w = H v_j - alpha v_j - beta v_{j-1}.

// Queues w <- w - alpha v - beta p with the coefficients that the product
// left in red.step.
static void fx_update(qcmg_hamiltonian* H, FxVec& w, const FxVec& v, const FxVec* p, FxReducer& red) {
  const size_t n = w.n;
  // Up to one pair of elements per thread of the large grid, the latency of
  // the few rounds counts: four resident blocks per SM (64 registers), one
  // round (853,776 states: 11.4 ms a solve, 13.1 ms with the other form). Above,
  // HBM: three blocks resident and 32 per SM launched, for an even last
  // round (165,636,900 states: 3.92 ms a step, 4.10 ms with the small form).
  const size_t blocks = std::max<size_t>(1, (n / 2 + 255) / 256);
  auto go = [&](auto kern, unsigned g) {
    kern<<<g, 256, 0, H->stream>>>(w.buf.p, v.buf.p, p ? p->buf.p : nullptr, n, red.step.p, red.part.p,
                                   H->fx.err.p, red.host.p, ++red.seq);
  };
  if (blocks <= red.update_blocks)
    go(k_fx_update<4>, (unsigned)std::min<size_t>(blocks, red.update_blocks / 8));
  else
    go(k_fx_update<3>, red.update_blocks);
  QCMG_CUDA(cudaGetLastError());
}

// Waits for the step queued last: w's exponent and size, alpha and |w|^2.
// The host's copy is polled for as long as a small sector's step takes, where
// the few microseconds of a stream wait count (step 50 us at 853,776 states); a
// longer step is left to the stream wait, which spins, yields or blocks as the
// caller set its device to do (165,636,900 states: 4 ms a step).
constexpr std::chrono::microseconds kPollFor(200);
static void fx_collect(qcmg_hamiltonian* H, FxVec& w, FxReducer& red, double* alpha, double* norm2) {
  const FxStep& h = *red.host.p;
  auto arrived = [&] { return __atomic_load_n(&red.host.p->seq, __ATOMIC_ACQUIRE) == red.seq; };
  const auto start = std::chrono::steady_clock::now();
  for (unsigned spin = 1; !arrived(); ++spin) {
    if (spin % 64 || std::chrono::steady_clock::now() - start < kPollFor) continue;
    QCMG_CUDA(cudaStreamSynchronize(H->stream));
    if (arrived()) break;
    throw Error(QCMG_ERR_CUDA, "a Lanczos step did not report its scalars");
  }
  if (h.err) throw Error(QCMG_ERR_CUDA, "a bulk copy into shared memory did not complete in time");
  w.E = h.Eo;
  w.mb = bitlen(h.qmax);
  *alpha = h.alpha;
  const double r = std::ldexp((double)h.n_hi, 64) + (double)h.n_lo;
  *norm2 = w.c * w.c * std::ldexp(r, kDotShift + 2 * h.Eo);
}

// One stored vector's term of the ground state.
struct FxTerm {
  const int64_t* q;
  int64_t m;
  int s;
};

// psi_i = 2^E sum_k round(q_k,i m_k 2^-s_k): the integer sum that adding the
// terms one by one gives, in any order.  Every vector is read once.
__global__ void __launch_bounds__(256) k_fx_combine(const FxTerm* __restrict__ t, int nt, size_t n,
                                                    int E, double* __restrict__ psi) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  int64_t g = 0;
#pragma unroll 8
  for (int k = 0; k < nt; ++k) g += mul_fix(__ldcs(t[k].q + i), t[k].m, t[k].s);
  psi[i] = fx_to_f64(g, E);
}

// Device memory for the Lanczos vectors of one solve: slots of n elements,
// 256-byte aligned, allocated many at a time.  get() returns null when the
// next allocation would take more than a quarter of the memory that was free
// at the start, or fails.
struct FxSlots {
  std::deque<DevBuf<int64_t>> blocks;
  size_t stride = 0, left = 0, budget = 0;
  int64_t* next = nullptr;
  explicit FxSlots(size_t n) : stride((n + 31) & ~(size_t)31) {}
  void measure() {
    size_t fr = 0, total = 0;
    QCMG_CUDA(cudaMemGetInfo(&fr, &total));
    budget = std::max(fr / 4, 3 * stride * 8);
  }
  bool room_for(size_t cnt) const { return cnt <= budget / (stride * 8); }
  int64_t* get(size_t want) {
    if (left == 0) {
      const size_t bytes = stride * 8;
      const size_t cnt = std::max<size_t>(std::min(want, ((size_t)1 << 30) / bytes), blocks.empty() ? 3 : 1);
      if (cnt * bytes > budget) return nullptr;
      blocks.emplace_back();
      try {
        blocks.back().alloc(cnt * stride);
      } catch (const Error& e) {
        if (e.code != QCMG_ERR_NOMEM || blocks.size() == 1) throw;
        cudaGetLastError();
        return nullptr;
      }
      budget -= cnt * bytes;
      left = cnt;
      next = blocks.back().p;
    }
    int64_t* r = next;
    next += stride;
    --left;
    return r;
  }
};

LanczosResult fx_lanczos(qcmg_hamiltonian* H, const double* x0_dev, double tol, int max_iter,
                         double* psi_dev) {
  LanczosResult res;
  cudaStream_t s = H->stream;
  const size_t n = H->dim;
  FxReducer red;
  int sms = 0;
  QCMG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, H->device));
  red.init(sms, s);
  DevBuf<unsigned long long> tmp;
  FxSlots slots(n);
  // The Lanczos vectors are kept when the ground state is wanted and 300 of
  // them (a solve takes 80 to 250) fit in a quarter of the free memory: psi
  // is then one pass over them instead of a second run of the recurrence
  // (3x4 cluster, 220 steps: a product and an update per step against 1.5 GB
  // read once).
  slots.measure();
  bool keep = psi_dev != nullptr && slots.room_for((size_t)std::min(max_iter + 2, 300));
  const size_t want = keep ? 64 : 3;
  FxVec x0, vbuf[3];
  vbuf[0].buf.borrow(slots.get(want), n);
  for (FxVec& b : vbuf) b.n = n;
  x0.buf.borrow(vbuf[0].buf.p, n);
  x0.n = n;
  fx_from_f64(x0_dev, n, x0, s, tmp);
  struct Kept {
    const int64_t* q;
    int E;
    double c;
  };
  // a step queued in vain (or before an error) is over before its buffers go
  Drain drain{s};
  std::vector<Kept> kept;
  TridiagLowest lowest;
  std::vector<double> z;
  // the recurrence; replay: on the recorded coefficients, accumulating gs
  auto run = [&](bool replay, FxVec* gs) {
    FxVec* v = &vbuf[0];
    FxVec* p = &vbuf[1];
    FxVec* w = &vbuf[2];
    if (replay) fx_from_f64(x0_dev, n, *v, s, tmp);
    v->E = x0.E;
    v->mb = x0.mb;
    v->c = x0.c;
    bool have_p = false;
    double beta_prev = 0.0;
    const int nsteps = replay ? (int)z.size() : max_iter + 1;
    auto queue = [&](int j) {  // w <- H v - alpha v - beta p
      if (!replay && keep) {
        kept.push_back({v->buf.p, v->E, v->c});
        int64_t* q = slots.get(want);
        if (!q) {  // no room for more: a replay will follow
          keep = false;
          q = const_cast<int64_t*>(kept[0].q);  // neither v nor p: j >= 2 here
        }
        w->buf.borrow(q, n);
      } else if (!replay && j < 2) {
        w->buf.borrow(slots.get(want), n);
      }
      // alpha = <v, H v> comes out of the product's second pass
      fx_matvec(H, *v, *w, nullptr, 0.0, &red, have_p ? p : nullptr, beta_prev);
      fx_update(H, *w, *v, have_p ? p : nullptr, red);
    };
    // On sectors whose step takes tens of microseconds the convergence test
    // takes as long: the next step is queued first and runs meanwhile (one
    // step is computed in vain).
    const bool ahead = !replay && n < ((size_t)4 << 20);
    if (!replay) queue(0);
    for (int j = 0; j < nsteps; ++j) {
      if (replay) {
        // gs += z_j v_j
        int64_t m;
        int e;
        split_double(z[j] * v->c, &m, &e);
        k_fx_axpy<<<grid_ew(n), 256, 0, s>>>(gs->buf.p, v->buf.p, n, 0, m, gs->E - v->E - e);
        QCMG_CUDA(cudaGetLastError());
        if (j + 1 == nsteps) break;
        queue(j);
      }
      double a = 0.0, n2 = 0.0;
      fx_collect(H, *w, red, &a, &n2);
      const double b = replay ? res.beta[j] : std::sqrt(n2);
      auto converged = [&] {
        res.energy = lowest(res.alpha, res.beta, z);
        double ritz = std::fabs(z.back() * b);
        if (!std::isfinite(res.energy) || !std::isfinite(ritz))
          throw Error(QCMG_ERR_NUMERIC, "Lanczos produced a non-finite value");
        if (ritz <= tol || b == 0.0) return true;
        if ((int)res.alpha.size() > max_iter)
          throw Error(QCMG_ERR_NOCONV,
                      "Lanczos procedure exceeded " + std::to_string(max_iter) + " iterations");
        return false;
      };
      bool early = false;
      if (!replay) {
        res.alpha.push_back(a);
        res.beta.push_back(b);
        early = ahead && j + 1 < nsteps && std::isfinite(a) && std::isfinite(b) && b > 0.0;
        if (!early && converged()) break;
      }
      // rotate: p <- v, v <- w / beta, w <- old p.  The division only changes
      // the lazy scale; its power of two moves into the exponent (exact), so
      // c stays in [0.5, 1) and neither c nor 2^E drifts out of double range
      // over hundreds of iterations.
      int k2 = 0;
      w->c = std::frexp(w->c / b, &k2);
      w->E += k2;
      FxVec* t = p;
      p = v;
      v = w;
      w = t;
      have_p = true;
      beta_prev = b;
      if (!replay && j + 1 < nsteps) queue(j + 1);
      if (early && converged()) break;
    }
  };
  run(false, nullptr);
  res.niter = (int)res.alpha.size();
  if (!psi_dev) return res;
  double bnd = 0.0;
  for (double zj : z) bnd += std::fabs(zj);
  const int gE = ceil_log2(bnd) - kFxBits;  // |psi_i| <= sum_j |z_j| |v_j|_max <= sum |z_j|
  if (keep) {
    std::vector<FxTerm> t(z.size());
    for (size_t j = 0; j < z.size(); ++j) {
      int e;
      split_double(z[j] * kept[j].c, &t[j].m, &e);
      t[j].q = kept[j].q;
      t[j].s = gE - kept[j].E - e;
    }
    DevBuf<FxTerm> dt;
    dt.upload(t.data(), t.size(), s);
    k_fx_combine<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(dt.p, (int)t.size(), n, gE, psi_dev);
    QCMG_CUDA(cudaGetLastError());
    QCMG_CUDA(cudaStreamSynchronize(s));
    return res;
  }
  FxVec gs;
  gs.alloc(n);
  QCMG_CUDA(cudaMemsetAsync(gs.buf.p, 0, n * 8, s));
  gs.E = gE;
  gs.c = 1.0;
  gs.mb = kFxBits;
  run(true, &gs);
  fx_to_f64(gs, psi_dev, s);
  QCMG_CUDA(cudaStreamSynchronize(s));
  return res;
}

}  // namespace qcmg
