// Factorized Hubbard matrix-vector product, FP64:
//   y[iu + du*id] (+)= sum_J T_up[iu,J] x[J + du*id]      (up hops, in-slab)
//                   + sum_J T_dn[id,J] x[iu + du*J]      (down hops, slab axpys)
//                   + (d_up[iu] + d_dn[id] + W(u, d)) x[iu + du*id]
// The vector is stored as the reference stores it (src_ed/ED_basis.cpp:142-165):
// column-major du x dd, the up index fastest, one contiguous "slab" per down
// index.  One CTA owns one slab at a time: it stages x's slab in shared
// memory (all up-hop gathers then hit shared memory), streams the down-hop
// neighbour slabs from global memory with coalesced loads (they are shared
// by up to ~2*bonds CTAs and mostly hit L2), and writes its y slab once.
// This is the arithmetic of HS_factorized_operator::multiply_add
// (src_ed/Operators/HS_factorized_operator.hpp:57-84) and
// HS_interaction_operator::multiply_add (HS_interaction_operator.hpp:62-70),
// reorganized per output element so that y is read and written once.  Half
// bases of at most 65,536 states take k_matvec_ell below; k_matvec_f64 is the
// form without their slot tables.
#include "qcmg_internal.h"

namespace qcmg {

template <int INTER, bool SMEM>
__global__ void __launch_bounds__(512)
k_matvec_f64(uint32_t du, uint32_t dd, int L,
             const uint32_t* __restrict__ rp_up, const uint32_t* __restrict__ col_up,
             const double* __restrict__ val_up, const double* __restrict__ diag_up,
             const uint32_t* __restrict__ rp_dn, const uint32_t* __restrict__ col_dn,
             const double* __restrict__ val_dn, const double* __restrict__ diag_dn,
             const uint32_t* __restrict__ bin_up, const uint32_t* __restrict__ bin_dn, double U,
             const double* __restrict__ wdn, const double* __restrict__ x, double* __restrict__ y,
             int accumulate, const int* skip) {
  if (skip && *(volatile const int*)skip >= 0) return;
  extern __shared__ double xs[];
  for (uint32_t a = blockIdx.x; a < dd; a += gridDim.x) {
    const double* xa = x + (size_t)a * du;
    if (SMEM) {
      __syncthreads();
      for (uint32_t i = threadIdx.x; i < du; i += blockDim.x) xs[i] = xa[i];
      __syncthreads();
    }
    const double* xr = SMEM ? xs : xa;
    const uint32_t k0 = rp_dn[a], k1 = rp_dn[a + 1];
    const double dda = diag_dn[a];
    const uint32_t dbits = bin_dn[a];
    double* ya = y + (size_t)a * du;
    for (uint32_t i = threadIdx.x; i < du; i += blockDim.x) {
      double acc = 0.0;
      const uint32_t j0 = rp_up[i], j1 = rp_up[i + 1];
      for (uint32_t k = j0; k < j1; ++k) acc = fma(val_up[k], xr[col_up[k]], acc);
      for (uint32_t k = k0; k < k1; ++k) acc = fma(val_dn[k], x[(size_t)col_dn[k] * du + i], acc);
      double d = diag_up[i] + dda;
      if (INTER == QCMG_INTER_ONSITE) {
        d += U * (double)__popc(bin_up[i] & dbits);
      } else if (INTER == QCMG_INTER_GENERAL) {
        uint32_t u = bin_up[i];
        const double* w = wdn + (size_t)a * L;
        while (u) {
          d += w[__ffs(u) - 1];
          u &= u - 1;
        }
      }
      double out = fma(d, xr[i], acc);
      if (accumulate) out += ya[i];
      ya[i] = out;
    }
  }
}

// The product from the slot form of the up hops.  A CTA takes part of a slab
// (the whole slab staged in shared memory, rows [part) of it computed).
//
// GB300's FP64 pipe (two FMAs per SM and cycle) is the floor: ~31 hops per
// state on the 3x4 cluster with t', 16 of them up. The CSR's row-by-row reads
// cost more than that: neighbouring rows lie 190 bytes apart, so each of a
// warp's loads took 32 L1 wavefronts; the slot form reads one 4-byte word per
// hop, coalesced, and the hop's value from a small table. U popc comes from a
// table too (a conversion to FP64 is an FP64 instruction).
// 853,776 states: 72.8 us -> 59.5 us (floor 50 us); the 4x4 sector of
// 165,636,900 states: 15.3 ms -> 9.95 ms.
constexpr int kMaxVals = 2048;

template <int INTER>
__global__ void __launch_bounds__(512)
k_matvec_ell(uint32_t du, uint32_t dd, int L, int parts, const uint32_t* __restrict__ ell,
             const uint16_t* __restrict__ len, const double* __restrict__ vtab, int nval,
             const double* __restrict__ diag_up, const uint32_t* __restrict__ rp_dn,
             const uint32_t* __restrict__ col_dn, const double* __restrict__ val_dn,
             const double* __restrict__ diag_dn, const uint32_t* __restrict__ bin_up,
             const uint32_t* __restrict__ bin_dn, double U, const double* __restrict__ wdn,
             const double* __restrict__ x, double* __restrict__ y, int accumulate,
             const int* skip) {
  if (skip && *(volatile const int*)skip >= 0) return;
  extern __shared__ double xs[];  // du, then the value table, then U popc
  double* vt = xs + du;
  double* ut = vt + nval;
  const uint32_t a = blockIdx.x / parts, part = blockIdx.x - a * parts;
  const uint32_t rows = (du + parts - 1) / parts;
  const uint32_t i0 = part * rows, i1 = min(du, i0 + rows);
  const double* xa = x + (size_t)a * du;
  for (uint32_t i = threadIdx.x; i < du; i += blockDim.x) xs[i] = xa[i];
  for (int i = threadIdx.x; i < nval; i += blockDim.x) vt[i] = vtab[i];
  if (INTER == QCMG_INTER_ONSITE && threadIdx.x <= 32) ut[threadIdx.x] = U * (double)threadIdx.x;
  __syncthreads();
  const uint32_t k0 = rp_dn[a], k1 = rp_dn[a + 1];
  const double dda = diag_dn[a];
  const uint32_t dbits = bin_dn[a];
  double* ya = y + (size_t)a * du;
  for (uint32_t i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
    const int n = len[i];
    double acc = 0.0;
#pragma unroll 4
    for (int k = 0; k < n; ++k) {
      const uint32_t e = __ldg(ell + (size_t)k * du + i);
      acc = fma(vt[e >> 16], xs[e & 0xffffu], acc);
    }
#pragma unroll 4
    for (uint32_t k = k0; k < k1; ++k)
      acc = fma(__ldg(val_dn + k), __ldg(x + (size_t)__ldg(col_dn + k) * du + i), acc);
    double d = diag_up[i] + dda;
    if (INTER == QCMG_INTER_ONSITE) {
      d += ut[__popc(bin_up[i] & dbits)];
    } else if (INTER == QCMG_INTER_GENERAL) {
      uint32_t u = bin_up[i];
      const double* w = wdn + (size_t)a * L;
      while (u) {
        d += w[__ffs(u) - 1];
        u &= u - 1;
      }
    }
    double out = fma(d, xs[i], acc);
    if (accumulate) out += ya[i];
    ya[i] = out;
  }
}

// One launch of the product: a kernel of either form with its grid, handed
// to `launch(kernel, grid, threads, smem, args...)`.
template <int INTER, class Launch>
static void product_launch(qcmg_hamiltonian* H, const double* x, double* y, bool accumulate,
                           const int* skip, Launch&& launch) {
  auto& up = H->up;
  auto& dn = H->dn;
  int sms = 0, max_optin = 0;
  QCMG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, H->device));
  QCMG_CUDA(cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, H->device));
  const size_t slot_smem = ((size_t)H->du + up.nval + 33) * sizeof(double);
  if (up.nval > 0 && up.nval <= kMaxVals && slot_smem <= (size_t)max_optin) {
    // parts of a slab: enough CTAs for several rounds per SM, at least two
    // warps of rows each
    int parts = 1;
    while (parts < 8 && (size_t)H->dd * parts < (size_t)sms * 12 && H->du / (2 * parts) >= 64) parts *= 2;
    const uint32_t rows = (H->du + parts - 1) / parts;
    const int threads = rows >= 512 ? 512 : (rows >= 256 ? 256 : 128);
    QCMG_CHECK_ARG((size_t)H->dd * parts < (1ull << 31), "sector too large for one launch");
    auto kern = k_matvec_ell<INTER>;
    if (slot_smem > 48 * 1024)
      QCMG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, max_optin));
    launch(kern, (unsigned)(H->dd * parts), threads, slot_smem, H->du, H->dd, H->L, parts,
           (const uint32_t*)up.ell, (const uint16_t*)up.len, (const double*)up.vtab, up.nval,
           (const double*)up.diag.p, (const uint32_t*)dn.rowptr.p, (const uint32_t*)dn.col.p,
           (const double*)dn.val.p, (const double*)dn.diag.p, (const uint32_t*)up.bin.p,
           (const uint32_t*)dn.bin.p, H->U, (const double*)H->wdn.p, x, y, accumulate ? 1 : 0, skip);
    return;
  }
  // half bases too large for the slot form: rows from the CSR, the slab in
  // shared memory where it fits
  const size_t smem = (size_t)H->du * sizeof(double);
  const int threads = H->du >= 512 ? 512 : (H->du >= 256 ? 256 : 128);
  const unsigned grid = std::max(1u, (unsigned)std::min<size_t>(H->dd, (size_t)sms * 8));
  const bool in_smem = smem <= (size_t)max_optin;
  auto kern = in_smem ? k_matvec_f64<INTER, true> : k_matvec_f64<INTER, false>;
  if (in_smem && smem > 48 * 1024)
    QCMG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  launch(kern, grid, threads, in_smem ? smem : (size_t)0, H->du, H->dd, H->L,
         (const uint32_t*)up.rowptr.p, (const uint32_t*)up.col.p, (const double*)up.val.p,
         (const double*)up.diag.p, (const uint32_t*)dn.rowptr.p, (const uint32_t*)dn.col.p,
         (const double*)dn.val.p, (const double*)dn.diag.p, (const uint32_t*)up.bin.p,
         (const uint32_t*)dn.bin.p, H->U, (const double*)H->wdn.p, x, y, accumulate ? 1 : 0, skip);
}

template <class Launch>
static void product_any(qcmg_hamiltonian* H, const double* x, double* y, bool accumulate,
                        const int* skip, Launch&& launch) {
  switch (H->inter_kind) {
    case QCMG_INTER_NONE: product_launch<QCMG_INTER_NONE>(H, x, y, accumulate, skip, launch); break;
    case QCMG_INTER_ONSITE: product_launch<QCMG_INTER_ONSITE>(H, x, y, accumulate, skip, launch); break;
    default: product_launch<QCMG_INTER_GENERAL>(H, x, y, accumulate, skip, launch); break;
  }
}

void matvec_node(qcmg_hamiltonian* H, const double* x, double* y, bool accumulate, GraphChain& gc) {
  product_any(H, x, y, accumulate, nullptr, [&](auto kern, unsigned grid, int threads, size_t smem, auto... args) {
    gc.add(kern, dim3(grid), dim3(threads), smem, args...);
  });
}

void matvec(qcmg_hamiltonian* H, const double* x, double* y, bool accumulate, const int* skip) {
  if (H->dim == 0) return;
  product_any(H, x, y, accumulate, skip, [&](auto kern, unsigned grid, int threads, size_t smem, auto... args) {
    kern<<<grid, threads, smem, H->stream>>>(args...);
    QCMG_CUDA(cudaGetLastError());
  });
}

}  // namespace qcmg
