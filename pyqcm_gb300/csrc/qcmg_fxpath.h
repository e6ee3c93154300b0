// FX64 fast path (fixed-point Krylov vectors): host-side declarations.
#pragma once

#include <cstdint>

#include "qcmg_internal.h"
#include "qcmg_krylov.h"
#include "qcmg_pool.h"

namespace qcmg {

struct I128;

// Scalars of one Lanczos step, written on the device: alpha and the update's
// coefficients by the last block of the product's second pass, the norm by
// the last block of the update.
struct FxStep {
  double alpha;
  long long ma, mb;    // mantissas of alpha c_v / c_w and beta c_p / c_w
  int sw, sa, sb, Eo;  // shifts of the three terms, exponent of the result
  long long n_hi;      // sum of squares >> kDotShift, 128 bits
  unsigned long long n_lo, qmax;
  int err;             // bounded-wait failure flag of the product kernels
  unsigned ticket;     // blocks of the running kernel that are done
  // the host's copy: number of the step whose values stand above
  unsigned long long seq;
};

struct FxReducer {
  DevBuf<I128> part;
  DevBuf<FxStep> step;
  PinnedBuf<FxStep> host;  // written by the device
  unsigned long long seq = 0;  // of the step queued last
  unsigned update_blocks = 0;
  void init(int sms, cudaStream_t s);
};

// Prepares the fixed-point tables; false if the Hamiltonian does not have
// one hop magnitude per spin (then the FP64 path is used).
bool fx_prepare(qcmg_hamiltonian* H);
// (absmax: the largest |x_i| where it is known, else negative and found here
// with a wait for the stream)
void fx_from_f64(const double* x, size_t n, FxVec& v, cudaStream_t s,
                 DevBuf<unsigned long long>& tmp, double absmax = -1.0);
void fx_to_f64(const FxVec& v, double* x, cudaStream_t s);
// With dot set, the product's second pass also computes alpha = <x, y> (for
// the finished y) and the coefficients of y - alpha x - beta p into
// dot->step (p may be null).
void fx_matvec(qcmg_hamiltonian* H, const FxVec& x, FxVec& y, const FxVec* yin, double gamma,
               FxReducer* dot = nullptr, const FxVec* p = nullptr, double beta = 0.0);
// Throws if a kernel of the fast path reported a bounded-wait failure.
void fx_check_error(qcmg_hamiltonian* H);
// Whether a product of FP64 vectors takes the fixed-point passes: where they
// apply, from 2^21 states on.  Below, converting x and y there and back (five
// launches and two host waits) costs more than the FP64 product: 4,900
// states 61 us against 6 us, 853,776 states 88 against 52 us, 2,944,656
// states (13-site chain) 149 against 119 us; the 4x4 sector of 165,636,900
// states ~4.5 ms against 9.95 ms.
inline bool fx_for_f64(qcmg_hamiltonian* H) {
  return H->use_fx && H->dim >= ((size_t)1 << 21) && fx_prepare(H);
}
// y (+)= H x on FP64 device vectors through the fixed-point product.
void fx_matvec_f64(qcmg_hamiltonian* H, const double* x, double* y, bool accumulate,
                   double absmax = -1.0);
// y (+)= H x with x on the device and y in page-locked host memory, written
// through its device-side address yh (zero copy); product_done (optional) is
// recorded between the product and the pass into y.  With m > 0, the old
// values of y's first m elements are read from ypre on the device (a
// prefetched copy, complete once ypre_ready fires) instead of host memory.
void fx_matvec_to_host(qcmg_hamiltonian* H, const double* x, double* yh, bool accumulate,
                       cudaEvent_t product_done = nullptr, const double* ypre = nullptr,
                       size_t m = 0, cudaEvent_t ypre_ready = nullptr);
LanczosResult fx_lanczos(qcmg_hamiltonian* H, const double* x0_dev, double tol, int max_iter,
                         double* psi_dev);

}  // namespace qcmg
