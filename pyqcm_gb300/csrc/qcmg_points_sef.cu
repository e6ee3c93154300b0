// Point kernels of the Potthoff functional for L = 1..16 (a translation unit of
// their own: the kernels are unrolled, and compile in parallel).
#include "qcmg_points.cuh"

namespace qcmg {

void launch_sef_points(int L, const LuArgs& A, cudaStream_t s) {
  if (A.nk > 0 && A.nw > 0) launch_lu<false, kMaxPointL>(L, A, s);
}

}  // namespace qcmg
