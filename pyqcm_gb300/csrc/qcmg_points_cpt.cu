// Point kernels of the periodized Green function for L = 1..16 (a translation unit of
// their own: the kernels are unrolled, and compile in parallel).
#include "qcmg_points.cuh"

namespace qcmg {

void launch_cpt_points(int L, const LuArgs& A, cudaStream_t s) {
  if (A.nk > 0 && A.nw > 0) launch_lu<true, kMaxPointL>(L, A, s);
}

}  // namespace qcmg
