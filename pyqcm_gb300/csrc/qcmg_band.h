// Band-Lanczos steps with their coefficients on the device (qcmg_band.cu).
#pragma once

#include <cmath>
#include <vector>

#include "qcmg_internal.h"

namespace qcmg {

constexpr int kBandMax = 16;  // start vectors

struct BandRun {
  int M = 0;  // steps taken: the result's size, or the step whose vector deflated
  double ev_old = 1e12, last_change = INFINITY;  // state of the convergence probe
};

// Runs the band recurrence of band_lanczos (qcmg_krylov.cu) from p start
// vectors phi (device memory) for at most M0 steps on the handle's stream,
// with the vectors v_k in ring[k % (2 p + 1)]; fills the projected matrix t
// (M0 x M0, column-major) and the start vectors' projections P (p x M0).
// True: converged or M0 steps done. False: the norm of v_M fell below
// acc_defl; rows up to M - 1 are filled and the ring holds v_{M-p} .. v_{M-1}
// (normalized) and v_M .. v_{M+p-1} (not yet).
bool band_steps(qcmg_hamiltonian* H, int p, const double* phi, int M0, double acc_defl,
                double acc_band, const std::vector<double*>& ring, std::vector<double>& t,
                std::vector<double>& P, BandRun& run);

}  // namespace qcmg
