// Lanczos on sectors small enough to live in the shared memory of one
// thread-block cluster (qcmg_chip.cu).
#pragma once

#include <vector>

#include "qcmg_internal.h"

namespace qcmg {

// Whether the sector takes the on-chip recurrence.
bool chip_fits(const qcmg_hamiltonian* H);

struct ChipResult {
  std::vector<double> alpha, beta, z;
  double energy = 0.0;
  int niter = 0;
  int status = QCMG_OK;  // or QCMG_ERR_NUMERIC, QCMG_ERR_NOCONV
};

// Ground states of n sectors that fit, from their start vectors x0 (device
// memory), with the stopping rule of LanczosEigenvalue (pyqcm
// src_ed/Hamiltonian/Lanczos.hpp:64-93) tested after every step; psi (may be
// null, entries may be null) receives the ground-state vectors in host
// memory.  All handles on one device, locked by the caller.  Several host
// threads share the sectors; each launches on a stream of its own.
void chip_lanczos(int n, qcmg_hamiltonian* const* Hs, const double* const* x0, double tol,
                  int max_iter, double* const* psi, ChipResult* res);

// Whether the band Lanczos of p start vectors runs on chip.
bool chip_band_fits(const qcmg_hamiltonian* H, int p);

// Band Lanczos steps on chip from p start vectors phi (device memory), at most
// M0 of them, on the handle's stream: fills the projected matrix t (M0 x M0,
// column-major) and the start vectors' projections P (p x M0) as
// band_lanczos does and sets *M to the steps taken. False when a vector
// deflates (or a coefficient is not finite): the general path then decides.
bool chip_band(qcmg_hamiltonian* H, int p, const double* phi, int M0, double acc_defl,
               double acc_band, std::vector<double>& t, std::vector<double>& P, int* M);

}  // namespace qcmg
