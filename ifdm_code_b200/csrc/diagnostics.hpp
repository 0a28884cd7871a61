// diagnostics.hpp -- device diagnostics of the wave function (diagnostics.cu).
#pragma once

#include "step_engine.hpp"

#include <cuda_runtime.h>

#include <string>

namespace ifdm {

constexpr int kMaxBins = 64;

// Doubles of workspace the calls below need for an N-box.
size_t diag_work_doubles(int N);

// P(k) of delta = |psi|^2 / <|psi|^2> - 1 of the box in nbins bins of |kappa|
// (kappa the integer wave vector, k = 2 pi kappa / L, L the box side): bin b
// holds edges[b] <= |kappa| < edges[b+1]; edges null: log-spaced from 1 to N/2.
// field: room for N^3 complex128 on the device; work: diag_work_doubles(N);
// S: psi's unit.  k_out: mean k of each bin's modes; pk_out: <|delta_k|^2> L^3 /
// N^6; modes_out: modes per bin; mean_rho: <|psi|^2>.  Any output may be null.
std::string power_spectrum(const EngineView &v, double S, double2 *field, double *work, double L, int nbins,
                           const double *edges, double *k_out, double *pk_out, long long *modes_out, double *mean_rho,
                           cudaStream_t s);

// Means over the grid of |psi|^2, |grad psi|^2 (spectral derivative, k = pi
// kappa / xmax with kappa per axis in -N/2 .. N/2-1, xmax the half box), phi
// |psi|^2 and |psi|^4: out[0..3].  field, work, S as above.
std::string field_means(const EngineView &v, double S, double2 *field, double *work, double xmax, double out[4],
                        cudaStream_t s);

}  // namespace ifdm
