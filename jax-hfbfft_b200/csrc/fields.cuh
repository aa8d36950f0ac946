// Derivative fields of the densities (skyrme.cu), shared with the energies.
#pragma once
#include "hfb_ctx.cuh"

namespace hfb {

// Per isospin, kNDeriv fields of n^3 doubles:
//   [0] div J   [1] lap rho   [2..4] grad rho   [5..7] curl s
//   [8..10] curl j   [11] div j
// With ``mean_field`` false only div J, lap rho and curl j are formed.
constexpr int kNDeriv = 12;
int density_derivatives(hfb_ctx_s* c, const double* rho, const double* cur, const double* sd, const double* so,
                        bool mean_field, double** dv_out, cudaStream_t st);

}  // namespace hfb
