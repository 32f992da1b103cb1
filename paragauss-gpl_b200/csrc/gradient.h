// gradient.h -- post-SCF XC nuclear gradient on the device.
//
// dE_xc/dR_A of E_xc = sum_g w_g f(rho(r_g), gamma(r_g)) with the grid
// attached to the atoms (r_g = R_host + fixed offset) and w_g = w_raw(g)
// W_host(r_g), the Becke weight of the host atom: the derivative of the
// discrete energy the build integrates, as the reference's post-SCF
// gradients with moving grid and weight gradients (post_scf_module.f90
// :2930-3060, density_calc_ph_nl, grid_module.f90 becke1).
//
// With X^s = Phi P^s and Y^s_j = d_j Phi P^s (per tile of points, its listed functions),
//   q^s_mu,k(g) = 2 [a_s d_k phi_mu X^s_mu + sum_j b_sj (d_k d_j phi_mu X^s_mu + d_k phi_mu Y^s_j,mu)],
// a_s = w df/drho_s and b_s = w (2 df/dgamma_ss grad rho_s + df/dgamma_ab grad rho_s'), the
// orbital terms are  -sum_g q_mu(g) to atom(mu)  and  +sum_mu q_mu(g) to host(g);
// the weight term is sum_g w_raw f dW_host(r_g)/dR.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "kernels.h"

namespace pgxc {

struct ScreenPlan;

// [slot][128] planes of a chunk: phi, grad phi, (GGAs) Hessian, and the products
int64_t grad_planes(bool gga, bool mgga, int ispin);

// One gradient's buffers and kind.
struct GradOrbitals;
struct TileLists;
struct GradChunk {
  bool gga, mgga;            // meta-GGAs set both
  int ispin, functional, natm;
  const double* P[2];        // density matrices, leading dimension BuildArgs::ldc
  const GradOrbitals* orb[2]; // not null: the orbitals instead
  const int* fatom;          // atom of each function
  const TileLists* lists;    // room for the lists of any chunk
  double* rows;              // grad_planes planes of `plane` doubles
  int64_t plane;
  int64_t ld;                // points of the largest chunk
  double* den;               // 7 ispin ld: rho, grad rho, 2 tau_j
  double* coef;              // 5 ispin ld: a, b, c
  double* ef;                // w_raw f of every point of the plan
  double* exc;               // sum w f is added
  double* grad;              // the orbital terms are added
};
// The orbital terms of chunk c of the plan (grad_plan_create): -sum_g q to atom(mu)
// and +sum_mu q to host(g); also ef and E_xc.
void launch_grad_chunk(const GradChunk& g, const BuildArgs& a, ScreenPlan* sp, size_t c, cudaStream_t st);

// The weight term sum_g ef_g dW_host(r_g)/dR over the chunk's points; dist is
// the natm x natm atom distance matrix followed by its reciprocals (the
// table of launch_becke); scratch holds 3.5 natm ld doubles.
void launch_grad_weights(const double* atoms, const double* dist, int natm, const double* px, const double* py,
                         const double* pz, const int* owner, int64_t p0, int64_t nvalid, int64_t ld, const double* ef,
                         double* scratch, double* grad, cudaStream_t st);

}  // namespace pgxc
