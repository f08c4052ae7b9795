// Internal interface of the tensor-core per-k kernels (dm_mma.cu), any nb <= 72.
#pragma once

#include "common.cuh"
#include "dm.cuh"

namespace cpphf {

// One line-search trial: U(tau) to U (a full field), diag(U^H Ft U) to ew; a
// launch after the accepted trial returns at once.
int dm_mma_trial(const double2* dQ, const double2* Ft, const double* p, const double* d_p, const double* w, double* ew,
                 double2* U, int64_t nk, int nb, double T_r, double shrink, int last_trial, double fallback,
                 DmScalars* S, cudaStream_t st);
// Q <- Q U(tau_final): U of the accepted trial as dm_mma_trial left it; for the
// fallback step U and ew are formed here.
int dm_mma_retract(double2* Q, const double2* dQ, const double2* Ft, double* ew, const double2* U, int64_t nk, int nb,
                   const DmScalars* S, cudaStream_t st);
// P = herm(Q diag(p) Q^H), p = e, or with mu p = expit((mu - e) / T), stored to p_out
int dm_mma_density(const double2* Q, const double* e, const double* mu, double T, double* p_out, double2* P, int64_t nk,
                   int nb, cudaStream_t st);
// F <- Q^H F Q with eps, the gradient G, g_p and S->grad_norm, S->lam_pc
int dm_mma_rot_grad(const double2* Q, double2* F, const double* p, const double* w, double* eps, double2* G, double* g_p,
                    int64_t nk, int nb, double T_r, double denom_scale, DmScalars* S, cudaStream_t st);
// SCF density and commutator residuals of Hermitian F, D (S->grad_norm, S->lam_pc)
int scf_mma_residuals(const double2* F, const double2* D, const double2* Pn, const double* w, int64_t nk, int nb,
                      DmScalars* S, double2* comm_out, cudaStream_t st);

}  // namespace cpphf
