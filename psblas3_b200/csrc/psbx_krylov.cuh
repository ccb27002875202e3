// psbx_krylov.cuh -- solver state shared by the Krylov drivers
// (psbx_krylov.cu: a kernel per step) and the one-kernel solver of small
// systems (psbx_persist.cu).
#pragma once

#include "psbx_internal.cuh"

// ST_XUPD: a GMRES cycle ended (converged or nl steps); x is updated next.
enum { ST_RUN = 0, ST_DONE = 1, ST_BREAK = 2, ST_XUPD = 3 };

struct KState {
  double rho, rho_old, sigma, alpha, beta, omega, tau;
  double bn2, bni, ani, r0n2;
  double errnum, errden, eps;
  double gamma, delta, theta1, theta2;  // FCG
  double scal;                          // GMRES: scale of the next basis vector
  int itmax, istop;
  int it, itx;
  int status;
  int r0set;
  int first;                            // FCG: first step after a restart
  int gm_m, gm_conv;                    // GMRES: basis vectors in the x update; converged
};

// One-kernel CG / BiCGSTAB (psbx_persist.cu).  persist_fits: whether the
// system is in its range; persist_solve: runs the solve and fills opt like
// the drivers, or leaves *ran 0 with nothing done (itmax beyond its range, rows
// that would keep one block busy while the others wait, or a device that cannot
// hold the kernel's blocks at once).
bool persist_fits(const HllView &A, bool bicg);
bool persist_fits(const EllView &A, bool bicg);
bool persist_fits(const CsrView &A, bool bicg);
int persist_solve(const HllView &A, bool bicg, const double *dinv, const double *b, double *x,
                  psbx_SolverOptions *opt, int *ran);
int persist_solve(const EllView &A, bool bicg, const double *dinv, const double *b, double *x,
                  psbx_SolverOptions *opt, int *ran);
int persist_solve(const CsrView &A, bool bicg, const double *dinv, const double *b, double *x,
                  psbx_SolverOptions *opt, int *ran);
