// Multilevel preconditioner of the scalar elliptic solves (mg.cu).
#pragma once
#include "grmp_internal.h"

// spmv_config reported by a solve that the multilevel preconditioner ran
// (plus the row-loop code of its SpMV, e.g. 90404)
constexpr int kMgConfig = 90000;

// Conjugate gradients with the hierarchy where the matrix takes them, mixed
// ones that fail once more in FP64.  *done = false: not taken or not converged
// (maxiter, no progress, breakdown); the Jacobi solvers go on with *p, from x
// if it is nearer than the caller's start, else from that.  *checked: the
// diagonal has been found positive and finite (the Jacobi solvers need not look
// again).  present: with what there is already, nothing is allocated.
int grmp_mg_cg(grmp_matrix A, const double *b, double *x, grmp_solve_params *p, grmp_solve_stats *st, bool *done,
               bool *checked, bool present = false);
// BiCGStab with the FP64 hierarchy for the scalar Jacobian of a Newton step;
// vec: nine vectors of the matrix's rows.  *done = false: not taken or not
// converged, x is as it was.
int grmp_mg_bicgstab(grmp_matrix A, const double *b, double *x, const grmp_solve_params *p, double *const vec[9],
                     double *partial, void *state, grmp_solve_stats *st, bool *done, bool *checked);
void grmp_mg_free(grmp_matrix A);
// Frees the context's hierarchies until `bytes` more fit (all of them where that
// cannot be told).  They are made again when there is room; one that has been
// freed three times only when there is room for the last such request as well
// (a program that allocates and frees between solves would pay the analysis
// at every solve).  False: there was none.
bool grmp_mg_reclaim(grmp_context ctx, size_t bytes);
