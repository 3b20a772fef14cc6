// Multilevel preconditioner of the scalar elliptic solves (mg.cu).
#pragma once
#include "grmp_internal.h"

// spmv_config reported by a solve that the multilevel preconditioner ran
// (plus the row-loop code of its SpMV, e.g. 90404)
constexpr int kMgConfig = 90000;

// Whether grmp_solve takes the multilevel solver for this matrix (scalar
// H1P1 / H1P2 with a diffusion term, not reaction dominated); builds or
// refreshes what it needs.  *use = 0: the Jacobi solvers.  *checked: the
// diagonal has been found positive and finite (the Jacobi solvers need not look again).
// bicg: for grmp_mg_bicgstab, which pays from fewer rows.
int grmp_mg_prepare(grmp_matrix A, bool mixed, int *use, bool *checked, bool bicg = false);
// Conjugate gradients with the hierarchy where the matrix takes them, mixed
// ones that fail once more in FP64.  *done = false: not taken or not converged
// (maxiter, no progress, breakdown); the Jacobi solvers go on with *p, from x
// if it is nearer than the caller's start, else from that.
int grmp_mg_cg(grmp_matrix A, const double *b, double *x, grmp_solve_params *p, grmp_solve_stats *st, bool *done,
               bool *checked);
// BiCGStab with the prepared FP64 hierarchy for the scalar Jacobian of a Newton
// step; vec: nine vectors of the matrix's rows.  *done = false: it did not
// converge and x is as it was.
int grmp_mg_bicgstab(grmp_matrix A, const double *b, double *x, const grmp_solve_params *p, double *const vec[9],
                     double *partial, void *state, grmp_solve_stats *st, bool *done);
// Whether a hierarchy with numeric storage of this precision exists.
bool grmp_mg_ready(grmp_matrix A, bool mixed);
void grmp_mg_free(grmp_matrix A);
