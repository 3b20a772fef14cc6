// Multilevel hierarchy of a scalar elliptic matrix: the patterns (host side).
#pragma once
#include <cstdint>
#include <vector>

struct MgCsr {
    std::vector<int32_t> rp, ci;   // rows, ascending columns
};

// One coarsening step from a level of n rows to nc: the prolongation P, its
// transpose R, the product A P (also the pattern of the smoothed
// prolongation Q), its transpose, and the next level's matrix P^T A P.
// perm arrays give, for each entry of a transpose, its position in the
// original.
struct MgStep {
    int n = 0, nc = 0;
    bool geometric = false;              // P2 -> P1 interpolation, else smoothed aggregation
    bool lump = false;                   // rows of P lack aggregates that they couple to (their values go to the row's own)
    std::vector<int32_t> agg;            // aggregate of each row (smoothed aggregation)
    MgCsr P, R, AP, QT, Ac;
    std::vector<int32_t> Rperm, QTperm;
};

struct MgSymbolic {
    std::vector<MgStep> step;            // step[0]: fine level
};

constexpr int kMgBottom = 96;            // rows of a level that is solved densely
constexpr int kMgMaxLevels = 14;

constexpr double kMgProlong = 1.32;      // w of the prolongation smoothing, P = (I - w D A) P_agg

// The cells of the matrix's space: cell DoFs [ncells][ld] (dim + 1 vertices,
// then, P2, edges) and the mesh.
struct MgCells {
    int dim = 0, ncells = 0, ld = 0;
    const int32_t *celldofs = nullptr, *cells = nullptr;
    const double *coords = nullptr;
};

// Builds the steps of a matrix with pattern A (n rows).  p2: of a P2 space, the
// first step then interpolates from the vertices.  cell_terms: the matrix has
// terms on cells only (face terms couple vertices that have no stiffness in
// common: nothing is left out then).  stretched: every step aggregates, along
// strong couplings.  m is read for p2 or stretched only.  fine_q: the
// transpose of Q also for step 0.  Returns 0, or 1 when the matrix does not coarsen.
int mg_symbolic_build(int n, const MgCsr &A, const MgCells &m, bool p2, bool cell_terms, bool stretched, bool fine_q,
                      MgSymbolic *S);
