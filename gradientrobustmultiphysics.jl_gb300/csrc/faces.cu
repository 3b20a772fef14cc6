// Interior-face (ON_IFACES) terms with discontinuous operators: the gradient
// jump [grad u] = grad u|T1 - grad u|T2 across each interior face
// (Jump(Gradient), update_dii4op!, src/assemblypatterns.jl:103-153).
//
//   * BilinearForm([Jump(Gradient), Jump(Gradient)], Action(input |F|^p);
//     AT = ON_IFACES, factor tau): tau |F| |F|^p sum_q w_q [grad phi_i].[grad phi_j],
//     the interior-penalty stabilisation of
//     examples/Example203_ReactionConvectionDiffusion2D.jl:89-92;
//   * ItemIntegrator([Jump(Gradient)], ...; AT = ON_IFACES): per-face
//     integrals of |[grad u]|^2 or ([grad u].n_F)^2 times |F|^p, the jump part
//     of the error estimator of examples/Example210_PoissonLshapeAdaptive2D.jl:58-75.
//
// A face couples the DoFs of its two cells, so a matrix with face terms holds
// the DoFs of the face neighbours of each row's cells (pattern.cu).  Values
// come face by face into face matrices and are added row by row (deterministic,
// no atomics).  Quadrature points
// of a face are placed by barycentric weights over the face's vertices in
// ascending global vertex order, so both cells see the same points.
#include "element.cuh"
#include "grmp_internal.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

namespace {

constexpr int TPB = 256;
inline int nblk(long long n, int tpb = TPB) { return (int)((n + tpb - 1) / tpb); }

// ------------------------------------------------------------------ adjacency
__global__ void k_face_count(long long n, int nf, const int32_t *cell_faces, int32_t *cnt, int32_t *fc) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int F = cell_faces[i];
    const int slot = atomicAdd(&cnt[F], 1);
    if (slot < 2) fc[2 * (size_t)F + slot] = (int32_t)(i / nf);
}

// lower cell id first, -1 for the missing neighbour of a boundary face
__global__ void k_face_order(int32_t nfaces, const int32_t *cnt, int32_t *fc, int *bad) {
    const int F = blockIdx.x * blockDim.x + threadIdx.x;
    if (F >= nfaces) return;
    const int n = cnt[F];
    if (n < 1 || n > 2) {
        atomicExch(bad, 1);
        fc[2 * (size_t)F] = fc[2 * (size_t)F + 1] = -1;
        return;
    }
    if (n == 1) {
        fc[2 * (size_t)F + 1] = -1;
        return;
    }
    const int a = fc[2 * (size_t)F], b = fc[2 * (size_t)F + 1];
    fc[2 * (size_t)F] = min(a, b);
    fc[2 * (size_t)F + 1] = max(a, b);
}

__global__ void k_cell_nbr(long long n, int nf, const int32_t *cell_faces, const int32_t *fc, int32_t *nbr) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int F = cell_faces[i], c = (int)(i / nf);
    const int a = fc[2 * (size_t)F], b = fc[2 * (size_t)F + 1];
    nbr[i] = b < 0 ? -1 : (a == c ? b : a);
}

// ------------------------------------------------------------------ element evaluation
// local vertices of the faces of a simplex (the mesh module's local face
// numbering: triangles [0,1], [1,2], [2,0]; tetrahedra [0,1,2], [0,1,3],
// [1,2,3], [0,2,3])
__device__ __forceinline__ int face_vertex(int dim, int f, int k) {
    if (dim == 2) return (f + k) % 3;
    const int t[4][3] = {{0, 1, 2}, {0, 1, 3}, {1, 2, 3}, {0, 2, 3}};
    return t[f][k];
}

// the face's vertices in ascending global vertex order, as local vertices of the cell
template <int DIM>
__device__ __forceinline__ void face_canon(const int32_t *cells, int cell, int f, int loc[DIM]) {
    int gid[DIM];
    for (int k = 0; k < DIM; k++) {
        loc[k] = face_vertex(DIM, f, k);
        gid[k] = cells[(size_t)cell * (DIM + 1) + loc[k]];
    }
    for (int i = 1; i < DIM; i++)
        for (int j = i; j > 0 && gid[j] < gid[j - 1]; j--) {
            int t = gid[j]; gid[j] = gid[j - 1]; gid[j - 1] = t;
            t = loc[j]; loc[j] = loc[j - 1]; loc[j - 1] = t;
        }
}

// end points of the P2 edge functions (h1_p2.jl:134-165)
template <int DIM>
__device__ __forceinline__ int edge_vertex(int e, int k) {
    if (DIM == 2) return (e + k) % 3;
    const int t[6][2] = {{0, 1}, {0, 2}, {0, 3}, {1, 2}, {1, 3}, {2, 3}};
    return t[e][k];
}

// gradient of local basis function a at barycentric coordinates lam from the
// gradients gl of those: grad lam_a (P1); (4 lam_a - 1) grad lam_a at the
// vertices and 4 (lam_i grad lam_j + lam_j grad lam_i) on the edges (P2)
template <int DIM, int NB>
__device__ __forceinline__ void basis_grad(int a, const double lam[DIM + 1], const double gl[DIM + 1][DIM], double g[DIM]) {
    if (a <= DIM) {
        const double c = NB == DIM + 1 ? 1.0 : 4.0 * lam[a] - 1.0;
#pragma unroll
        for (int k = 0; k < DIM; k++) g[k] = __dmul_rn(c, gl[a][k]);
    } else {
        const int i = edge_vertex<DIM>(a - DIM - 1, 0), j = edge_vertex<DIM>(a - DIM - 1, 1);
        const double ci = 4.0 * lam[i], cj = 4.0 * lam[j];
#pragma unroll
        for (int k = 0; k < DIM; k++) g[k] = fma(ci, gl[j][k], __dmul_rn(cj, gl[i][k]));
    }
}

// barycentric coordinates in the cell of the point with weights w over the face's canonical vertices
template <int DIM>
__device__ __forceinline__ void face_point(const double *w, const int loc[DIM], double lam[DIM + 1]) {
#pragma unroll
    for (int v = 0; v <= DIM; v++) {
        lam[v] = 0.0;
#pragma unroll
        for (int k = 0; k < DIM; k++) lam[v] = loc[k] == v ? w[k] : lam[v];
    }
}

template <int DIM>
__device__ __forceinline__ void cell_grad(const double *coords, const int32_t *cells, int c, double g[DIM + 1][DIM]) {
    double X[(DIM + 1) * DIM], A[3][3], G[3][3], vol;
#pragma unroll
    for (int v = 0; v <= DIM; v++)
#pragma unroll
        for (int k = 0; k < DIM; k++) X[v * DIM + k] = coords[(size_t)cells[(size_t)c * (DIM + 1) + v] * DIM + k];
    simplex_geometry_rn<DIM>(X, A, G, vol);
#pragma unroll
    for (int k = 0; k < DIM; k++) {
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < DIM; j++) {
            g[j + 1][k] = G[k][j];
            s -= G[k][j];
        }
        g[0][k] = s;
    }
}

// gradients of the barycentric coordinates of every cell, [cell][vertex][k]:
// once per cell instead of once per face and side (nine or four FP64 divisions)
template <int DIM>
__global__ void k_cell_grads(int ncells, const double *coords, const int32_t *cells, double *gl) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncells) return;
    double g[DIM + 1][DIM];
    cell_grad<DIM>(coords, cells, c, g);
#pragma unroll
    for (int v = 0; v <= DIM; v++)
#pragma unroll
        for (int k = 0; k < DIM; k++) gl[((size_t)c * (DIM + 1) + v) * DIM + k] = g[v][k];
}

// (where memory is short there is no table, gl == nullptr, and they are computed here)
template <int DIM>
__device__ __forceinline__ void load_grads(const double *gl, const double *coords, const int32_t *cells, int c,
                                           double g[DIM + 1][DIM]) {
    if (!gl) {
        cell_grad<DIM>(coords, cells, c, g);
        return;
    }
#pragma unroll
    for (int v = 0; v <= DIM; v++)
#pragma unroll
        for (int k = 0; k < DIM; k++) g[v][k] = gl[((size_t)c * (DIM + 1) + v) * DIM + k];
}

template <int DIM>
__device__ __forceinline__ int face_in_cell(const int32_t *cell_faces, int c, int F) {
    int f = 0;
    for (int g = 0; g <= DIM; g++)
        if (cell_faces[(size_t)c * (DIM + 1) + g] == F) f = g;
    return f;
}

__device__ __forceinline__ double power_of(double x, double p) {
    const int k = (int)p;
    if ((double)k == p && k >= 0 && k <= 8) {
        double r = 1.0;
        for (int i = 0; i < k; i++) r *= x;
        return r;
    }
    return pow(x, p);
}

struct FaceRule {
    int nq;
    double lam[32][3];   // barycentric weights over the face's canonical vertices
    double w[32];        // weights (sum 1 over the face)
};

struct FaceTermDev {
    double factor, power;
};

// ------------------------------------------------------------------ face bilinear terms
// one point's contribution to an entry of a face's matrix from the jumps of two
// functions (explicit fma: both kernels that form entries round alike)
template <int DIM>
__device__ __forceinline__ double face_point_entry(const double a[DIM], const double b[DIM], double w, double s) {
    double d = 0.0;
#pragma unroll
    for (int k = 0; k < DIM; k++) d = fma(a[k], b[k], d);
    return fma(w, d, s);
}

// adds v to the entry of column col in the row [r0, r1)
__device__ __forceinline__ void add_entry(int r0, int r1, const int32_t *cols, int32_t col, double v, double *v64,
                                          float *v32, int *missing) {
    int lo = r0, hi = r1;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (cols[mid] < col) lo = mid + 1;
        else hi = mid;
    }
    if (lo >= r1 || cols[lo] != col) {
        atomicExch(missing, 1);
        return;
    }
    v64[lo] += v;
    if (v32) v32[lo] += (float)v;
}

struct FaceGeom {
    const int32_t *cell_faces, *cells, *celldofs;
    const double *coords, *gl, *fvol;
};

// Face matrices, then rows.  k_face_mats: a block takes fb faces; a thread per
// (face, point) puts the jump of every function of the two cells into shared
// memory, then a thread per entry i <= j of a face's matrix sums over the
// points and writes both halves.  The functions are numbered: the lower cell's,
// then those of the upper cell that the lower one lacks (fcol: their DoFs,
// fn: their number).  k_face_add: LPR lanes per row, a lane per column, walk
// the row's cells in ascending order and their interior faces (a face that two
// cells of the row share comes from the lower one) and add the row of the
// face's matrix: within a chunk of faces (kFaceBytes) the same order of
// additions as adding face by face in one thread, no atomics.  The chunks depend
// on the mesh alone, so the bits do too.
//
// Bound by FP64 issue in k_face_mats (45 entries x 2 points x 3 operations a
// face for P2 triangles) and by the face matrices' write and read (63 MB for
// 96,840 faces).  A thread per row that evaluated the jumps of both cells again
// for every (row, face) took 1.58 ms on 129,600 P2 rows; now 134 + 111 us.
template <int DIM, int NB>
__global__ void __launch_bounds__(128) k_face_mats(int F0, int nf, int fb, const int32_t *face_cells,
                                                   const int32_t *cell_faces, const int32_t *cells, const double *coords,
                                                   const int32_t *celldofs, const double *gl, const double *fvol,
                                                   FaceTermDev t, FaceRule r, double *mats, int32_t *fcol, int32_t *fn) {
    constexpr int NC = 2 * NB;
    extern __shared__ __align__(16) unsigned char fsm[];
    double *J = reinterpret_cast<double *>(fsm);                      // [fb][nq][NC][DIM]
    double *sc = J + (size_t)fb * r.nq * NC * DIM;                    // [fb]
    int *num = reinterpret_cast<int *>(sc + fb), *map = num + fb;     // [fb], [fb][NB] column of the upper cell's function
    const int base = blockIdx.x * fb, cnt = min(fb, nf - base);
    __shared__ int nmax;
    if (threadIdx.x == 0) nmax = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
        const int F = F0 + base + i, c1 = face_cells[2 * (size_t)F], c2 = face_cells[2 * (size_t)F + 1];
        int n = 0;
        if (c1 >= 0 && c2 >= 0) {
            int32_t d1[NB];
            int32_t *col = fcol + (size_t)(base + i) * NC;
            n = NB;
#pragma unroll
            for (int b = 0; b < NB; b++) col[b] = d1[b] = celldofs[(size_t)c1 * NB + b];
            for (int b = 0; b < NB; b++) {
                const int32_t d = celldofs[(size_t)c2 * NB + b];
                int m = -1;
#pragma unroll
                for (int e = 0; e < NB; e++)
                    if (d1[e] == d) m = e;
                if (m < 0) {
                    m = n++;
                    col[m] = d;
                }
                map[i * NB + b] = m;
            }
            const double fv = fvol[F];
            sc[i] = t.factor * fv * power_of(fv, t.power);
        }
        num[i] = n;
        fn[base + i] = n;
        atomicMax(&nmax, n);
    }
    __syncthreads();
    for (int w = threadIdx.x; w < cnt * r.nq; w += blockDim.x) {
        const int i = w / r.nq, q = w - i * r.nq;
        if (!num[i]) continue;
        const int F = F0 + base + i;
        double *Jq = J + (size_t)w * NC * DIM;
#pragma unroll 1
        for (int side = 0; side < 2; side++) {
            const int c = face_cells[2 * (size_t)F + side];
            int loc[DIM];
            double lam[DIM + 1], g[DIM + 1][DIM];
            face_canon<DIM>(cells, c, face_in_cell<DIM>(cell_faces, c, F), loc);
            face_point<DIM>(r.lam[q], loc, lam);
            load_grads<DIM>(gl, coords, cells, c, g);
#pragma unroll
            for (int b = 0; b < NB; b++) {
                double d[DIM];
                basis_grad<DIM, NB>(b, lam, g, d);
                const int m = side ? map[i * NB + b] : b;
#pragma unroll
                for (int k = 0; k < DIM; k++) {
                    if (!side) Jq[m * DIM + k] = d[k];
                    else Jq[m * DIM + k] = m < NB ? Jq[m * DIM + k] - d[k] : -d[k];
                }
            }
        }
    }
    __syncthreads();
    const int NP = max(1, nmax * (nmax + 1) / 2);
    for (int w = threadIdx.x; w < cnt * NP; w += blockDim.x) {
        const int i = w / NP, e = w - i * NP, n = num[i];
        // entry e of the lower triangle, row by row
        int a = (int)((sqrtf(8.0f * (float)e + 1.0f) - 1.0f) * 0.5f);
        if ((a + 1) * (a + 2) / 2 <= e) a++;
        if (a * (a + 1) / 2 > e) a--;
        const int b = e - a * (a + 1) / 2;
        if (a >= n) continue;
        const double *Ja = J + (size_t)i * r.nq * NC * DIM + a * DIM, *Jb = Ja + (b - a) * DIM;
        double s = 0.0;
        for (int q = 0; q < r.nq; q++, Ja += NC * DIM, Jb += NC * DIM) {
            double a_[DIM], b_[DIM];
#pragma unroll
            for (int k = 0; k < DIM; k++) a_[k] = Ja[k], b_[k] = Jb[k];
            s = face_point_entry<DIM>(a_, b_, r.w[q], s);
        }
        s *= sc[i];
        double *M = mats + (size_t)(base + i) * NC * NC;
        M[a * n + b] = s;
        M[b * n + a] = s;
    }
}

template <int DIM, int NB, int LPR>
__global__ void __launch_bounds__(128) k_face_add(int32_t nrows, int F0, int nf, const int32_t *inc_ptr,
                                                  const int32_t *inc_cell, const int32_t *cell_faces,
                                                  const int32_t *nbr, const double *mats, const int32_t *fcol,
                                                  const int32_t *fn, const int32_t *rowptr, const int32_t *cols,
                                                  double *v64, float *v32, int *missing) {
    constexpr int NC = 2 * NB, NF = DIM + 1;
    static_assert(NC <= LPR, "a lane per column");
    const long long g = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / LPR;
    const int lane = threadIdx.x & 31, sub = lane & (LPR - 1), first = lane & ~(LPR - 1);
    const unsigned mask = (LPR == 32 ? 0xffffffffu : ((1u << LPR) - 1u) << first);
    if (g >= nrows) return;
    const int row = (int)g, r0 = rowptr[row], r1 = rowptr[row + 1];
    for (int p = inc_ptr[row]; p < inc_ptr[row + 1]; p++) {
        const int c = inc_cell[p];
        for (int f = 0; f < NF; f++) {
            const int c2 = nbr[(size_t)c * NF + f];
            if (c2 < 0) continue;
            const int i = cell_faces[(size_t)c * NF + f] - F0;
            if (i < 0 || i >= nf) continue;
            const int n = fn[i];
            const int32_t col = sub < n ? fcol[(size_t)i * NC + sub] : -1;
            const unsigned own = __ballot_sync(mask, col == row);
            const int a = __ffs(own >> first) - 1;
            if (c2 < c && a < NB) continue;   // taken from the lower of the row's two cells
            if (col >= 0) add_entry(r0, r1, cols, col, mats[(size_t)i * NC * NC + a * n + sub], v64, v32, missing);
            __syncwarp(mask);   // the next face may meet the same entries from other lanes
        }
    }
}

// The same without face matrices, where there is no memory for them: a thread
// per row takes the row's faces in the same order and forms every entry as
// k_face_mats does, bit for bit.  129,600 P2 rows: assembly 1.4 ms (0.32 with matrices).
template <int DIM, int NB>
__global__ void __launch_bounds__(128) k_face_rows(int32_t nrows, int F0, int nf, const int32_t *inc_ptr,
                                                   const int32_t *inc_cell, const int32_t *nbr, const int32_t *rowptr,
                                                   const int32_t *cols, double *v64, float *v32, int *missing, FaceGeom m,
                                                   FaceTermDev t, FaceRule r) {
    constexpr int NF = DIM + 1, NC = 2 * NB;
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= nrows) return;
    const int r0 = rowptr[row], r1 = rowptr[row + 1];
    for (int p = inc_ptr[row]; p < inc_ptr[row + 1]; p++) {
        const int c = inc_cell[p];
        for (int f = 0; f < NF; f++) {
            const int o = nbr[(size_t)c * NF + f];
            if (o < 0) continue;
            const int F = m.cell_faces[(size_t)c * NF + f];
            if (F < F0 || F >= F0 + nf) continue;
            const int c1 = min(c, o), c2 = max(c, o);
            // the functions as k_face_mats numbers them, and the row's own
            int32_t col[NC];
            int map[NB], n = NB, a = -1;
            for (int b = 0; b < NB; b++) {
                col[b] = m.celldofs[(size_t)c1 * NB + b];
                if (col[b] == row) a = b;
            }
            if (o < c && a >= 0) continue;   // taken from the lower of the row's two cells
            for (int b = 0; b < NB; b++) {
                const int32_t d = m.celldofs[(size_t)c2 * NB + b];
                int k = -1;
                for (int e = 0; e < NB; e++)
                    if (col[e] == d) k = e;
                if (k < 0) {
                    k = n++;
                    col[k] = d;
                    if (d == row) a = k;
                }
                map[b] = k;
            }
            if (a < 0) continue;   // (the row is a function of its own cell)
            double s[NC];
            for (int e = 0; e < n; e++) s[e] = 0.0;
            for (int q = 0; q < r.nq; q++) {
                double J[NC][DIM];
                for (int side = 0; side < 2; side++) {
                    const int cc = side ? c2 : c1;
                    int loc[DIM];
                    double lam[DIM + 1], g[DIM + 1][DIM];
                    face_canon<DIM>(m.cells, cc, face_in_cell<DIM>(m.cell_faces, cc, F), loc);
                    face_point<DIM>(r.lam[q], loc, lam);
                    load_grads<DIM>(m.gl, m.coords, m.cells, cc, g);
#pragma unroll
                    for (int b = 0; b < NB; b++) {
                        double d[DIM];
                        basis_grad<DIM, NB>(b, lam, g, d);
                        const int e = side ? map[b] : b;
#pragma unroll
                        for (int k = 0; k < DIM; k++) J[e][k] = !side ? d[k] : (e < NB ? J[e][k] - d[k] : -d[k]);
                    }
                }
                for (int e = 0; e < n; e++) s[e] = face_point_entry<DIM>(J[a], J[e], r.w[q], s[e]);
            }
            const double fv = m.fvol[F], sc = t.factor * fv * power_of(fv, t.power);
            for (int e = 0; e < n; e++) add_entry(r0, r1, cols, col[e], __dmul_rn(s[e], sc), v64, v32, missing);
        }
    }
}

// ------------------------------------------------------------------ jump integrator
// coefficients of the barycentric gradients in the gradient of a P1 / P2 function
template <int DIM, int NB>
__device__ __forceinline__ void grad_coefs(const double u[NB], const double lam[DIM + 1], double cf[DIM + 1]) {
#pragma unroll
    for (int v = 0; v <= DIM; v++) cf[v] = NB == DIM + 1 ? u[v] : u[v] * (4.0 * lam[v] - 1.0);
    if constexpr (NB > DIM + 1) {
#pragma unroll
        for (int e = 0; e < NB - DIM - 1; e++) {
            const int i = edge_vertex<DIM>(e, 0), j = edge_vertex<DIM>(e, 1);
            cf[j] += u[DIM + 1 + e] * (4.0 * lam[i]);
            cf[i] += u[DIM + 1 + e] * (4.0 * lam[j]);
        }
    }
}

// A thread per face; grad u = sum_v cf_v grad lam_v on either side.  With the
// derivative of every basis function at every point and the geometry of both
// cells taken per face it was 130 us for 97,200 faces (P2, two points), now
// 38 us; bound by FP64 issue.
template <int DIM, int NB>
__global__ void __launch_bounds__(128) k_face_jumps(int32_t nfaces, const int32_t *face_cells, const int32_t *cell_faces,
                                                    const int32_t *cells, const double *coords, const double *gl,
                                                    const int32_t *celldofs,
                                                    const double *u, const double *fnormals, const double *fvol,
                                                    int kind, double power, double factor, FaceRule r, double *out) {
    const int F = blockIdx.x * blockDim.x + threadIdx.x;
    if (F >= nfaces) return;
    const int c1 = face_cells[2 * (size_t)F], c2 = face_cells[2 * (size_t)F + 1];
    if (c1 < 0 || c2 < 0) {
        out[F] = 0.0;
        return;
    }
    int loc1[DIM], loc2[DIM];
    face_canon<DIM>(cells, c1, face_in_cell<DIM>(cell_faces, c1, F), loc1);
    face_canon<DIM>(cells, c2, face_in_cell<DIM>(cell_faces, c2, F), loc2);
    double g1[DIM + 1][DIM], g2[DIM + 1][DIM], u1[NB], u2[NB];
    load_grads<DIM>(gl, coords, cells, c1, g1);
    load_grads<DIM>(gl, coords, cells, c2, g2);
#pragma unroll
    for (int b = 0; b < NB; b++) {
        u1[b] = u[celldofs[(size_t)c1 * NB + b]];
        u2[b] = u[celldofs[(size_t)c2 * NB + b]];
    }
    double acc = 0.0;
    for (int q = 0; q < r.nq; q++) {
        double lam[DIM + 1], a1[DIM + 1], a2[DIM + 1];
        face_point<DIM>(r.lam[q], loc1, lam);
        grad_coefs<DIM, NB>(u1, lam, a1);
        face_point<DIM>(r.lam[q], loc2, lam);
        grad_coefs<DIM, NB>(u2, lam, a2);
        double J[DIM];
#pragma unroll
        for (int k = 0; k < DIM; k++) {
            double p = 0.0, m = 0.0;
#pragma unroll
            for (int v = 0; v <= DIM; v++) {
                p += a1[v] * g1[v][k];
                m += a2[v] * g2[v][k];
            }
            J[k] = p - m;
        }
        double val = 0.0;
        if (kind == 1) {
            double jn = 0.0;
#pragma unroll
            for (int k = 0; k < DIM; k++) jn += J[k] * fnormals[(size_t)F * DIM + k];
            val = jn * jn;
        } else {
#pragma unroll
            for (int k = 0; k < DIM; k++) val += J[k] * J[k];
        }
        acc += r.w[q] * val;
    }
    const double fv = fvol[F];
    out[F] = acc * power_of(fv, power) * fv * factor;
}

// the table, or nullptr where it does not fit
double *cell_grads(grmp_mesh m) {
    grmp_context ctx = m->ctx;
    double *gl = nullptr;
    if (grmp_alloc_spare(ctx, (void **)&gl, (size_t)m->ncells * (m->dim + 1) * m->dim * 8)) {
        cudaGetLastError();
        ctx->last_error.clear();
        return nullptr;
    }
    if (m->dim == 2) k_cell_grads<2><<<nblk(m->ncells, 128), 128, 0, ctx->stream>>>(m->ncells, m->d_coords, m->d_cells, gl);
    else k_cell_grads<3><<<nblk(m->ncells, 128), 128, 0, ctx->stream>>>(m->ncells, m->d_coords, m->d_cells, gl);
    ctx->launches++;
    return gl;
}

// face matrices in flight: a chunk of faces at a time where all would take more
constexpr size_t kFaceBytes = (size_t)512 << 20;

// rule on the face's reference element (edge or triangle) as barycentric weights
int face_rule(grmp_context ctx, int dim, int order, FaceRule *r) {
    double (*x)[3] = new double[GRMP_MAXQ][3];
    double *w = new double[GRMP_MAXQ];
    const int nq = grmp_quadrature(dim - 1, order, x, w);
    const bool ok = nq > 0 && nq <= 32;
    if (ok) {
        r->nq = nq;
        for (int q = 0; q < nq; q++) {
            if (dim == 2) {
                r->lam[q][0] = 1.0 - x[q][0];
                r->lam[q][1] = x[q][0];
                r->lam[q][2] = 0.0;
            } else {
                r->lam[q][0] = 1.0 - x[q][0] - x[q][1];
                r->lam[q][1] = x[q][0];
                r->lam[q][2] = x[q][1];
            }
            r->w[q] = w[q];
        }
    }
    delete[] x;
    delete[] w;
    return ok ? GRMP_OK : grmp_fail(ctx, GRMP_ERR_UNSUPPORTED, "no face rule of order %d", order);
}

}  // namespace

int grmp_mesh_neighbors(grmp_mesh m) {
    grmp_context ctx = m->ctx;
    if (m->d_cell_nbr && m->d_face_cells) return GRMP_OK;
    if (m->nfaces <= 0) return grmp_fail(ctx, GRMP_ERR_INVALID_ARG, "face terms need the mesh's faces (set or build them)");
    const int nf = m->dim + 1;
    const long long n = (long long)m->ncells * nf;
    int32_t *cnt = nullptr, *fc = nullptr, *nbr = nullptr;
    int *bad = nullptr;
    int rc = grmp_alloc(ctx, (void **)&cnt, (size_t)m->nfaces * 4);
    if (!rc) rc = grmp_alloc(ctx, (void **)&fc, (size_t)m->nfaces * 8);
    if (!rc) rc = grmp_alloc(ctx, (void **)&nbr, (size_t)n * 4);
    if (!rc) rc = grmp_alloc(ctx, (void **)&bad, 4);
    int hbad = 0;
    if (!rc) {
        cudaMemsetAsync(cnt, 0, (size_t)m->nfaces * 4, ctx->stream);
        cudaMemsetAsync(bad, 0, 4, ctx->stream);
        k_face_count<<<nblk(n), TPB, 0, ctx->stream>>>(n, nf, m->d_cell_faces, cnt, fc);
        GRMP_LAUNCHED(ctx);
        k_face_order<<<nblk(m->nfaces), TPB, 0, ctx->stream>>>(m->nfaces, cnt, fc, bad);
        GRMP_LAUNCHED(ctx);
        k_cell_nbr<<<nblk(n), TPB, 0, ctx->stream>>>(n, nf, m->d_cell_faces, fc, nbr);
        GRMP_LAUNCHED(ctx);
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(&hbad, bad, 4, cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) rc = grmp_cuda_fail(ctx, e, "face adjacency");
        else if (hbad) rc = grmp_fail(ctx, GRMP_ERR_INVALID_ARG, "face adjacency: a face has no cell or more than two");
    }
    grmp_free(ctx, cnt, (size_t)m->nfaces * 4);
    grmp_free(ctx, bad, 4);
    if (rc) {
        grmp_free(ctx, fc, (size_t)m->nfaces * 8);
        grmp_free(ctx, nbr, (size_t)n * 4);
        return rc;
    }
    m->d_face_cells = fc;
    m->d_cell_nbr = nbr;
    return GRMP_OK;
}

int grmp_face_assemble(grmp_matrix A, int nterms, const grmp_bilinear_term *terms, int precision) {
    grmp_space s = A->space;
    grmp_mesh m = s->mesh;
    grmp_context ctx = m->ctx;
    const int dim = m->dim;
    if (s->ncomp != 1 || (s->fe != GRMP_FE_H1P1 && s->fe != GRMP_FE_H1P2))
        return grmp_fail(ctx, GRMP_ERR_UNSUPPORTED, "face terms: scalar H1P1 / H1P2 spaces");
    int rc = grmp_mesh_neighbors(m);
    if (rc) return rc;
    int *dmiss = nullptr;
    rc = grmp_alloc(ctx, (void **)&dmiss, 4);
    if (rc) return rc;
    cudaMemsetAsync(dmiss, 0, 4, ctx->stream);
    // scratch: gradients of the cells, matrices and columns of a chunk of faces; without room for them
    // the rows form their entries themselves
    double *gl = nullptr, *mats = nullptr;
    int32_t *fcol = nullptr, *fn = nullptr;
    const int nc = 2 * s->nb;
    const size_t per = (size_t)nc * nc * 8;
    const int chunk = (int)std::min<size_t>((size_t)m->nfaces, kFaceBytes / per);
    gl = cell_grads(m);
    // matrices, columns and numbers of a chunk in one piece
    if (grmp_alloc_spare(ctx, (void **)&mats, (size_t)chunk * (per + nc * 4 + 4))) {
        cudaGetLastError();
        ctx->last_error.clear();
    } else {
        fcol = reinterpret_cast<int32_t *>(mats + (size_t)chunk * nc * nc);
        fn = fcol + (size_t)chunk * nc;
    }
    auto release = [&]() {
        grmp_free(ctx, dmiss, 4);
        grmp_free(ctx, gl, (size_t)m->ncells * (dim + 1) * dim * 8);
        grmp_free(ctx, mats, (size_t)chunk * (per + nc * 4 + 4));
    };
    const FaceGeom geo{m->d_cell_faces, m->d_cells, s->d_celldofs, m->d_coords, gl, m->d_face_volumes};
    double *v64 = precision != GRMP_FP32 ? A->d_vals64 : nullptr;
    float *v32 = precision != GRMP_FP64 ? A->d_vals32 : nullptr;
    const int p = grmp_fe_polyorder(s->fe, dim);
    for (int i = 0; i < nterms && !rc; i++) {
        FaceRule r;
        std::memset(&r, 0, sizeof(r));
        // Jump(Gradient) x Jump(Gradient) on the face geometry: 2 (p - 1) + bonus
        int order = 2 * (p - 1) + terms[i].bonus_quadorder;
        rc = face_rule(ctx, dim, order < 0 ? 0 : order, &r);
        if (rc) break;
        FaceTermDev t{terms[i].factor, terms[i].param[0]};
        // the FP32 values get the FP64 contributions rounded; v64 is always
        // present here (the cell assembly that precedes this allocates it)
        double *w64 = v64;
        float *w32 = v32;
        if (!w64) {
            rc = grmp_fail(ctx, GRMP_ERR_UNSUPPORTED, "face terms: FP64 values are required (use FP64 or FP64_FP32)");
            break;
        }
        auto go = [&](auto mat, auto add, auto rows, int nb, int lpr) {
            const int nc = 2 * nb;
            const size_t fsm = ((size_t)r.nq * nc * dim + 1) * 8 + (1 + nb) * 4;
            const int fb = (int)std::max<size_t>(1, std::min<size_t>(32, (size_t)46 * 1024 / fsm));
            for (int F0 = 0; F0 < m->nfaces; F0 += chunk) {
                const int nf = std::min(chunk, m->nfaces - F0);
                if (!mats) {
                    rows<<<nblk(A->nrows, 128), 128, 0, ctx->stream>>>(
                        A->nrows, F0, nf, s->d_inc_ptr, s->d_inc_cell, m->d_cell_nbr, A->d_rowptr, A->d_cols, w64, w32,
                        dmiss, geo, t, r);
                    GRMP_LAUNCHED(ctx);
                    continue;
                }
                mat<<<nblk(nf, fb), 128, fb * fsm + 8, ctx->stream>>>(F0, nf, fb, m->d_face_cells, m->d_cell_faces,
                                                                      m->d_cells, m->d_coords, s->d_celldofs, gl, m->d_face_volumes,
                                                                      t, r, mats, fcol, fn);
                GRMP_LAUNCHED(ctx);
                add<<<nblk((long long)A->nrows * lpr, 128), 128, 0, ctx->stream>>>(
                    A->nrows, F0, nf, s->d_inc_ptr, s->d_inc_cell, m->d_cell_faces, m->d_cell_nbr, mats, fcol, fn,
                    A->d_rowptr, A->d_cols, w64, w32, dmiss);
                GRMP_LAUNCHED(ctx);
            }
        };
        if (dim == 2 && s->nb == 3) go(k_face_mats<2, 3>, k_face_add<2, 3, 8>, k_face_rows<2, 3>, 3, 8);
        else if (dim == 2 && s->nb == 6) go(k_face_mats<2, 6>, k_face_add<2, 6, 16>, k_face_rows<2, 6>, 6, 16);
        else if (dim == 3 && s->nb == 4) go(k_face_mats<3, 4>, k_face_add<3, 4, 8>, k_face_rows<3, 4>, 4, 8);
        else go(k_face_mats<3, 10>, k_face_add<3, 10, 32>, k_face_rows<3, 10>, 10, 32);
    }
    int hmiss = 0;
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(&hmiss, dmiss, 4, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    release();
    if (!rc && e != cudaSuccess) rc = grmp_cuda_fail(ctx, e, "face terms");
    if (!rc && hmiss)
        rc = grmp_fail(ctx, GRMP_ERR_INVALID_ARG, "face terms: the pattern lacks face couplings (build it with the face terms)");
    return rc;
}

extern "C" int grmp_item_face_jumps(grmp_space s, grmp_vector u, int kind, double power, double factor,
                                    int bonus_quadorder, double *face_values, double *total) {
    if (!s || !u || (kind != 0 && kind != 1)) return GRMP_ERR_INVALID_ARG;
    grmp_mesh m = s->mesh;
    grmp_context ctx = m->ctx;
    if (u->ctx != ctx || u->n != s->ndofs) return grmp_fail(ctx, GRMP_ERR_INVALID_ARG, "face jumps: vector mismatch");
    cudaSetDevice(ctx->device);
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    if (s->ncomp != 1 || (s->fe != GRMP_FE_H1P1 && s->fe != GRMP_FE_H1P2))
        return grmp_fail(ctx, GRMP_ERR_UNSUPPORTED, "face jumps: scalar H1P1 / H1P2 spaces");
    int rc = grmp_mesh_neighbors(m);
    if (rc) return rc;
    const int dim = m->dim, p = grmp_fe_polyorder(s->fe, dim);
    FaceRule r;
    std::memset(&r, 0, sizeof(r));
    int order = 2 * (p - 1) + bonus_quadorder;
    rc = face_rule(ctx, dim, order < 0 ? 0 : order, &r);
    if (rc) return rc;
    double *dout = nullptr;
    rc = grmp_alloc(ctx, (void **)&dout, (size_t)m->nfaces * 8);
    if (rc) return rc;
    double *gl = cell_grads(m);
    const size_t glb = (size_t)m->ncells * (dim + 1) * dim * 8;
    auto go = [&](auto kern) {
        kern<<<nblk(m->nfaces, 128), 128, 0, ctx->stream>>>(m->nfaces, m->d_face_cells, m->d_cell_faces, m->d_cells, m->d_coords, gl,
                                                       s->d_celldofs, u->d, m->d_face_normals,
                                                       m->d_face_volumes, kind, power, factor, r, dout);
    };
    if (dim == 2 && s->nb == 3) go(k_face_jumps<2, 3>);
    else if (dim == 2 && s->nb == 6) go(k_face_jumps<2, 6>);
    else if (dim == 3 && s->nb == 4) go(k_face_jumps<3, 4>);
    else go(k_face_jumps<3, 10>);
    GRMP_LAUNCHED(ctx);
    std::vector<double> h((size_t)m->nfaces);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(h.data(), dout, h.size() * 8, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    grmp_free(ctx, dout, (size_t)m->nfaces * 8);
    grmp_free(ctx, gl, glb);
    if (e != cudaSuccess) return grmp_cuda_fail(ctx, e, "face jumps");
    double sum = 0.0;   // ascending face order (evaluate!, itemintegrator.jl:314-330)
    for (double v : h) sum += v;
    if (face_values) std::memcpy(face_values, h.data(), h.size() * 8);
    if (total) *total = sum;
    return GRMP_OK;
}
