// Multilevel preconditioned conjugate gradients for scalar elliptic matrices
// (H1P1 / H1P2 spaces with a diffusion term), FP64 and mixed.
//
// Jacobi-PCG needs O(1/h) iterations (64^3 P2 Poisson 1,031, 128^2 P2 1,203)
// and each is bound by the latency of its gathers and grid barriers, so what
// pays is fewer iterations.  The preconditioner is one multilevel cycle:
//
//   z = V(r)                        (small and medium systems: fine_mult)
//   z = c D_0 r + P_0 V(P_0^T r)    (large ones)
//
// a symmetric V(1,1) cycle, additive on the fine level of large systems (its
// Jacobi part costs no product with the fine matrix, so an iteration keeps one
// fine SpMV).  P_0 of a P2 space
// interpolates from the vertices (P1 is in P2); all other levels are smoothed
// aggregation, P = (I - w D A) P_agg.  D = 1 / sum_j |a_ij| (l1-Jacobi:
// convergent for every SPD matrix without an eigenvalue estimate).  With
// S = w D the cycle on level l is
//
//   r_{l+1} = Q^T r_l,      e_l = 2 S r_l - S A S r_l + Q e_{l+1},
//   Q = P - S A P,
//
// which is one pre- and one post-smoothing step written with the smoothed
// prolongation Q: one phase down and one up per level (two grid barriers
// instead of four); Q is formed with the coarse matrices from A P.
//
// The hierarchy's patterns are built once per matrix pattern on the host
// (mg_symbolic.cpp); its values are formed on the device at every solve, from
// the matrix as it is then.  Rows without off-diagonal values (Dirichlet rows
// of either kind) are left out of the coarse spaces.  Everything is in the
// precision of the iteration (FP32 inside the FP64 refinement of mixed
// solves, FP64 throughout in FP64 solves), every sum has a fixed order.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <vector>

#include "mg.h"
#include "mg_symbolic.h"
#include "pcg_device.cuh"

namespace {

constexpr int kTB = 256;
constexpr int kMgT = 384;         // threads per block of the solvers: two blocks fit an SM at 85 registers a thread
// lanes per row of an operator by mean entries a row: 4 up to kShortRow (vertex
// level on right angles: 7), 8, and a warp from kLongRow (transposes of wide
// aggregates: 100-600).  FP64 with kManyRows rows and more is bound by the FP64
// unit (two lanes a clock: a step of the shuffle reduction costs as much as a
// multiplication of all lanes) and takes fewer: 61^3 P1, phases of an
// iteration, restriction / up / fine level 27 / 22 / 44 us before, 15 / 19 / 35 us now.
constexpr int kShortRow = 10, kLongRow = 48, kManyRows = 8192;
template <typename T>
int lanes_of(size_t entries, int rows) {
    if (sizeof(T) == 8 && rows >= kManyRows)
        return entries <= (size_t)24 * rows ? 2 : (entries <= (size_t)64 * rows ? 4 : (entries <= (size_t)400 * rows ? 8 : 32));
    return entries <= (size_t)kShortRow * rows ? 4 : (entries <= (size_t)kLongRow * rows ? 8 : 32);
}
constexpr double kSmooth = 1.7;   // w of the smoothing steps and c of the fine level (l1-scaled: spectrum in (0, 1])
// reaction-dominated matrices (energy of the constant function against the
// diagonal) converge in a few dozen Jacobi iterations: they keep that solver.
// The look costs a pass over the matrix and a stop of the stream (which then
// serves the Jacobi solver's diagonal check too), once per set of values
constexpr double kMaxReaction = 0.02;
// Jacobians that take more BiCGStab iterations than kMaxBicg (15-50 on smooth
// iterates, up to 95 on white noise, where Jacobi takes 200-800), or have not
// gained a digit after kStallBicg, are left to the Jacobi iteration
constexpr int kMaxBicg = 200, kStallBicg = 40;
// Conjugate gradients are given up when, kStall iterations times k = 2, 3, ...
// on, the residual has not fallen by k digits: mixed solves then go on with the
// FP64 cycle, FP64 ones with the Jacobi iteration.  Coefficients that jump by
// 1e5 and more across element sides, and long strips fixed at one end, lose the FP32
// recurrence its conjugacy (80^2 P1 squares, contrast 1e6, to 1e-8: no convergence in
// 20,000 FP32 iterations, 274 in FP64; Jacobi 990 / 2,163 in FP64 / mixed).  What converges
// keeps ahead of that: lognormal coefficients with sigma 3 (435 iterations to 1e-11)
// have lost five digits at 128; FP64 at contrast 1e6 two at 128, four to six at 256.
constexpr int kStall32 = 64, kStall64 = 128;
// (rn0, the start's residual, waits in shared memory: it is needed once in kStall
// iterations, and registers are what the iterations are short of)
__device__ __forceinline__ bool mg_behind(int it, int every, double rn, const double *rn0) {
    double lim = *rn0;
    for (int k = it / every; k > 0; k--) lim *= 0.1;
    return rn > lim;
}

// Rows from which the multilevel solver is taken: where whole passes are no
// slower than with Jacobi-PCG for constant coefficients (lognormal ones gain
// more).  Multilevel / Jacobi, constant, ms: 2D mixed 121 rows 0.35 / 0.43; 2D
// FP64 225 rows 0.73 / 0.70, 441 rows 1.02 / 1.01 (P1), 0.89 / 1.30 (P2); 3D P1
// mixed 2,197 rows 0.72 / 0.70, 4,913 rows 0.81 / 0.95; 3D P1 FP64 1,000 rows
// 0.78 / 0.73, 2,197 rows 0.93 / 0.98; 3D P2 mixed 1,331 rows 0.93 / 0.90, 2,197
// rows 0.94 / 1.02; 3D P2 FP64 729 rows 1.11 / 1.07, 1,331 rows 1.20 / 1.28.
// BiCGStab (a Jacobi iteration there costs 43 us): Newton steps of 441 rows 1.2 / 2.6-2.9.
int min_rows(int dim, int fe, bool mixed, bool bicg) {
    if (bicg) return dim == 2 ? 200 : 500;
    if (dim == 2) return mixed ? 120 : 440;
    if (fe == GRMP_FE_H1P2) return mixed ? 2000 : 1300;
    return mixed ? 2500 : 2000;
}

// Whether the fine level is smoothed multiplicatively too, which costs a
// product with the matrix, one with Q_0 and a longer restriction an iteration and saves
// 30-50 % of the iterations: while an iteration is mostly phases and barriers.
// Additive / multiplicative, whole passes, ms: 2D P2 1,089 rows 0.76 / 0.72
// (37 / 21 iterations), 63,001 rows 2.35 / 1.77, FP64 641,601 rows 9.9 / 10.7; 2D
// P1 491,401 rows mixed 6.3 / 4.7, FP64 10.4 / 7.9; 3D P1 238,328 rows FP64
// 5.61 / 5.46 (46 / 26), 531,441 rows 10.4 / 10.8; 3D P2 6,859 rows 1.73 / 1.16,
// 117,649 rows mixed 2.9 / 2.5, FP64 4.2 / 4.4, 804,357 rows mixed 9.4 / 10.5.
bool fine_mult(int dim, int fe, int n) { return n <= (dim == 3 && fe == GRMP_FE_H1P2 ? 80000 : 400000); }

template <typename T>
struct alignas(2 * sizeof(T)) Pair {
    T a, b;
};

template <typename T>
struct MgLv {
    int n;
    const int32_t *rp, *ci;       // A
    const T *v, *D;
    const int32_t *qrp, *qci;     // Q: n x next n
    const T *qv;
    const int32_t *trp, *tci;     // Q^T
    const T *tv;
    int lanes, tlanes;            // lanes per row of A and Q (one choice: the same lane owns a row in both), of Q^T
    T *r, *y, *e;
};

template <typename T>
struct MgDev {
    int nl, dense, rlanes;        // levels, dense inverse at the bottom, lanes per row of P_0^T
    const int32_t *prp, *pci;     // P_0 and its transpose
    const T *pv;
    const int2 *ell;              // P_0 of a P2 space as two entries a row (nullptr: CSR)
    const Pair<T> *ellv;
    const int32_t *rrp, *rci;
    const T *rv;
    const T *D0, *binv;
    // fine level smoothed multiplicatively: Q_0 (its transpose is in rrp, rci, rv), lanes per row of A
    // and Q_0, A in the cycle's precision and a vector
    int mult, flanes;
    const int32_t *frp, *fci, *q0rp, *q0ci;
    const T *fv, *q0v;
    T *z0;
    MgLv<T> lv[kMgMaxLevels + 1];
};

// ------------------------------------------------------------------ values of the hierarchy
// D, the rows without coupling, and (level 0) per-block sums of the positive
// row sums and diagonals of the rows away from eliminated DoFs, bad diagonals
template <typename T, int kCl>
__global__ void __launch_bounds__(kTB) k_mg_rows(int n, const int32_t *rp, const int32_t *ci, const T *v, T *D,
                                                 uint8_t *iso, const uint8_t *fixed, double2 *part, int *bad) {
    __shared__ double sh[32 * 2];
    const int lane = threadIdx.x & (kCl - 1);
    double s0 = 0.0, s1 = 0.0;
    for (long long base = blockIdx.x * (long long)(kTB / kCl); base < n; base += (long long)gridDim.x * (kTB / kCl)) {
        const int i = (int)base + threadIdx.x / kCl;
        T off = 0, d = 0, sum = 0;
        int zero = 0;
        if (i < n)
            for (int k = rp[i] + lane; k < rp[i + 1]; k += kCl) {
                const T a = v[k];
                sum += a;
                if (ci[k] == i) d = a;
                else {
                    off += fabs(a);
                    if (a == T(0) && fixed) zero |= fixed[ci[k]];   // an eliminated coupling
                }
            }
        for (int o = kCl / 2; o > 0; o >>= 1) {
            off += __shfl_xor_sync(0xffffffffu, off, o);
            d += __shfl_xor_sync(0xffffffffu, d, o);
            sum += __shfl_xor_sync(0xffffffffu, sum, o);
            zero |= __shfl_xor_sync(0xffffffffu, zero, o);
        }
        if (i < n && lane == 0) {
            const T s = off + fabs(d);
            const bool lone = off <= T(1e-8) * fabs(d);
            D[i] = s > T(0) ? T(1) / s : T(1);
            iso[i] = lone;
            if (bad && (!(d > T(0)) || !isfinite((double)s))) atomicExch(bad, 1);
            if (!lone && !zero) {
                s0 += sum > T(0) ? (double)sum : 0.0;
                s1 += (double)d;
            }
        }
    }
    if (!part) return;
    double v2[2] = {s0, s1};
    block_sum<2>(v2, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = make_double2(v2[0], v2[1]);
}

// vertex interpolation: 1 at a vertex, 1/2 from the two ends of an edge; fixed DoFs neither receive nor give
template <typename T>
__global__ void k_mg_prol_geo(int n, const int32_t *prp, const int32_t *pci, const int32_t *vrow, const uint8_t *iso,
                              T *pv, Pair<T> *ellv) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int b = prp[i], e = prp[i + 1];
    T w[2] = {T(0), T(0)};
    for (int q = b; q < e; q++) {
        w[q - b] = iso[i] || iso[vrow[pci[q]]] ? T(0) : (e - b == 1 ? T(1) : T(0.5));
        pv[q] = w[q - b];
    }
    ellv[i] = Pair<T>{w[0], w[1]};
}

// position of column c in a row's ascending columns, -1 if it is not there
__device__ __forceinline__ int mg_find(const int32_t *cols, int n, int c) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (cols[mid] < c) lo = mid + 1;
        else hi = mid;
    }
    return lo < n && cols[lo] == c ? lo : -1;
}

// P = (I - w D A) P_agg, L lanes a row (1 on long levels; 16 on short ones,
// whose rows hold hundreds of entries: 3,000 rows 57 us with one lane)
template <typename T, int L>
__global__ void k_mg_prol_agg(int n, const int32_t *rp, const int32_t *ci, const T *v, const T *D, const uint8_t *iso,
                              const int32_t *agg, const int32_t *prp, const int32_t *pci, T *pv) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) / L, lane = threadIdx.x & (L - 1);
    const bool in = i < n;   // whole warps take part in the shuffles
    const int kb = in ? rp[i] : 0, ke = in ? rp[i + 1] : 0, own = in ? agg[i] : -1;
    const bool lone = in && iso[i];
    const T w = in ? (T)kMgProlong * D[i] : T(0);
    const int q0 = in ? prp[i] : 0;
    int nq = in ? prp[i + 1] - q0 : 0;
    if (L > 1) nq = __reduce_max_sync(0xffffffffu, nq);
    for (int q = q0; q < q0 + nq; q++) {
        const int t = in && q < prp[i + 1] ? pci[q] : -1;
        T s = 0;
        for (int k = kb + lane; k < ke; k += L)
            if (agg[ci[k]] == t) s += v[k];
        for (int o = L / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0 && t >= 0) pv[q] = lone ? T(0) : (t == own ? T(1) : T(0)) - w * s;
    }
}

// Couplings to aggregates that a row of P lacks (weak ones, on stretched
// meshes) go to its own aggregate, so that rows without Dirichlet neighbours
// keep their sum of one; 8 lanes a row
template <typename T>
__global__ void k_mg_prol_lump(int n, const int32_t *rp, const int32_t *ci, const T *v, const T *D, const uint8_t *iso,
                               const int32_t *agg, const int32_t *prp, const int32_t *pci, T *pv) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) / 8, lane = threadIdx.x & 7;
    const bool in = i < n && !iso[i];   // whole warps take part in the shuffles
    const int q0 = in ? prp[i] : 0, nq = in ? prp[i + 1] - q0 : 0;
    T s = 0;
    if (in)
        for (int k = rp[i] + lane; k < rp[i + 1]; k += 8)
            if (mg_find(pci + q0, nq, agg[ci[k]]) < 0) s += v[k];
    for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (in && lane == 0) pv[q0 + mg_find(pci + q0, nq, agg[i])] -= (T)kMgProlong * D[i] * s;
}

// Sparse products, a group of lanes per row of the result.  The factor rows
// that make up a result row are taken one after another, the lanes take the
// entries of one of them (distinct columns: no two lanes add to one place, so
// the order is fixed) and add into the row's accumulators in shared memory;
// rows longer than kRowCap accumulate in the result itself.  FP64: passing
// the entries round by shuffles to a lane per result entry issued a 32-lane
// FP64 addition for each one (2 lanes a clock): 61^3 P1, all levels, 2.9 ms a
// pass with that, see the caller for this form.
constexpr int kRowCap = 64;

// A P, 8 lanes a row
template <typename T>
__global__ void __launch_bounds__(kTB) k_mg_ap(int n, const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                                               const T *__restrict__ v, const int32_t *__restrict__ prp,
                                               const int32_t *__restrict__ pci, const T *__restrict__ pv,
                                               const int32_t *__restrict__ arp, const int32_t *aci, T *av) {
    constexpr int L = 8;
    __shared__ T sacc[kTB / L][kRowCap];
    __shared__ int32_t scol[kTB / L][kRowCap];
    const int lane = threadIdx.x & (L - 1), g = threadIdx.x / L;
    const int ng = gridDim.x * (kTB / L), pad = (n + 3) & ~3;   // whole warps go round together
    for (int i = blockIdx.x * (kTB / L) + g; i < pad; i += ng) {
        const int kb = i < n ? rp[i] : 0, m = i < n ? rp[i + 1] - kb : 0;
        const int t0 = i < n ? arp[i] : 0, nt = i < n ? arp[i + 1] - t0 : 0;
        const bool small = nt <= kRowCap;
        T *acc = small ? sacc[g] : av + t0;
        const int32_t *cols = small ? scol[g] : aci + t0;
        for (int t = lane; t < nt; t += L) {
            acc[t] = T(0);
            if (small) scol[g][t] = aci[t0 + t];
        }
        __syncwarp();
        const int longest = __reduce_max_sync(0xffffffffu, m);
        for (int k0 = 0; k0 < longest; k0 += L) {
            int p0 = 0, len = 0;
            T a = 0;
            if (k0 + lane < m) {
                const int j = ci[kb + k0 + lane];
                a = v[kb + k0 + lane];
                p0 = prp[j];
                len = prp[j + 1] - p0;
            }
            const int steps = min(L, longest - k0);
            for (int k = 0; k < steps; k++) {
                const int b = __shfl_sync(0xffffffffu, p0, k, L), ln = __shfl_sync(0xffffffffu, len, k, L);
                const T ak = __shfl_sync(0xffffffffu, a, k, L);
                for (int q = lane; q < ln; q += L) {
                    const int s = mg_find(cols, nt, pci[b + q]);
                    if (s >= 0) acc[s] += ak * pv[b + q];
                }
                __syncwarp();
            }
        }
        if (small)
            for (int t = lane; t < nt; t += L) av[t0 + t] = acc[t];
        __syncwarp();
    }
}

// The same for the vertex interpolation (two entries a row of P), 16 lanes a
// row and a lane per result entry: the row's entries and their pairs are
// passed round by shuffles.  64^3 P2 (55.6M entries), FP32: 1.95 ms a pass
// with the form above, 0.85 ms with this one, bound by the shuffles.
template <typename T>
__global__ void __launch_bounds__(kTB) k_mg_ap_geo(int n, const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                                                   const T *__restrict__ v, const int2 *__restrict__ ell,
                                                   const Pair<T> *__restrict__ ellv, const int32_t *__restrict__ arp,
                                                   const int32_t *__restrict__ aci, T *av) {
    constexpr int L = 16;
    const int lane = threadIdx.x & (L - 1);
    const int ng = gridDim.x * (kTB / L), pad = (n + 1) & ~1;
    for (int i = blockIdx.x * (kTB / L) + threadIdx.x / L; i < pad; i += ng) {
        const int kb = i < n ? rp[i] : 0, ke = i < n ? rp[i + 1] : 0;
        const int t0 = i < n ? arp[i] : 0, te = i < n ? arp[i + 1] : 0;
        const int chunks = __reduce_max_sync(0xffffffffu, (te - t0 + L - 1) / L);
        const int longest = __reduce_max_sync(0xffffffffu, ke - kb);
        for (int tc = 0; tc < chunks; tc++) {
            const int tb = t0 + tc * L + lane;
            const int mine = tb < te ? aci[tb] : -1;
            T acc = 0;
            for (int k0 = 0; k0 < longest; k0 += L) {
                int2 c = make_int2(-2, -2);
                T wa = 0, wb = 0;
                if (kb + k0 + lane < ke) {
                    const int j = ci[kb + k0 + lane];
                    const T a = v[kb + k0 + lane];
                    c = ell[j];
                    const Pair<T> w = ellv[j];
                    wa = a * w.a;
                    wb = a * w.b;
                }
                const int m = min(L, longest - k0);
                for (int k = 0; k < m; k++) {
                    const int ca = __shfl_sync(0xffffffffu, c.x, k, L), cb = __shfl_sync(0xffffffffu, c.y, k, L);
                    const T xa = __shfl_sync(0xffffffffu, wa, k, L), xb = __shfl_sync(0xffffffffu, wb, k, L);
                    if (ca == mine) acc += xa;
                    if (cb == mine) acc += xb;
                }
            }
            if (tb < te) av[tb] = acc;
        }
    }
}

// cells whose longest edge is more than kStretch times their smallest height
constexpr double kStretch = 4.0;   // 2.0 on squares split in triangles, 2.45 on Kuhn cubes
template <int DIM>
__global__ void k_mg_stretched(int ncells, const double *coords, const int32_t *cells, int *count) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    bool s = false;
    if (c < ncells) {
        double X[DIM + 1][DIM], longest = 0.0, face = 0.0;
        for (int v = 0; v <= DIM; v++)
            for (int k = 0; k < DIM; k++) X[v][k] = coords[(size_t)cells[(size_t)c * (DIM + 1) + v] * DIM + k];
        for (int a = 0; a < DIM; a++)
            for (int b = a + 1; b <= DIM; b++) {
                double l = 0.0;
                for (int k = 0; k < DIM; k++) l += (X[a][k] - X[b][k]) * (X[a][k] - X[b][k]);
                longest = fmax(longest, l);
            }
        if (DIM == 2) {
            // longest edge squared against twice the area
            const double det = (X[1][0] - X[0][0]) * (X[2][1] - X[0][1]) - (X[1][1] - X[0][1]) * (X[2][0] - X[0][0]);
            s = longest > kStretch * fabs(det);
        } else {
            // longest edge times twice the largest face's area against six volumes
            double det = 0.0;
            for (int f = 0; f < 4; f++) {
                const int o = f == 0 ? 1 : 0, a = f <= 1 ? 2 : 1, b = f <= 2 ? 3 : 2;   // the face without vertex f
                double u[3], w[3], n[3];
                for (int k = 0; k < 3; k++) {
                    u[k] = X[a][k % DIM] - X[o][k % DIM];
                    w[k] = X[b][k % DIM] - X[o][k % DIM];
                }
                for (int k = 0; k < 3; k++) n[k] = u[(k + 1) % 3] * w[(k + 2) % 3] - u[(k + 2) % 3] * w[(k + 1) % 3];
                face = fmax(face, n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
                if (f == 0) {
                    det = 0.0;
                    for (int k = 0; k < 3; k++) det += n[k] * (X[0][k % DIM] - X[1][k % DIM]);
                }
            }
            s = sqrt(longest * face) > kStretch * fabs(det);
        }
    }
    const unsigned m = __ballot_sync(0xffffffffu, s);
    if ((threadIdx.x & 31) == 0 && m) atomicAdd(count, __popc(m));
}

// next level's matrix P^T (A P), 16 lanes a row; a row without values (only
// fixed DoFs below it) becomes the identity's.  Couplings that the pattern
// leaves out (filtered vertex level) are added to the diagonal.
template <typename T>
__global__ void __launch_bounds__(kTB) k_mg_rap(int nc, const int32_t *__restrict__ rrp, const int32_t *__restrict__ rci,
                                                const int32_t *__restrict__ rperm, const T *__restrict__ pv,
                                                const int32_t *__restrict__ arp, const int32_t *__restrict__ aci,
                                                const T *__restrict__ av, const int32_t *__restrict__ crp,
                                                const int32_t *cci, T *cv) {
    constexpr int L = 16;
    __shared__ T sacc[kTB / L][kRowCap];
    __shared__ int32_t scol[kTB / L][kRowCap];
    const int lane = threadIdx.x & (L - 1), g = threadIdx.x / L;
    const int ng = gridDim.x * (kTB / L), pad = (nc + 1) & ~1;
    for (int I = blockIdx.x * (kTB / L) + g; I < pad; I += ng) {
        const int t0 = I < nc ? crp[I] : 0, nt = I < nc ? crp[I + 1] - t0 : 0;
        const int kb = I < nc ? rrp[I] : 0, m = I < nc ? rrp[I + 1] - kb : 0;
        const bool small = nt <= kRowCap;
        T *acc = small ? sacc[g] : cv + t0;
        const int32_t *cols = small ? scol[g] : cci + t0;
        for (int t = lane; t < nt; t += L) {
            acc[t] = T(0);
            if (small) scol[g][t] = cci[t0 + t];
        }
        __syncwarp();
        T lump = 0;
        const int longest = __reduce_max_sync(0xffffffffu, m);
        for (int k0 = 0; k0 < longest; k0 += L) {
            int a0 = 0, len = 0;
            T w = 0;
            if (k0 + lane < m) {
                const int i = rci[kb + k0 + lane];
                w = pv[rperm[kb + k0 + lane]];
                a0 = arp[i];
                len = w == T(0) ? 0 : arp[i + 1] - a0;
            }
            const int steps = min(L, longest - k0);
            for (int k = 0; k < steps; k++) {
                const int b = __shfl_sync(0xffffffffu, a0, k, L), ln = __shfl_sync(0xffffffffu, len, k, L);
                const T wk = __shfl_sync(0xffffffffu, w, k, L);
                for (int q = lane; q < ln; q += L) {
                    const int s = mg_find(cols, nt, aci[b + q]);
                    const T x = wk * av[b + q];
                    if (s >= 0) acc[s] += x;
                    else lump += x;
                }
                __syncwarp();
            }
        }
        bool any = false;
        for (int t = lane; t < nt; t += L) any = any || acc[t] != T(0);
        for (int o = L / 2; o > 0; o >>= 1) {
            any = __shfl_xor_sync(0xffffffffu, (int)any, o) || any;
            lump += __shfl_xor_sync(0xffffffffu, lump, o);
        }
        for (int t = lane; t < nt; t += L) cv[t0 + t] = acc[t] + (cols[t] == I ? (any ? lump : T(1)) : T(0));
        __syncwarp();
    }
}

// The two products on short levels: a block per result row.  Its entries are
// many (aggregates of hundreds of rows) and the rows few, so one group of
// lanes a row is a serial chain on a few SMs (61^3 P1, levels of 779 and 16
// rows: P^T A P 283 and 240 us, A P 63 and 47).  32 groups of 8 lanes take
// the factor rows in turn into accumulators of their own in shared memory,
// summed in the groups' order.  RAP = false: A P; true: P^T (A P), with the
// lumping and the identity rows of k_mg_rap.
constexpr int kWideG = 32;
template <typename T, bool RAP>
__global__ void __launch_bounds__(kTB) k_mg_wide(const int32_t *__restrict__ lrp, const int32_t *__restrict__ lci, const int32_t *__restrict__ lperm,
                                                 const T *__restrict__ lv, const int32_t *__restrict__ frp,
                                                 const int32_t *__restrict__ fci, const T *__restrict__ fv,
                                                 const int32_t *__restrict__ orp, const int32_t *__restrict__ oci, T *ov) {
    constexpr int L = kTB / kWideG;
    extern __shared__ __align__(16) unsigned char wsm[];
    T *acc = reinterpret_cast<T *>(wsm);   // [kWideG][nt], then the row's columns
    __shared__ T slump[kWideG];
    __shared__ int sany;
    const int I = blockIdx.x, lane = threadIdx.x & (L - 1), g = threadIdx.x / L;
    const int t0 = orp[I], nt = orp[I + 1] - t0, kb = lrp[I], m = lrp[I + 1] - kb;
    int32_t *cols = reinterpret_cast<int32_t *>(acc + kWideG * nt);
    for (int t = threadIdx.x; t < nt; t += kTB) cols[t] = oci[t0 + t];
    for (int t = threadIdx.x; t < kWideG * nt; t += kTB) acc[t] = T(0);
    if (threadIdx.x == 0) sany = 0;
    __syncthreads();
    T *mine = acc + g * nt;
    T lump = 0;
    const unsigned mask = ((1u << L) - 1u) << (threadIdx.x & 31 & ~(L - 1));
    for (int k = g; k < m; k += kWideG) {
        const int j = lci[kb + k];
        const T w = lv[RAP ? lperm[kb + k] : kb + k];
        const int b = frp[j], ln = RAP && w == T(0) ? 0 : frp[j + 1] - b;
        for (int q = lane; q < ln; q += L) {
            const int s = mg_find(cols, nt, fci[b + q]);
            const T x = w * fv[b + q];
            if (s >= 0) mine[s] += x;
            else lump += x;
        }
        __syncwarp(mask);
    }
    if (RAP) {
        for (int o = L / 2; o > 0; o >>= 1) lump += __shfl_xor_sync(0xffffffffu, lump, o);
        if (lane == 0) slump[g] = lump;
    }
    __syncthreads();
    bool any = false;
    for (int t = threadIdx.x; t < nt; t += kTB) {
        T s = 0;
        for (int q = 0; q < kWideG; q++) s += acc[q * nt + t];
        any = any || s != T(0);
        if (RAP) acc[t] = s;   // this thread's column of group 0: read by nobody else
        else ov[t0 + t] = s;
    }
    if (!RAP) return;
    if (any) sany = 1;
    __syncthreads();
    T all = 0;
    for (int q = 0; q < kWideG; q++) all += slump[q];
    for (int t = threadIdx.x; t < nt; t += kTB) ov[t0 + t] = acc[t] + (cols[t] == I ? (sany ? all : T(1)) : T(0));
}

// Q = P - w D (A P), in place of A P (both rows ascending)
template <typename T>
__global__ void k_mg_q(int n, const int32_t *prp, const int32_t *pci, const T *pv, const int32_t *arp,
                       const int32_t *aci, const T *D, T *av) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int q = prp[i];
    const int qe = prp[i + 1];
    const T w = (T)kSmooth * D[i];
    for (int t = arp[i]; t < arp[i + 1]; t++) {
        T x = -w * av[t];
        while (q < qe && pci[q] < aci[t]) q++;
        if (q < qe && pci[q] == aci[t]) x += pv[q];
        av[t] = x;
    }
}

template <typename T>
__global__ void k_mg_perm(int n, const int32_t *perm, const T *a, T *b) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) b[i] = a[perm[i]];
}

// dense inverse of the bottom matrix (n <= kMgBottom = 96) by Gauss-Jordan,
// one block: 16 warps by 32 lanes hold six rows by three columns each in
// registers, row and column k of a step come through shared memory (two
// buffers: one barrier a step).  With the matrix in shared memory and a
// division per element index it took 0.9 us a step (81 rows FP32 76 us), now
// 23 us.  A direction that is zero to rounding (pure Neumann problems) is
// left out.
template <typename T>
__global__ void __launch_bounds__(512) k_mg_binv(int n, const int32_t *rp, const int32_t *ci, const T *v, T *inv) {
    static_assert(kMgBottom == 96, "six rows by three columns a thread");
    extern __shared__ __align__(16) unsigned char mg_smem[];
    T *M = reinterpret_cast<T *>(mg_smem);
    __shared__ T col[2][kMgBottom], row[2][kMgBottom], diag[kMgBottom];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = threadIdx.x; k < n * n; k += blockDim.x) M[k] = T(0);
    __syncthreads();
    for (int i = warp; i < n; i += 16)
        for (int k = rp[i] + lane; k < rp[i + 1]; k += 32) {
            const int j = ci[k];
            M[i * n + j] = v[k];
            if (j == i) diag[i] = v[k];
        }
    __syncthreads();
    T m[6][3];
#pragma unroll
    for (int a = 0; a < 6; a++)
#pragma unroll
        for (int b = 0; b < 3; b++) {
            const int i = warp + 16 * a, j = lane + 32 * b;
            m[a][b] = i < n && j < n ? M[i * n + j] : T(0);
        }
    const T eps = sizeof(T) == 8 ? T(1e-13) : T(1e-5);
    // k = 16 ka + q: the register row ka and column ka / 2 of step k are known to the compiler
#pragma unroll
    for (int ka = 0; ka < 6; ka++) {
        const int kb = ka / 2;
#pragma unroll 1
        for (int q = 0; q < 16; q++) {
            const int k = 16 * ka + q;
            if (k >= n) break;
            T *ck = col[k & 1], *rk = row[k & 1];
            const bool mycol = lane == (k & 31), myrow = warp == q;
            if (mycol)
#pragma unroll
                for (int a = 0; a < 6; a++) ck[warp + 16 * a] = m[a][kb];
            if (myrow)
#pragma unroll
                for (int b = 0; b < 3; b++) rk[lane + 32 * b] = m[ka][b];
            __syncthreads();
            const T d = ck[k];
            const T p = d > eps * diag[k] ? T(1) / d : T(0);
            // column k takes -c p and row k takes r: zero the column, then r with p in its place
            T r[3];
#pragma unroll
            for (int b = 0; b < 3; b++) r[b] = rk[lane + 32 * b] * p;
            r[kb] = mycol ? p : r[kb];
#pragma unroll
            for (int a = 0; a < 6; a++) {
                const T c = ck[warp + 16 * a];
                m[a][kb] = mycol ? T(0) : m[a][kb];
#pragma unroll
                for (int b = 0; b < 3; b++) m[a][b] -= c * r[b];
            }
#pragma unroll
            for (int b = 0; b < 3; b++) m[ka][b] = myrow ? r[b] : m[ka][b];
        }
    }
#pragma unroll
    for (int a = 0; a < 6; a++)
#pragma unroll
        for (int b = 0; b < 3; b++) {
            const int i = warp + 16 * a, j = lane + 32 * b;
            if (i < n && j < n) inv[i * n + j] = m[a][b];
        }
}

// ------------------------------------------------------------------ the cycle
// One block: a system whose iteration fits one SM's L1 needs no grid barrier
// at all (about 3 us a phase), only __syncthreads.
struct BlockSync {
    static constexpr int kThreads = 1024, kBlocks = 1;
    __device__ __forceinline__ BlockSync(SolveState *, double *, long long) {}
    __device__ __forceinline__ bool barrier() {
        __syncthreads();
        return true;
    }
    template <int NV>
    __device__ __forceinline__ bool sum(double *v, double *sh) {
        block_sum<NV>(v, sh);
        return true;
    }
    template <int NV>
    __device__ __forceinline__ bool sumf(float *v, float *sh) {
        block_sum_f<NV>(v, sh);
        return true;
    }
};
struct MgGridSync : GridSync {
    static constexpr int kThreads = kMgT, kBlocks = 2;
    __device__ __forceinline__ MgGridSync(SolveState *st, double *part, long long spin) : GridSync{st, part, spin, 0} {}
};

// rows of a coarse operator over the grid
template <typename T, typename G, typename E>
__device__ __forceinline__ void mg_rows(int n, const int32_t *rp, const int32_t *ci, const T *v, int lanes, G gather,
                                        E epi) {
    const CsrSource<T> src{ci, v};
    if (sizeof(T) == 8 && lanes == 2) spmv_rows<2, 4, true, T>(n, rp, src, gather, epi);
    else if (lanes == 4) spmv_rows<4, 2, true, T>(n, rp, src, gather, epi);
    else if (lanes == 8) spmv_rows<8, 2, true, T>(n, rp, src, gather, epi);
    else spmv_rows<32, 4, false, T>(n, rp, src, gather, epi);
}

// r, y of a level from the one above it
template <typename T>
__device__ __forceinline__ void mg_down(const int32_t *rp, const int32_t *ci, const T *v, int lanes, const T *src,
                                        const MgLv<T> &to) {
    mg_rows(
        to.n, rp, ci, v, lanes, [&](int c) { return src[c]; },
        [&](int i, T s) {
            to.r[i] = s;
            to.y[i] = (T)kSmooth * to.D[i] * s;
        });
}

// e of a level: 2 y - w D A y, then + Q e of the next
template <typename T>
__device__ __forceinline__ void mg_up(const MgLv<T> &l, const T *enext) {
    mg_rows(
        l.n, l.rp, l.ci, l.v, l.lanes, [&](int c) { return ((const T *)l.y)[c]; },
        [&](int i, T s) { l.e[i] = T(2) * l.y[i] - (T)kSmooth * l.D[i] * s; });
    mg_rows(
        l.n, l.qrp, l.qci, l.qv, l.lanes, [&](int c) { return enext[c]; }, [&](int i, T s) { l.e[i] += s; });
}

// e of level 1 from r: restriction, the levels below, back up.  The caller
// has passed a barrier since r was written; returns after the barrier that
// follows e.  False: a barrier wait gave up.  Every block solves the bottom
// level for itself (its product with the dense inverse costs less than a
// barrier).
template <typename T, class SY>
__device__ __forceinline__ bool mg_cycle(const MgDev<T> &m, const T *r, T *eb, SY &sy) {
    mg_down(m.rrp, m.rci, m.rv, m.rlanes, r, m.lv[1]);
    if (!sy.barrier()) return false;
    const int bottom = m.nl - 1;
    for (int l = 1; l < bottom; l++) {
        mg_down(m.lv[l].trp, m.lv[l].tci, m.lv[l].tv, m.lv[l].tlanes, (const T *)m.lv[l].r, m.lv[l + 1]);
        if (!sy.barrier()) return false;
    }
    const MgLv<T> &b = m.lv[bottom];
    const T *enext = b.y;   // no dense inverse: the smoothing step
    if (m.dense) {
        T *rb = eb + kMgBottom;
        for (int i = threadIdx.x; i < b.n; i += blockDim.x) rb[i] = b.r[i];
        __syncthreads();
        const int lane = threadIdx.x & 3;
        const int pad = (b.n + 7) & ~7;   // whole warps take part in the shuffles
        for (int i = threadIdx.x >> 2; i < pad; i += blockDim.x >> 2) {
            T s = 0;
            if (i < b.n)
                for (int j = lane; j < b.n; j += 4) s += __ldg(m.binv + i * b.n + j) * rb[j];
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            if (i < b.n && lane == 0) eb[i] = s;
        }
        __syncthreads();
        enext = eb;
    }
    if (bottom == 1) {   // two levels: the fine level reads e from memory
        if (blockIdx.x == 0)
            for (int i = threadIdx.x; i < b.n; i += blockDim.x) b.e[i] = enext[i];
        return sy.barrier();
    }
    for (int l = bottom - 1; l >= 1; l--) {
        mg_up(m.lv[l], enext);
        enext = m.lv[l].e;
        if (!sy.barrier()) return false;
    }
    return true;
}

// z_i of the fine level
template <typename T>
__device__ __forceinline__ T mg_fine(const MgDev<T> &m, int i, T ri) {
    T z = (T)kSmooth * __ldg(m.D0 + i) * ri;
    if (m.ell) {
        const int2 c = __ldg(m.ell + i);
        const Pair<T> w = m.ellv[i];
        const T *e = m.lv[1].e;
        return z + (w.a * e[c.x] + w.b * e[c.y]);
    }
    const int e = __ldg(m.prp + i + 1);
    for (int q = __ldg(m.prp + i); q < e; q++) z += __ldg(m.pv + q) * m.lv[1].e[__ldg(m.pci + q)];
    return z;
}

// z = M^-1 r on the fine level after mg_cycle; epi(i, z_i) by the thread that
// owns row i.  Multiplicative: z = 2 S r - S A S r + Q e, as on the levels
// below (no barrier more: S r is formed where it is gathered).
template <typename T, typename E>
__device__ __forceinline__ void mg_fine_rows(const MgDev<T> &m, int n, const T *r, E epi) {
    if (!m.mult) {
        const int gtid = blockIdx.x * blockDim.x + threadIdx.x, gsz = gridDim.x * blockDim.x;
#pragma unroll 4
        for (int i = gtid; i < n; i += gsz) epi(i, mg_fine(m, i, r[i]));
        return;
    }
    const T *D0 = m.D0, *e1 = m.lv[1].e;
    T *z0 = m.z0;
    mg_rows(
        n, m.frp, m.fci, m.fv, m.flanes, [&](int c) { return (T)kSmooth * __ldg(D0 + c) * r[c]; },
        [&](int i, T s) {
            const T w = (T)kSmooth * __ldg(D0 + i);
            z0[i] = T(2) * w * r[i] - w * s;
        });
    mg_rows(
        n, m.q0rp, m.q0ci, m.q0v, m.flanes, [&](int c) { return e1[c]; }, [&](int i, T s) { epi(i, z0[i] + s); });
}

// ------------------------------------------------------------------ FP64 solver
template <int TPR, int U, bool PIPE, class SY>
__global__ void __launch_bounds__(SY::kThreads, SY::kBlocks)
    k_mgcg64(int n, const int32_t *rowptr, const int32_t *cols, const double *vals, const double *b, double *x, double *r,
             double *z, double *p, double *q, double *partial, SolveState *st, double abstol, double reltol, int maxit,
             int guess, long long spin, const __grid_constant__ MgDev<double> m) {
    __shared__ double sh[32 * 4];
    __shared__ double eb[2 * kMgBottom], rn0;
    SY sy(st, partial, spin);
    const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
    const int gsz = gridDim.x * blockDim.x;
    if (guess) spmv_grid<TPR, U, PIPE, double, double, double, false, true>(n, rowptr, cols, vals, x, r, nullptr, b);
    if (!sy.barrier()) return;
    double v[2] = {0, 0};
    for (int i = gtid; i < n; i += gsz) {
        const double ri = guess ? r[i] : b[i];
        if (!guess) {
            r[i] = ri;
            x[i] = 0.0;
        }
        p[i] = 0.0;
        v[0] += ri * ri;
        v[1] += b[i] * b[i];
    }
    if (!sy.template sum<2>(v, sh)) return;
    const double bn = sqrt(v[1]);
    const double tol = fmax(abstol, reltol * bn);
    if (threadIdx.x == 0) rn0 = sqrt(v[0]);
    int it = 0;
    bool conv = sqrt(v[0]) <= tol;
    double rz = 0.0;
    while (!conv && it < maxit) {
        if (!mg_cycle(m, (const double *)r, eb, sy)) return;
        double w[1] = {0};
        mg_fine_rows(m, n, (const double *)r, [&](int i, double zi) {
            z[i] = zi;
            w[0] += r[i] * zi;
        });
        if (!sy.template sum<1>(w, sh)) return;
        const double beta = it == 0 ? 0.0 : w[0] / rz;
        rz = w[0];
        for (int i = gtid; i < n; i += gsz) p[i] = z[i] + beta * p[i];
        if (!sy.barrier()) return;
        double d[1];
        d[0] = spmv_grid<TPR, U, PIPE, double, double, double, true, false>(n, rowptr, cols, vals, p, q, p, nullptr);
        if (!sy.template sum<1>(d, sh)) return;
        const double pq = d[0];
        if (!(pq > 0) || !isfinite(pq) || !isfinite(rz)) {
            if (gtid == 0) atomicCAS(&st->status, 0, (int)GRMP_ERR_NAN);
            break;
        }
        const double alpha = rz / pq;
        double rr[1] = {0};
        for (int i = gtid; i < n; i += gsz) {
            x[i] += alpha * p[i];
            const double ri = r[i] - alpha * q[i];
            r[i] = ri;
            rr[0] += ri * ri;
        }
        if (!sy.template sum<1>(rr, sh)) return;
        it++;
        conv = sqrt(rr[0]) <= tol;
        if (it % kStall64 == 0 && it > kStall64 && !conv && mg_behind(it, kStall64, sqrt(rr[0]), &rn0)) break;
    }
    if (!sy.barrier()) return;
    double t[1];
    t[0] = spmv_grid<TPR, U, PIPE, double, double, double, true, true>(n, rowptr, cols, vals, x, r, nullptr, b);
    if (!sy.template sum<1>(t, sh)) return;
    if (gtid == 0) {
        st->iters = it;
        st->outer = 0;
        st->nearer = sqrt(t[0]) < rn0;
        st->relres = sqrt(t[0]) / (bn > 0 ? bn : 1.0);
        if (st->status == 0 && !(sqrt(t[0]) <= fmax(tol, 0.0) || conv)) st->status = GRMP_ERR_NOT_CONVERGED;
    }
}

// ------------------------------------------------------------------ FP64 BiCGStab
// The scalar Jacobians of a Newton step (not symmetric): BiCGStab (van der
// Vorst 1992) preconditioned from the right by the same cycle, built from the
// Jacobian itself.  x is written only when the iteration has converged: the
// caller falls back to the Jacobi iteration from the same start otherwise.
// Bound like the other solvers by the latency of the cycle's phases, two
// cycles an iteration.  41^2 P2 Jacobian (6,889 rows, relres 1e-11): Jacobi
// 278-308 iterations, 11.9 ms; here 9 to 13 iterations, 0.87 to 1.10 ms.
template <int TPR, int U, bool PIPE, class SY>
__global__ void __launch_bounds__(SY::kThreads, SY::kBlocks)
    k_mgbicg64(int n, const int32_t *rowptr, const int32_t *cols, const double *vals, const double *b, double *x,
               double *xs, double *r, double *rh, double *p, double *v, double *s, double *t, double *ph, double *shv,
               double *partial, SolveState *st, double abstol, double reltol, int maxit, int guess, long long spin,
               const __grid_constant__ MgDev<double> m) {
    __shared__ double sh[32 * 4];
    __shared__ double eb[2 * kMgBottom];
    SY sy(st, partial, spin);
    const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
    const int gsz = gridDim.x * blockDim.x;
    if (guess) spmv_grid<TPR, U, PIPE, double, double, double, false, true>(n, rowptr, cols, vals, x, r, nullptr, b);
    if (!sy.barrier()) return;
    double w0[2] = {0, 0};
    for (int i = gtid; i < n; i += gsz) {
        const double ri = guess ? r[i] : b[i];
        r[i] = ri;
        xs[i] = guess ? x[i] : 0.0;
        rh[i] = ri;
        p[i] = ri;
        w0[0] += ri * ri;
        w0[1] += b[i] * b[i];
    }
    if (!sy.template sum<2>(w0, sh)) return;
    double rho = w0[0], rr = w0[0];
    const double rr0 = w0[0], bn = sqrt(w0[1]);
    const double tol = fmax(abstol, reltol * bn);
    int it = 0;
    bool conv = sqrt(rr) <= tol, bad = false;
    while (!conv && it < maxit) {
        if (!mg_cycle(m, (const double *)p, eb, sy)) return;
        mg_fine_rows(m, n, (const double *)p, [&](int i, double zi) { ph[i] = zi; });
        if (!sy.barrier()) return;
        double d[1];
        d[0] = spmv_grid<TPR, U, PIPE, double, double, double, true, false>(n, rowptr, cols, vals, ph, v, rh, nullptr);
        if (!sy.template sum<1>(d, sh)) return;
        bad = !(d[0] != 0.0) || !isfinite(d[0]);
        if (bad) break;
        const double alpha = rho / d[0];
        double ss[1] = {0};
        for (int i = gtid; i < n; i += gsz) {
            const double si = r[i] - alpha * v[i];
            s[i] = si;
            ss[0] += si * si;
        }
        if (!sy.template sum<1>(ss, sh)) return;
        if (sqrt(ss[0]) <= tol) {   // converged on the half step
            for (int i = gtid; i < n; i += gsz) xs[i] += alpha * ph[i];
            it++;
            conv = true;
            break;
        }
        if (!mg_cycle(m, (const double *)s, eb, sy)) return;
        mg_fine_rows(m, n, (const double *)s, [&](int i, double zi) { shv[i] = zi; });
        if (!sy.barrier()) return;
        double ts[2] = {0, 0};
        spmv_rows<TPR, U, PIPE, double>(
            n, rowptr, CsrSource<double>{cols, vals}, [&](int c) { return shv[c]; },
            [&](int row, double tv) {
                t[row] = tv;
                ts[0] += tv * s[row];
                ts[1] += tv * tv;
            });
        if (!sy.template sum<2>(ts, sh)) return;
        bad = !(ts[1] > 0.0) || !isfinite(ts[1]);
        if (bad) break;
        const double omega = ts[0] / ts[1];
        double w2[2] = {0, 0};
        for (int i = gtid; i < n; i += gsz) {
            xs[i] += alpha * ph[i] + omega * shv[i];
            const double ri = s[i] - omega * t[i];
            r[i] = ri;
            w2[0] += rh[i] * ri;
            w2[1] += ri * ri;
        }
        if (!sy.template sum<2>(w2, sh)) return;
        it++;
        rr = w2[1];
        conv = sqrt(rr) <= tol;
        bad = !conv && (!(w2[0] != 0.0) || !(omega != 0.0) || !isfinite(w2[1]));
        if (bad || (it == kStallBicg && rr > 0.01 * rr0)) break;   // not a digit: the cycle does not suit this matrix
        const double beta = (w2[0] / rho) * (alpha / omega);
        rho = w2[0];
        for (int i = gtid; i < n; i += gsz) p[i] = r[i] + beta * (p[i] - omega * v[i]);
        if (!sy.barrier()) return;
    }
    double tr = rr;
    if (conv) {   // all threads alike: the true residual, and x
        if (!sy.barrier()) return;
        double q[1];
        q[0] = spmv_grid<TPR, U, PIPE, double, double, double, true, true>(n, rowptr, cols, vals, xs, r, nullptr, b);
        if (!sy.template sum<1>(q, sh)) return;
        tr = q[0];
        for (int i = gtid; i < n; i += gsz) x[i] = xs[i];
    }
    if (gtid == 0) {
        st->iters = it;
        st->outer = 0;
        st->relres = sqrt(tr) / (bn > 0 ? bn : 1.0);
        if (st->status == 0 && !conv) st->status = bad ? GRMP_ERR_NAN : GRMP_ERR_NOT_CONVERGED;
    }
}

// ------------------------------------------------------------------ mixed solver
// FP32 conjugate gradients with the FP32 cycle inside the FP64 refinement
// loop of the Jacobi mixed solver (solve.cu): the FP32 correction is folded
// into x when the FP32 residual has fallen by `delta`, the FP64 residual
// replaces it, the direction is kept unless the true residual stopped falling.
template <int TPR, int U, bool PIPE, class SY>
__global__ void __launch_bounds__(SY::kThreads, SY::kBlocks)
    k_mgcg_mixed(int n, const int32_t *rowptr, const int32_t *cols, const double *vals64, const float *vals32,
                 const double *b, double *x, float *r, float *q, float *xc, float2 *zp0, float2 *zp1, double *r64,
                 double *partial, SolveState *st, double abstol, double reltol, double delta, int maxit, int maxouter,
                 int guess, long long spin, const __grid_constant__ MgDev<float> m) {
    __shared__ double sh[32 * 4];
    __shared__ float shf[32 * 4];
    __shared__ float eb[2 * kMgBottom];
    __shared__ double rn0;
    SY sy(st, partial, spin);
    const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
    const int gsz = gridDim.x * blockDim.x;
    double v[2] = {0, 0};
    if (guess) {
        v[0] = spmv_grid<TPR, U, PIPE, double, double, double, true, true>(n, rowptr, cols, vals64, x, r64, nullptr, b);
    } else {
        for (int i = gtid; i < n; i += gsz) {
            x[i] = 0.0;
            r64[i] = b[i];
            v[0] += b[i] * b[i];
        }
    }
    for (int i = gtid; i < n; i += gsz) v[1] += b[i] * b[i];
    if (!sy.template sum<2>(v, sh)) return;
    const double bn = sqrt(v[1]);
    const double tol = fmax(abstol, reltol * bn);
    double rn64 = sqrt(v[0]), prev_rn64 = rn64;
    if (threadIdx.x == 0) rn0 = rn64;
    // the FP32 system is solved for the residual scaled to norm 1: the
    // correction and its residual stay in FP32's range at any size of b
    double scale = rn64 > 0 ? rn64 : 1.0;
    for (int i = gtid; i < n; i += gsz) {
        r[i] = (float)(r64[i] / scale);
        zp0[i] = make_float2(0.f, 0.f);
        xc[i] = 0.f;
    }
    if (!sy.barrier()) return;
    int it = 0, outer = 0, stall = 0;
    bool conv = rn64 <= tol;
    float rz = 0.f, rmax = 1.f;
    bool restart = true;
    float2 *cur = zp0, *nxt = zp1;
    float rn32 = 1.f;
    while (!conv && it < maxit && outer < maxouter) {
        do {   // to the next look at the progress: out of the iterations' way (46^3 P2 6.64 ms with it among them, 6.53 now)
            if (!mg_cycle(m, (const float *)r, eb, sy)) return;
            float w[1] = {0.f};
            mg_fine_rows(m, n, (const float *)r, [&](int i, float zi) {
                cur[i].x = zi;
                w[0] += r[i] * zi;
            });
            if (!sy.template sumf<1>(w, shf)) return;
            const float beta = restart ? 0.f : w[0] / rz;
            rz = w[0];
            // q = A p with p = z + beta p formed while gathering; the owner of a row stores p
            float dot = 0.f;
            spmv_rows<TPR, U, PIPE, float>(
                n, rowptr, CsrSource<float>{cols, vals32},
                [&](int c) {
                    const float2 e = cur[c];
                    return fmaf(beta, e.y, e.x);
                },
                [&](int i, float s) {
                    const float2 e = cur[i];
                    const float pi = fmaf(beta, e.y, e.x);
                    nxt[i].y = pi;
                    q[i] = s;
                    dot += pi * s;
                });
            float d[1] = {dot};
            if (!sy.template sumf<1>(d, shf)) return;
            const float pq = d[0];
            if (!(pq > 0.f) || !isfinite(pq) || !isfinite(rz)) {
                if (gtid == 0) atomicCAS(&st->status, 0, (int)GRMP_ERR_NAN);
                goto done;
            }
            const float alpha = rz / pq;
            float u[1] = {0.f};
            {   // four rows a thread, 16-byte accesses
                float4 *xc4 = reinterpret_cast<float4 *>(xc), *r4 = reinterpret_cast<float4 *>(r);
                const float4 *q4 = reinterpret_cast<const float4 *>(q), *nx4 = reinterpret_cast<const float4 *>(nxt);
                const int n4 = n >> 2;
                for (int i = gtid; i < n4; i += gsz) {
                    const float4 a = nx4[2 * i], c = nx4[2 * i + 1], qq = q4[i];
                    float4 rr = r4[i], xx = xc4[i];
                    xx.x += alpha * a.y;
                    xx.y += alpha * a.w;
                    xx.z += alpha * c.y;
                    xx.w += alpha * c.w;
                    rr.x -= alpha * qq.x;
                    rr.y -= alpha * qq.y;
                    rr.z -= alpha * qq.z;
                    rr.w -= alpha * qq.w;
                    xc4[i] = xx;
                    r4[i] = rr;
                    u[0] += rr.x * rr.x + rr.y * rr.y + rr.z * rr.z + rr.w * rr.w;
                }
                for (int i = 4 * n4 + gtid; i < n; i += gsz) {
                    xc[i] += alpha * nxt[i].y;
                    const float ri = r[i] - alpha * q[i];
                    r[i] = ri;
                    u[0] += ri * ri;
                }
            }
            if (!sy.template sumf<1>(u, shf)) return;
            it++;
            rn32 = sqrtf(u[0]);
            restart = false;
            if (rn32 <= (float)delta * rmax || (double)rn32 * scale <= tol || it >= maxit) {
                for (int i = gtid; i < n; i += gsz) {
                    x[i] += (double)xc[i] * scale;
                    xc[i] = 0.f;
                }
                if (!sy.barrier()) return;
                double t[1];
                t[0] = spmv_grid<TPR, U, PIPE, double, double, double, true, true>(n, rowptr, cols, vals64, x, r64, nullptr, b);
                if (!sy.template sum<1>(t, sh)) return;
                outer++;
                rn64 = sqrt(t[0]);
                conv = rn64 <= tol;
                if (conv || it >= maxit) goto done;
                restart = rn64 > 0.5 * prev_rn64;
                stall = (rn64 > 0.9 * prev_rn64) ? stall + 1 : 0;
                prev_rn64 = rn64;
                if (stall >= 16) goto done;
                // rescale: directions and rz are of the old scale
                const float f = (float)(scale / rn64);
                scale = rn64;
                rz *= f * f;
                for (int i = gtid; i < n; i += gsz) {
                    r[i] = (float)(r64[i] / scale);
                    nxt[i].y *= f;
                }
                rmax = rn32 = 1.f;
                if (!sy.barrier()) return;
            }
            float2 *tmp = cur;
            cur = nxt;
            nxt = tmp;
        } while (it % kStall32 != 0 && it < maxit && outer < maxouter);
        if (it % kStall32 == 0 && it > kStall32 && mg_behind(it, kStall32, (double)rn32 * scale, &rn0))
            break;   // x: as of the last refinement
    }
done:
    if (gtid == 0) {
        st->iters = it;
        st->outer = outer;
        st->nearer = rn64 < rn0;
        st->relres = rn64 / (bn > 0 ? bn : 1.0);
        if (st->status == 0 && !conv) st->status = GRMP_ERR_NOT_CONVERGED;
    }
}

}  // namespace

// ---------------------------------------------------------------------- host side
struct MgCache {
    MgSymbolic S;
    bool mult = false;   // multiplicative smoothing of the fine level
    std::vector<std::pair<void *, size_t>> bufs;   // patterns
    struct Step {
        int32_t *agg = nullptr, *vrow = nullptr;
        int2 *ell = nullptr;
        int32_t *prp, *pci, *rrp, *rci, *rperm, *arp, *aci, *trp = nullptr, *tci = nullptr, *tperm = nullptr, *crp, *cci;
        size_t np, na, nt, nc;   // entries of P, A P, Q^T, next A
        int longa, longc;        // longest rows of A P and the next A
    };
    std::vector<Step> step;
    // numeric storage per precision (0: FP64, 1: FP32), one allocation each
    struct Num {
        void *p = nullptr;
        size_t bytes = 0;
        std::vector<char *> pv, av, tv, cv, D, iso, r, y, e;
        char *rv0 = nullptr, *ellv = nullptr, *binv = nullptr, *part = nullptr, *vec = nullptr, *z0 = nullptr, *x0 = nullptr;
    } num[2];
};

namespace {

inline size_t al(size_t v) { return (v + 255) & ~(size_t)255; }

template <typename V>
int mg_up_vec(grmp_context ctx, MgCache &C, const std::vector<V> &v, V **out) {
    const size_t bytes = std::max<size_t>(1, v.size()) * sizeof(V);
    void *p = nullptr;
    int rc = grmp_alloc_spare(ctx, &p, bytes);
    if (rc) return rc;
    C.bufs.push_back({p, bytes});
    *out = (V *)p;
    if (v.empty()) return GRMP_OK;
    cudaError_t e = cudaMemcpyAsync(p, v.data(), v.size() * sizeof(V), cudaMemcpyHostToDevice, ctx->stream);
    return e == cudaSuccess ? GRMP_OK : grmp_cuda_fail(ctx, e, "multilevel patterns");
}

// Whether more than a twentieth of the mesh's cells are stretched: the
// aggregates then follow strong couplings, for which the host forms the unit
// stiffness of every level (first solve of a pattern: 160 x 160 P1 9 ms instead of
// 4, 40^3 P1 32 to 47 instead of 13, 20^3 P2 62 to 77 instead of 15).
int mg_stretched(grmp_mesh m, bool *out) {
    grmp_context ctx = m->ctx;
    int *cnt = nullptr, h = 0;
    int rc = grmp_alloc_spare(ctx, (void **)&cnt, 4);
    if (rc) return rc;
    cudaMemsetAsync(cnt, 0, 4, ctx->stream);
    if (m->dim == 2) k_mg_stretched<2><<<nblk(m->ncells), 256, 0, ctx->stream>>>(m->ncells, m->d_coords, m->d_cells, cnt);
    else k_mg_stretched<3><<<nblk(m->ncells), 256, 0, ctx->stream>>>(m->ncells, m->d_coords, m->d_cells, cnt);
    GRMP_LAUNCHED(ctx);
    cudaError_t e = grmp_readback(ctx, &h, cnt, 4);
    grmp_free(ctx, cnt, 4);
    if (e != cudaSuccess) return grmp_cuda_fail(ctx, e, "multilevel: cells");
    *out = h > m->ncells / 20;
    return GRMP_OK;
}

// the probe's flag and per-block sums
constexpr int kProbeBlocks = 2048;
constexpr size_t kProbePart = (size_t)(kProbeBlocks + 1) * 16;

// numeric storage of one precision: values of every level, vectors, state.
// Its bytes; base: where it lies (nullptr: only the bytes)
template <typename T>
size_t mg_layout(grmp_matrix A, MgCache &C, char *base) {
    MgCache::Num &N = C.num[sizeof(T) == 8 ? 0 : 1];
    const int ns = (int)C.step.size();
    size_t at = 0;
    auto take = [&](size_t bytes) -> char * {
        const size_t o = at;
        at += al(bytes);
        return base ? base + o : nullptr;
    };
    N.pv.assign(ns, nullptr);
    N.av = N.tv = N.cv = N.pv;
    N.D.assign(ns + 1, nullptr);
    N.iso = N.r = N.y = N.e = N.D;
    for (int k = 0; k < ns; k++) {
        const MgCache::Step &d = C.step[k];
        N.pv[k] = take(d.np * sizeof(T));
        N.av[k] = take(d.na * sizeof(T));
        N.cv[k] = take(d.nc * sizeof(T));
        N.tv[k] = take(d.nt * sizeof(T));
    }
    N.rv0 = take(C.step[0].np * sizeof(T));
    N.ellv = take(C.S.step[0].geometric ? (size_t)A->nrows * 2 * sizeof(T) : 0);
    for (int k = 0; k <= ns; k++) {
        const size_t n = k < ns ? C.S.step[k].n : C.S.step[ns - 1].nc;
        N.D[k] = take(n * sizeof(T));
        N.iso[k] = take(n);
        if (k > 0) {
            N.r[k] = take(n * sizeof(T));
            N.y[k] = take(n * sizeof(T));
            N.e[k] = take(n * sizeof(T));
        }
    }
    N.z0 = take(C.mult ? (size_t)A->nrows * sizeof(T) : 0);
    N.binv = take((size_t)kMgBottom * kMgBottom * sizeof(T));
    N.part = take(kProbePart);
    // FP64: r z p q; mixed: r q xc, two pairs, FP64 residual
    const size_t n0 = A->nrows;
    N.vec = take(sizeof(T) == 8 ? 4 * al(n0 * 8) : 3 * al(n0 * 4) + 2 * al(n0 * 8) + al(n0 * 8));
    N.x0 = take(n0 * 8);   // the caller's start, while it may be needed again (last: between the others it cost 16^2 P2 mixed 5 %)
    return at + al((size_t)2 * kPartStride * 8) + al(sizeof(SolveState));
}

size_t mg_need(grmp_matrix A, MgCache &C, bool mixed) {
    return mixed ? mg_layout<float>(A, C, nullptr) : mg_layout<double>(A, C, nullptr);
}

// The patterns, on the device.  GRMP_ERR_BUDGET before anything is taken if they
// and the storage of this precision do not fit; A->mg_state = -1 if the matrix
// does not coarsen.
int mg_build(grmp_matrix A, bool mixed, MgCache *C) {
    grmp_space s = A->space;
    grmp_context ctx = s->mesh->ctx;
    const int n = A->nrows;
    const bool p2 = s->fe == GRMP_FE_H1P2;
    bool stretched = false;
    int rc = mg_stretched(s->mesh, &stretched);
    if (rc) return rc;
    MgCsr pattern;
    std::vector<int32_t> cd, cells;
    std::vector<double> coords;
    pattern.rp.resize((size_t)n + 1);
    pattern.ci.resize((size_t)A->nnz);
    cudaError_t e = cudaMemcpyAsync(pattern.rp.data(), A->d_rowptr, pattern.rp.size() * 4, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(pattern.ci.data(), A->d_cols, pattern.ci.size() * 4, cudaMemcpyDeviceToHost, ctx->stream);
    if (p2 || stretched) {
        cd.resize((size_t)s->mesh->ncells * s->ldofs);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(cd.data(), s->d_celldofs, cd.size() * 4, cudaMemcpyDeviceToHost, ctx->stream);
        cells.resize((size_t)s->mesh->ncells * (s->mesh->dim + 1));
        coords.resize((size_t)s->mesh->nverts * s->mesh->dim);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(cells.data(), s->mesh->d_cells, cells.size() * 4, cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(coords.data(), s->mesh->d_coords, coords.size() * 8, cudaMemcpyDeviceToHost, ctx->stream);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return grmp_cuda_fail(ctx, e, "multilevel: pattern download");
    C->mult = fine_mult(s->mesh->dim, s->fe, n);
    const MgCells m{s->mesh->dim, s->mesh->ncells, s->ldofs, cd.data(), cells.data(), coords.data()};
    if (mg_symbolic_build(n, pattern, m, p2, !A->face_coupled, stretched, C->mult, &C->S)) {
        A->mg_state = -1;
        return GRMP_OK;
    }
    const int ns = (int)C->S.step.size();
    C->step.resize(ns);
    size_t need = 0;
    for (int k = 0; k < ns; k++) {
        const MgStep &t = C->S.step[k];
        MgCache::Step &d = C->step[k];
        d.np = t.P.ci.size();
        d.na = t.AP.ci.size();
        d.nt = t.QT.ci.size();
        d.nc = t.Ac.ci.size();
        auto longest = [](const std::vector<int32_t> &r) {
            int l = 0;
            for (size_t i = 1; i < r.size(); i++) l = std::max(l, r[i] - r[i - 1]);
            return l;
        };
        d.longa = longest(t.AP.rp);
        d.longc = longest(t.Ac.rp);
        for (const MgCsr *x : {&t.P, &t.R, &t.AP, &t.QT, &t.Ac}) need += (x->rp.size() + x->ci.size()) * 4;
        need += (t.Rperm.size() + t.QTperm.size() + t.agg.size()) * 4 + (t.geometric ? (size_t)t.nc * 4 + (size_t)t.n * 8 : 0);
    }
    need += mg_need(A, *C, mixed);
    A->mg_floor[mixed] = need > A->mg_budget ? SIZE_MAX : need;
    if (need > A->mg_budget || (ctx->budget && need > ctx->budget - std::min(ctx->budget, ctx->in_use.load()))) return GRMP_ERR_BUDGET;
    for (int k = 0; k < ns && !rc; k++) {
        MgStep &t = C->S.step[k];
        MgCache::Step &d = C->step[k];
        auto up = [&](std::vector<int32_t> &v, int32_t **p) {
            if (!rc) rc = mg_up_vec(ctx, *C, v, p);
        };
        std::vector<int32_t> vrow;
        std::vector<int2> ell;
        if (t.geometric) {
            vrow.resize(t.nc);
            for (int i = 0; i < t.n; i++)
                if (t.P.rp[i + 1] - t.P.rp[i] == 1) vrow[t.P.ci[t.P.rp[i]]] = i;
            up(vrow, &d.vrow);
            ell.resize(t.n);
            for (int i = 0; i < t.n; i++) ell[i] = make_int2(t.P.ci[t.P.rp[i]], t.P.ci[t.P.rp[i + 1] - 1]);
            if (!rc) rc = mg_up_vec(ctx, *C, ell, &d.ell);
        } else {
            up(t.agg, &d.agg);
        }
        up(t.P.rp, &d.prp);
        up(t.P.ci, &d.pci);
        up(t.R.rp, &d.rrp);
        up(t.R.ci, &d.rci);
        up(t.Rperm, &d.rperm);
        up(t.AP.rp, &d.arp);
        up(t.AP.ci, &d.aci);
        up(t.Ac.rp, &d.crp);
        up(t.Ac.ci, &d.cci);
        if (k > 0 || C->mult) {
            up(t.QT.rp, &d.trp);
            up(t.QT.ci, &d.tci);
            up(t.QTperm, &d.tperm);
        }
        if (cudaStreamSynchronize(ctx->stream) != cudaSuccess && !rc) rc = GRMP_ERR_DEVICE;
        t.P = t.R = t.AP = t.QT = t.Ac = MgCsr();   // the sizes stay
        t.Rperm = t.QTperm = t.agg = std::vector<int32_t>();
    }
    if (!rc) A->mg_state = 1;
    return rc;
}

size_t mg_bytes(const MgCache &C) {
    size_t b = 0;
    for (auto &x : C.bufs) b += x.second;
    return b;
}

// whether there is still less room than this precision needs (the other one's storage counts as room)
bool mg_no_room(grmp_matrix A, bool mixed) {
    grmp_context ctx = A->space->mesh->ctx;
    const size_t floor = A->mg_floor[mixed], other = A->mg ? A->mg->num[!mixed].bytes : 0;
    if (floor == 0 || floor == SIZE_MAX) return floor > 0;
    if (ctx->budget && ctx->in_use - other + floor > ctx->budget) return true;
    return grmp_room(ctx) + other < floor;
}

// The hierarchy with storage of this precision.  *fits = false: there is no
// room for it now; the patterns and the other precision's storage then stay if
// that is in use.  Of two precisions that do not fit together the one asked for
// has the room, whatever was solved before.
int mg_make(grmp_matrix A, bool mixed, bool *fits) {
    grmp_context ctx = A->space->mesh->ctx;
    *fits = false;
    int rc = GRMP_OK;
    if (!A->mg) {
        std::unique_ptr<MgCache> C;
        try {
            C.reset(new MgCache);
            rc = mg_build(A, mixed, C.get());
        } catch (const std::exception &) {   // host memory: solved without the hierarchy, as when the device's is short
            cudaStreamSynchronize(ctx->stream);
            rc = GRMP_ERR_OUT_OF_MEMORY;
        }
        if (!rc && A->mg_state > 0) {
            A->mg = C.release();
            ctx->hier.push_back(A);
        } else if (C) {
            for (auto &b : C->bufs) grmp_free(ctx, b.first, b.second);
        }
    }
    if (!rc && A->mg_state < 0) return GRMP_OK;
    if (!rc) {
        MgCache &C = *A->mg;
        MgCache::Num &N = C.num[mixed], &O = C.num[!mixed];
        const size_t need = mg_need(A, C, mixed), pat = mg_bytes(C);
        A->mg_floor[mixed] = pat + need > A->mg_budget ? SIZE_MAX : need;
        rc = GRMP_ERR_BUDGET;
        if (pat + need + O.bytes <= A->mg_budget) rc = grmp_alloc_spare(ctx, &N.p, need);
        if ((rc == GRMP_ERR_BUDGET || rc == GRMP_ERR_OUT_OF_MEMORY) && O.p && pat + need <= A->mg_budget &&
            (!ctx->budget || ctx->in_use - O.bytes + need <= ctx->budget)) {
            cudaGetLastError();
            grmp_free(ctx, O.p, O.bytes);
            O.p = nullptr;
            O.bytes = 0;
            rc = grmp_alloc_spare(ctx, &N.p, need);
        }
        if (!rc) {
            N.bytes = need;
            mixed ? mg_layout<float>(A, C, (char *)N.p) : mg_layout<double>(A, C, (char *)N.p);
        } else if (!O.p) {   // patterns alone are of no use
            if (A->mg_floor[mixed] != SIZE_MAX) A->mg_floor[mixed] += pat;
            grmp_mg_free(A);
        }
    }
    if (rc == GRMP_ERR_BUDGET || rc == GRMP_ERR_OUT_OF_MEMORY) {
        ctx->last_error.clear();
        cudaGetLastError();
        return GRMP_OK;
    }
    if (rc) return rc;
    A->mg_floor[mixed] = 0;
    *fits = true;
    return GRMP_OK;
}

template <typename T>
const T *fine_values(grmp_matrix A);
template <>
const double *fine_values<double>(grmp_matrix A) { return A->d_vals64; }
template <>
const float *fine_values<float>(grmp_matrix A) { return A->d_vals32; }

// lanes per row of k_mg_rows (FP64: as in lanes_of)
template <typename T>
int rows_lanes(int n) { return sizeof(T) == 8 && n >= kManyRows ? 2 : 8; }

// D of the fine level, the diagonal check and the reaction share
template <typename T>
int mg_probe(grmp_matrix A, char *D, char *iso, char *part, double *react) {
    grmp_context ctx = A->space->mesh->ctx;
    const int n = A->nrows, cl = rows_lanes<T>(n);
    const int grid = std::max(1, std::min({nblk(n, kTB / cl), 4 * ctx->num_sms, kProbeBlocks}));
    cudaMemsetAsync(part, 0, 16, ctx->stream);   // the flag of a bad diagonal, then the blocks' sums
    auto kern = cl == 2 ? k_mg_rows<T, 2> : k_mg_rows<T, 8>;
    kern<<<grid, kTB, 0, ctx->stream>>>(n, A->d_rowptr, A->d_cols, fine_values<T>(A), (T *)D, (uint8_t *)iso,
                                        A->eliminated ? A->d_fixed : nullptr, (double2 *)part + 1, (int *)part);
    GRMP_LAUNCHED(ctx);
    double buf[2 * (kProbeBlocks + 1)];
    cudaError_t e = grmp_readback(ctx, buf, part, (size_t)(grid + 1) * 16);
    const double *h = buf + 2;
    int bad = 0;
    std::memcpy(&bad, buf, 4);
    if (e != cudaSuccess) return grmp_cuda_fail(ctx, e, "multilevel: diagonal");
    if (bad) return grmp_fail(ctx, GRMP_ERR_INVALID_ARG, "solve: non-positive or non-finite diagonal entry");
    double s = 0, d = 0;
    for (int b = 0; b < grid; b++) s += h[2 * b], d += h[2 * b + 1];
    *react = d > 0 ? s / d : 1.0;
    return GRMP_OK;
}

// the probe before there is a hierarchy, in memory of its own
template <typename T>
int mg_probe_first(grmp_matrix A, double *react) {
    grmp_context ctx = A->space->mesh->ctx;
    const size_t d = al((size_t)A->nrows * sizeof(T)), i = al((size_t)A->nrows), bytes = d + i + kProbePart;
    char *w = nullptr;
    int rc = grmp_alloc_spare(ctx, (void **)&w, bytes);
    if (rc) return rc;
    rc = mg_probe<T>(A, w, w + d, w + d + i, react);
    grmp_free(ctx, w, bytes);
    return rc;
}

// levels of at most kShortLevel rows give a row 16 lanes (k_mg_prol_agg) or a
// block; a row of a product with at most kWideCap columns fits the accumulators
// of k_mg_wide (kWideG x 700 x 8 bytes = 179 KB)
constexpr int kShortLevel = 4096, kWideCap = 700;
template <typename T, bool RAP>
size_t mg_wide_smem(int longest) {
    const size_t b = (size_t)kWideG * longest * sizeof(T) + (size_t)longest * 4;
    grmp_allow_smem(k_mg_wide<T, RAP>);
    return b;
}

template <typename T>
void mg_values(grmp_matrix A) {
    grmp_context ctx = A->space->mesh->ctx;
    cudaStream_t st = ctx->stream;
    MgCache &C = *A->mg;
    MgCache::Num &N = C.num[sizeof(T) == 8 ? 0 : 1];
    const int ns = (int)C.step.size();
    const int32_t *rp = A->d_rowptr, *ci = A->d_cols;
    const T *v = fine_values<T>(A);
    const int wide = 8 * ctx->num_sms;
    for (int k = 0; k < ns; k++) {
        const MgCache::Step &d = C.step[k];
        const int n = C.S.step[k].n, nc = C.S.step[k].nc;
        T *pv = (T *)N.pv[k], *av = (T *)N.av[k], *cv = (T *)N.cv[k], *D = (T *)N.D[k];
        if (k > 0) {
            const int cl = rows_lanes<T>(n);
            auto kern = cl == 2 ? k_mg_rows<T, 2> : k_mg_rows<T, 8>;
            kern<<<std::max(1, std::min(nblk(n, kTB / cl), wide)), kTB, 0, st>>>(
                n, rp, ci, v, D, (uint8_t *)N.iso[k], nullptr, nullptr, nullptr);
            GRMP_LAUNCHED(ctx);
        }
        if (d.vrow)
            k_mg_prol_geo<T><<<nblk(n), 256, 0, st>>>(n, d.prp, d.pci, d.vrow, (const uint8_t *)N.iso[k], pv,
                                                        (Pair<T> *)N.ellv);
        else if (n > kShortLevel)
            k_mg_prol_agg<T, 1><<<nblk(n, 128), 128, 0, st>>>(n, rp, ci, v, D, (const uint8_t *)N.iso[k], d.agg, d.prp,
                                                              d.pci, pv);
        else
            k_mg_prol_agg<T, 16><<<nblk((long long)n * 16, 128), 128, 0, st>>>(n, rp, ci, v, D, (const uint8_t *)N.iso[k],
                                                                               d.agg, d.prp, d.pci, pv);
        if (C.S.step[k].lump) {
            k_mg_prol_lump<T><<<nblk((long long)n * 8, 256), 256, 0, st>>>(n, rp, ci, v, D, (const uint8_t *)N.iso[k], d.agg,
                                                                          d.prp, d.pci, pv);
            GRMP_LAUNCHED(ctx);
        }
        if (d.vrow)
            k_mg_ap_geo<T><<<std::max(1, std::min(nblk((long long)n * 16), wide)), kTB, 0, st>>>(
                n, rp, ci, v, d.ell, (const Pair<T> *)N.ellv, d.arp, d.aci, av);
        else if (n <= kShortLevel && d.longa <= kWideCap)
            k_mg_wide<T, false><<<n, kTB, mg_wide_smem<T, false>(d.longa), st>>>(rp, ci, nullptr, v, d.prp, d.pci, pv,
                                                                                 d.arp, d.aci, av);
        else
            k_mg_ap<T><<<std::max(1, std::min(nblk((long long)n * 8), wide)), kTB, 0, st>>>(n, rp, ci, v, d.prp, d.pci,
                                                                                           pv, d.arp, d.aci, av);
        if (nc <= kShortLevel && d.longc <= kWideCap)
            k_mg_wide<T, true><<<nc, kTB, mg_wide_smem<T, true>(d.longc), st>>>(d.rrp, d.rci, d.rperm, pv, d.arp, d.aci, av,
                                                                                d.crp, d.cci, cv);
        else
            k_mg_rap<T><<<std::max(1, std::min(nblk((long long)nc * 16), wide)), kTB, 0, st>>>(
                nc, d.rrp, d.rci, d.rperm, pv, d.arp, d.aci, av, d.crp, d.cci, cv);
        ctx->launches += 3;
        if (k > 0 || C.mult) {
            k_mg_q<T><<<nblk(n, 128), 128, 0, st>>>(n, d.prp, d.pci, pv, d.arp, d.aci, D, av);
            k_mg_perm<T><<<nblk((long long)d.nt), 256, 0, st>>>((int)d.nt, d.tperm, av, (T *)N.tv[k]);
            ctx->launches += 2;
        } else {
            k_mg_perm<T><<<nblk((long long)d.np), 256, 0, st>>>((int)d.np, d.rperm, pv, (T *)N.rv0);
            GRMP_LAUNCHED(ctx);
        }
        rp = d.crp;
        ci = d.cci;
        v = cv;
    }
    const int nb = C.S.step[ns - 1].nc;
    k_mg_rows<T, 8><<<std::max(1, std::min(nblk(nb, kTB / 8), wide)), kTB, 0, st>>>(
        nb, rp, ci, v, (T *)N.D[ns], (uint8_t *)N.iso[ns], nullptr, nullptr, nullptr);
    GRMP_LAUNCHED(ctx);
    if (nb <= kMgBottom) {
        const size_t smem = (size_t)nb * nb * sizeof(T);
        grmp_allow_smem(k_mg_binv<T>);
        k_mg_binv<T><<<1, 512, smem, st>>>(nb, rp, ci, v, (T *)N.binv);
        GRMP_LAUNCHED(ctx);
    }
}

template <typename T>
MgDev<T> mg_device(grmp_matrix A) {
    MgCache &C = *A->mg;
    MgCache::Num &N = C.num[sizeof(T) == 8 ? 0 : 1];
    const int ns = (int)C.step.size();
    MgDev<T> m;
    std::memset(&m, 0, sizeof(m));
    m.nl = ns + 1;
    m.prp = C.step[0].prp;
    m.pci = C.step[0].pci;
    m.pv = (const T *)N.pv[0];
    m.rrp = C.step[0].rrp;
    m.rci = C.step[0].rci;
    m.rv = (const T *)N.rv0;
    m.ell = C.step[0].ell;
    m.ellv = (const Pair<T> *)N.ellv;
    m.D0 = (const T *)N.D[0];
    m.binv = (const T *)N.binv;
    m.dense = C.S.step[ns - 1].nc <= kMgBottom;
    auto lanes = lanes_of<T>;
    m.rlanes = lanes(C.step[0].np, C.S.step[0].nc);
    m.mult = C.mult;
    if (C.mult) {
        const MgCache::Step &d = C.step[0];
        m.rrp = d.trp;
        m.rci = d.tci;
        m.rv = (const T *)N.tv[0];
        m.rlanes = lanes(d.nt, C.S.step[0].nc);
        m.frp = A->d_rowptr;
        m.fci = A->d_cols;
        m.fv = fine_values<T>(A);
        m.q0rp = d.arp;
        m.q0ci = d.aci;
        m.q0v = (const T *)N.av[0];
        m.flanes = lanes(std::max((size_t)A->nnz, d.na), A->nrows);
        m.z0 = (T *)N.z0;
    }
    for (int l = 1; l <= ns; l++) {
        MgLv<T> &L = m.lv[l];
        L.n = C.S.step[l - 1].nc;
        L.rp = C.step[l - 1].crp;
        L.ci = C.step[l - 1].cci;
        L.v = (const T *)N.cv[l - 1];
        L.D = (const T *)N.D[l];
        if (l < ns) {
            L.lanes = lanes(std::max(C.step[l - 1].nc, C.step[l].na), L.n);
            L.tlanes = lanes(C.step[l].nt, C.S.step[l].nc);
            L.qrp = C.step[l].arp;
            L.qci = C.step[l].aci;
            L.qv = (const T *)N.av[l];
            L.trp = C.step[l].trp;
            L.tci = C.step[l].tci;
            L.tv = (const T *)N.tv[l];
        }
        L.r = (T *)N.r[l];
        L.y = (T *)N.y[l];
        L.e = (T *)N.e[l];
    }
    return m;
}

// Systems of at most this many nonzeros run in one block (its L1 holds matrix
// and vectors; on the FP64 pipe of one SM, two FMAs a clock, only the smallest
// gain).  One block / the grid, whole passes, lognormal, ms: mixed 2D P2 289
// rows 0.47 / 0.71, 1,681 rows (19 k nonzeros) 0.88 / 0.88, 2D P1 3,249 rows
// (22 k) 1.23 / 1.00, 3D P1 1,000 rows (13 k) 0.60 / 0.68; FP64 2D P1 441 rows
// (3 k) 1.13 / 1.14, 2D P2 441 rows (5 k) 1.06 / 1.05.
constexpr int kOneBlock32 = 18000, kOneBlock64 = 4000;

// grid: enough blocks for the rows, at most what fits; small systems take
// one block per SM, which makes the barriers cheaper
template <typename K>
int mg_grid(grmp_context ctx, K kern, int n, int tpr, int want) {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kMgT, 0);
    const int maxg = std::max(1, per_sm) * ctx->num_sms;
    if (want > 0) return std::min(want, maxg);
    const int need = std::max(1, nblk((long long)n * tpr, kMgT));
    const int cap = n <= 150000 ? ctx->num_sms : maxg;
    return std::min({need, cap, maxg});
}

template <typename K>
cudaError_t mg_start(grmp_context ctx, K kern, bool one, int n, int tpr, int want, void **args, int *grid) {
    *grid = one ? 1 : mg_grid(ctx, kern, n, tpr, want);
    GRMP_LAUNCHED(ctx);
    if (one) return cudaLaunchKernel((const void *)kern, dim3(1), dim3(BlockSync::kThreads), args, 0, ctx->stream);
    return cudaLaunchCooperativeKernel((const void *)kern, dim3(*grid), dim3(kMgT), args, 0, ctx->stream);
}

template <int TPR, int U, bool PIPE>
int mg_launch(grmp_matrix A, const double *b, double *x, const grmp_solve_params *p, bool mixed, int *grid) {
    grmp_context ctx = A->space->mesh->ctx;
    MgCache::Num &N = A->mg->num[mixed ? 1 : 0];
    const size_t n0 = A->nrows;
    char *part = (char *)N.p + N.bytes - al(sizeof(SolveState)) - al((size_t)2 * kPartStride * 8);
    SolveState *dst = (SolveState *)((char *)N.p + N.bytes - al(sizeof(SolveState)));
    double *partial = (double *)part;
    int n = A->nrows, mi = p->maxiter, guess = p->use_initial_guess ? 1 : 0;
    double at = p->abstol, rt = p->reltol;
    const int32_t *rp = A->d_rowptr, *ci = A->d_cols;
    const double *v64 = A->d_vals64;
    long long spin = ctx->wait_limit;
    cudaMemsetAsync(dst, 0, sizeof(SolveState), ctx->stream);
    cudaError_t e;
    if (!mixed) {
        const bool one = A->nnz <= kOneBlock64 && p->grid_blocks <= 0;
        auto kern = one ? k_mgcg64<TPR, U, PIPE, BlockSync> : k_mgcg64<TPR, U, PIPE, MgGridSync>;
        MgDev<double> m = mg_device<double>(A);
        double *r = (double *)N.vec, *z = (double *)(N.vec + al(n0 * 8)), *pp = (double *)(N.vec + 2 * al(n0 * 8));
        double *q = (double *)(N.vec + 3 * al(n0 * 8));
        void *args[] = {&n, &rp, &ci, &v64, &b, &x, &r, &z, &pp, &q, &partial, &dst, &at, &rt, &mi, &guess, &spin, &m};
        e = mg_start(ctx, kern, one, n, TPR, p->grid_blocks, args, grid);
    } else {
        const bool one = A->nnz <= kOneBlock32 && p->grid_blocks <= 0;
        auto kern = one ? k_mgcg_mixed<TPR, U, PIPE, BlockSync> : k_mgcg_mixed<TPR, U, PIPE, MgGridSync>;
        MgDev<float> m = mg_device<float>(A);
        const float *v32 = A->d_vals32;
        float *r = (float *)N.vec, *q = (float *)(N.vec + al(n0 * 4)), *xc = (float *)(N.vec + 2 * al(n0 * 4));
        char *w = N.vec + 3 * al(n0 * 4);
        float2 *zp0 = (float2 *)w, *zp1 = (float2 *)(w + al(n0 * 8));
        double *r64 = (double *)(w + 2 * al(n0 * 8));
        int mo = p->max_outer > 0 ? p->max_outer : 1000;
        // an iteration of this solver gains about as much as ten of the Jacobi one and
        // a refinement costs the same, so it waits for twice as many digits; not for
        // three times as many: FP32 directions of 128^2 P2 (condition 1e5) are noise by
        // then (22 to 23 iterations at 1e-2, 23 to 43 at 1e-3, depending on the right-hand side)
        const double d1 = p->inner_reltol > 0 && p->inner_reltol < 1 ? p->inner_reltol : 0.1;
        double delta = std::max(1e-3, d1 * d1);
        if (one) delta = std::max(1e-4, delta * delta);   // small systems: FP32 directions stay good
        void *args[] = {&n, &rp, &ci, &v64, &v32, &b, &x, &r, &q, &xc, &zp0, &zp1, &r64, &partial, &dst,
                        &at, &rt, &delta, &mi, &mo, &guess, &spin, &m};
        e = mg_start(ctx, kern, one, n, TPR, p->grid_blocks, args, grid);
    }
    return e == cudaSuccess ? GRMP_OK : grmp_cuda_fail(ctx, e, "multilevel solve launch");
}

template <int TPR, int U, bool PIPE>
int mg_launch_bicg(grmp_matrix A, const double *b, double *x, const grmp_solve_params *p, double *const vec[9],
                   double *partial, SolveState *dst, int *grid) {
    grmp_context ctx = A->space->mesh->ctx;
    int n = A->nrows, mi = std::min(p->maxiter, kMaxBicg), guess = p->use_initial_guess ? 1 : 0;
    double at = p->abstol, rt = p->reltol;
    const int32_t *rp = A->d_rowptr, *ci = A->d_cols;
    const double *v64 = A->d_vals64;
    long long spin = ctx->wait_limit;
    cudaMemsetAsync(dst, 0, sizeof(SolveState), ctx->stream);
    const bool one = A->nnz <= kOneBlock64 && p->grid_blocks <= 0;
    auto kern = one ? k_mgbicg64<TPR, U, PIPE, BlockSync> : k_mgbicg64<TPR, U, PIPE, MgGridSync>;
    MgDev<double> m = mg_device<double>(A);
    double *w[9];
    std::copy(vec, vec + 9, w);
    void *args[] = {&n, &rp, &ci, &v64, &b, &x, &w[0], &w[1], &w[2], &w[3], &w[4], &w[5], &w[6], &w[7], &w[8],
                    &partial, &dst, &at, &rt, &mi, &guess, &spin, &m};
    cudaError_t e = mg_start(ctx, kern, one, n, TPR, p->grid_blocks, args, grid);
    return e == cudaSuccess ? GRMP_OK : grmp_cuda_fail(ctx, e, "multilevel BiCGStab launch");
}

}  // namespace

void grmp_mg_free(grmp_matrix A) {
    if (!A) return;
    grmp_context ctx = A->space->mesh->ctx;
    // a garbage collector may destroy matrices on another thread than the one that allocates or solves
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    if (!A->mg) return;
    for (auto &b : A->mg->bufs) grmp_free(ctx, b.first, b.second);
    for (auto &N : A->mg->num) grmp_free(ctx, N.p, N.bytes);
    delete A->mg;
    A->mg = nullptr;
    ctx->hier.erase(std::find(ctx->hier.begin(), ctx->hier.end(), A));
}

bool grmp_mg_reclaim(grmp_context ctx, size_t bytes) {
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    bool any = false;
    while (!ctx->hier.empty() && !(any && ctx->budget && ctx->in_use + bytes <= ctx->budget)) {
        grmp_matrix A = ctx->hier.back();
        const size_t pat = mg_bytes(*A->mg), both = ++A->mg_reclaimed > 2 ? bytes : 0;
        for (int k = 0; k < 2; k++)
            if (A->mg_floor[k] != SIZE_MAX)
                A->mg_floor[k] = pat + both + (A->mg->num[k].p ? A->mg->num[k].bytes : mg_need(A, *A->mg, k));
        grmp_mg_free(A);
        any = true;
    }
    return any;
}

namespace {

// whether a hierarchy with numeric storage of this precision exists
bool mg_ready(grmp_matrix A, bool mixed) { return A->mg_state > 0 && A->mg && A->mg->num[mixed ? 1 : 0].p; }

// Whether the multilevel solver is for this matrix (scalar H1P1 / H1P2 with a
// diffusion term, not reaction dominated); builds or refreshes what it needs.
// *use = 0: the Jacobi solvers.  bicg: for BiCGStab, which pays from fewer rows.
int mg_prepare(grmp_matrix A, bool mixed, int *use, bool *checked, bool bicg = false) {
    *use = 0;
    *checked = false;
    grmp_space s = A->space;
    grmp_context ctx = s->mesh->ctx;
    const int bit = mixed ? 2 : 1;
    if (A->mg_state < 0 || A->imported || !A->elliptic || (A->reaction & bit) || s->ncomp != 1 ||
        (s->fe != GRMP_FE_H1P1 && s->fe != GRMP_FE_H1P2) || A->nrows < min_rows(s->mesh->dim, s->fe, mixed, bicg))
        return GRMP_OK;
    int rc = GRMP_OK;
    double react = 0.0;
    if (!mg_ready(A, mixed)) {
        if (mg_no_room(A, mixed)) return GRMP_OK;
        // the matrix is looked at first: analysis and storage are for those that the cycle is for
        rc = mixed ? mg_probe_first<float>(A, &react) : mg_probe_first<double>(A, &react);
        *checked = !rc;
        if (!rc && react > kMaxReaction) {
            A->reaction |= bit;
            return GRMP_OK;
        }
        bool fits = false;
        if (!rc) rc = mg_make(A, mixed, &fits);
        if (rc == GRMP_ERR_BUDGET || rc == GRMP_ERR_OUT_OF_MEMORY) {   // not even room to look
            ctx->last_error.clear();
            cudaGetLastError();
            return GRMP_OK;
        }
        if (rc || !fits) return rc;
    }
    MgCache::Num &N = A->mg->num[mixed ? 1 : 0];
    rc = mixed ? mg_probe<float>(A, N.D[0], N.iso[0], N.part, &react) : mg_probe<double>(A, N.D[0], N.iso[0], N.part, &react);
    if (rc) return rc;
    *checked = true;
    if (react > kMaxReaction) {
        A->reaction |= bit;
        return GRMP_OK;
    }
    if (mixed) mg_values<float>(A);
    else mg_values<double>(A);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return grmp_cuda_fail(ctx, e, "multilevel values");
    *use = 1;
    return GRMP_OK;
}

int mg_solve(grmp_matrix A, const double *b, double *x, bool mixed, grmp_solve_params *p, grmp_solve_stats *st,
                  bool *done) {
    grmp_context ctx = A->space->mesh->ctx;
    const double avg = (double)A->nnz / std::max(1, A->nrows);
    MgCache::Num &N = A->mg->num[mixed ? 1 : 0];
    const SolveState *dst = (const SolveState *)((char *)N.p + N.bytes - al(sizeof(SolveState)));
    *done = true;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    if (p->use_initial_guess)
        cudaMemcpyAsync(N.x0, x, (size_t)A->nrows * 8, cudaMemcpyDeviceToDevice, ctx->stream);
    cudaEventRecord(e0, ctx->stream);
    int grid = 0, code, rc;
    if (avg <= 8) {
        code = 204;
        rc = mg_launch<2, 4, true>(A, b, x, p, mixed, &grid);
    } else if (avg <= 20) {
        code = 404;
        rc = mg_launch<4, 4, true>(A, b, x, p, mixed, &grid);
    } else {
        code = 408;
        rc = mg_launch<4, 8, true>(A, b, x, p, mixed, &grid);
    }
    cudaEventRecord(e1, ctx->stream);
    SolveState hs;
    cudaError_t e = rc ? cudaSuccess : grmp_readback(ctx, &hs, dst, sizeof(hs));
    float ms = 0;
    if (!rc && e == cudaSuccess) cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc) return rc;
    if (e != cudaSuccess) return grmp_cuda_fail(ctx, e, "multilevel solve");
    st->status = hs.status;
    st->iterations = hs.iters;
    st->outer_iterations = hs.outer;
    st->final_relres = hs.relres;
    st->spmv_config = kMgConfig + code;
    st->grid_blocks = grid;
    st->solve_ms = ms;
    if (hs.status == GRMP_ERR_TIMEOUT) return grmp_fail(ctx, GRMP_ERR_TIMEOUT, "PCG: a grid barrier wait timed out");
    if (hs.status != GRMP_ERR_NOT_CONVERGED && hs.status != GRMP_ERR_NAN) return hs.status;
    // another solver goes on: from x if that is nearer, else from the start
    *done = false;
    if (hs.nearer) p->use_initial_guess = 1;
    else if (p->use_initial_guess)
        e = cudaMemcpyAsync(x, N.x0, (size_t)A->nrows * 8, cudaMemcpyDeviceToDevice, ctx->stream);
    return e == cudaSuccess ? GRMP_OK : grmp_cuda_fail(ctx, e, "multilevel solve");
}

}  // namespace

int grmp_mg_cg(grmp_matrix A, const double *b, double *x, grmp_solve_params *p, grmp_solve_stats *st, bool *done,
               bool *checked, bool present) {
    *done = *checked = false;
    for (int mixed = p->mode == GRMP_SOLVE_MIXED; mixed >= 0; mixed--) {
        if (present && !mg_ready(A, mixed)) return GRMP_OK;
        int use = 0;
        bool ok = false;
        int rc = mg_prepare(A, mixed, &use, &ok);
        *checked = *checked || ok;   // of the caller's precision: the first to be looked at
        if (rc || !use) return rc;
        rc = mg_solve(A, b, x, mixed, p, st, done);
        if (rc || *done || st->iterations >= p->maxiter) return rc;
    }
    return GRMP_OK;
}

int grmp_mg_bicgstab(grmp_matrix A, const double *b, double *x, const grmp_solve_params *p, double *const vec[9],
                     double *partial, void *state, grmp_solve_stats *st, bool *done, bool *checked) {
    grmp_context ctx = A->space->mesh->ctx;
    const double avg = (double)A->nnz / std::max(1, A->nrows);
    SolveState *dst = (SolveState *)state;
    *done = false;
    int use = 0;
    const int prc = mg_prepare(A, false, &use, checked, true);
    if (prc || !use) return prc;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, ctx->stream);
    int grid = 0;
    const int code = avg <= 8 ? 204 : 404;
    int rc = avg <= 8 ? mg_launch_bicg<2, 4, true>(A, b, x, p, vec, partial, dst, &grid)
                      : mg_launch_bicg<4, 4, true>(A, b, x, p, vec, partial, dst, &grid);
    cudaEventRecord(e1, ctx->stream);
    SolveState hs;
    cudaError_t e = rc ? cudaSuccess : grmp_readback(ctx, &hs, dst, sizeof(hs));
    float ms = 0;
    if (!rc && e == cudaSuccess) cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc) return rc;
    if (e != cudaSuccess) return grmp_cuda_fail(ctx, e, "multilevel BiCGStab");
    if (hs.status == GRMP_ERR_TIMEOUT)
        return grmp_fail(ctx, GRMP_ERR_TIMEOUT, "BiCGStab: a grid barrier wait timed out");
    *done = hs.status == GRMP_OK;
    if (!*done) return GRMP_OK;
    st->status = hs.status;
    st->iterations = hs.iters;
    st->final_relres = hs.relres;
    st->spmv_config = kMgConfig + code;
    st->grid_blocks = grid;
    st->solve_ms = ms;
    return GRMP_OK;
}
