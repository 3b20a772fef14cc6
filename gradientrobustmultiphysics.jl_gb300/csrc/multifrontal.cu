// Single-problem sparse direct solvers on the device (grmp_solve with
// mode GRMP_SOLVE_DIRECT or GRMP_SOLVE_MIXED_DIRECT).
//
// The reference solves every linear system with a sparse direct solver
// (UMFPACK through LinearSolve.jl, src/solvers.jl:89-101).  Here the matrix
// gets a multifrontal Cholesky factorisation over a nested-dissection tree
// (symbolic analysis: nd_symbolic.cpp, once per pattern, cached in the
// matrix; factorisation: forest.cu).
//  * DIRECT: FP64 factorisation, forward/backward solves (forest.cu),
//    residual refinement against the assembled FP64 matrix.
//  * MIXED_DIRECT: the factorisation and the triangular solves run in FP32
//    (the GB300 FP32 pipe is about 64x the FP64 rate) and precondition an
//    FP64 conjugate-gradient iteration on the assembled FP64 matrix, whose
//    residual decides convergence.
// Forward solves pass each front's contribution to its ancestors as an update
// vector read by the parent (no scatter, no atomics): results are
// reproducible run to run.
#include <algorithm>
#include <cmath>
#include <vector>

#include "forest.h"
#include "grmp_internal.h"

namespace {

constexpr int kTB = 256;   // threads per block

struct MfDev {
    const FoNode *node;
    const int32_t *lvl_nodes;
};

template <typename T>
__device__ __forceinline__ T warp_sum_t(T v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warp_sum_d(double v) { return warp_sum_t<double>(v); }

// ---------------------------------------------------------------- inverse-based solves
// For the FP32 preconditioner, applied once per CG iteration, each front
// keeps Q = [L11^-1 ; G] with G = L21 L11^-1 (same f x s layout as its
// factor columns).  Forward:  y_own = L11^-1 b_own,  u_struct += G b_own;
// backward: x_own = L11^-T y_own - G^T x_struct.  Every output is one dot
// product: a level is one or two fully parallel launches, with no
// sequential triangular chain inside a front.

// index idx in [lo, hi) with pref[idx] <= item < pref[idx + 1]
__device__ __forceinline__ int find_seg(const long long *pref, int lo, int hi, long long item) {
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (pref[mid] <= item) lo = mid;
        else hi = mid;
    }
    return lo;
}

// L11^-1 by 32 x 32 blocks: one thread block per (front, block column c).
// X_cc solves L_cc X = I; for b > c, X_bc solves L_bb X = -sum_{m=c}^{b-1} L_bm X_mc
// (the sum as a small GEMM by all threads, the 32-column triangular solve by
// one warp, each lane a column).  Block columns are independent.
template <typename T>
__global__ void __launch_bounds__(kTB) k_mf_invert(MfDev m, const long long *bcol, int nn, const T *L, T *Q) {
    __shared__ T Lbb[32][33];
    __shared__ T Tb[32][33];
    __shared__ T Ls[32][33];   // slab of L_b,[k0, k0+32)
    __shared__ T Xs[32][33];   // slab of X_[k0, k0+32),c
    const long long item = blockIdx.x;
    const int idx = find_seg(bcol, 0, nn, item);
    const FoNode nd = m.node[m.lvl_nodes[idx]];
    const int s = nd.s, c = (int)(item - bcol[idx]);
    const T *Lt = L + nd.L_off;
    T *Qt = Q + nd.L_off;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nbk = (s + 31) / 32;
    const int c0 = c * 32, cw = min(32, s - c0);
    for (int b = c; b < nbk; b++) {
        const int b0 = b * 32, bw = min(32, s - b0);
        // Tb = (b == c ? I : -sum_m L_bm X_mc), Lbb = L_bb.  The sum runs over
        // k in [c0, b0) (whole 32-slabs) with both factors staged in shared
        // memory, k ascending as a plain loop would take it.
        for (int q = tid; q < 32 * 32; q += blockDim.x) {
            const int r = q >> 5, cc = q & 31;
            Tb[r][cc] = (b == c && r == cc && r < bw) ? T(1) : T(0);
            Lbb[r][cc] = (r < bw && cc <= r) ? Lt[(long long)(b0 + r) * s + b0 + cc] : T(0);
        }
        if (b > c) {
            for (int k0 = c0; k0 < b0; k0 += 32) {
                __syncthreads();
                for (int q = tid; q < 32 * 32; q += blockDim.x) {
                    const int r = q >> 5, cc = q & 31;
                    Ls[r][cc] = r < bw ? Lt[(long long)(b0 + r) * s + k0 + cc] : T(0);
                    Xs[r][cc] = cc < cw ? Qt[(long long)(k0 + r) * s + c0 + cc] : T(0);
                }
                __syncthreads();
                for (int q = tid; q < 32 * 32; q += blockDim.x) {
                    const int r = q >> 5, cc = q & 31;
                    T acc = Tb[r][cc];
#pragma unroll 8
                    for (int kk = 0; kk < 32; kk++) acc -= Ls[r][kk] * Xs[kk][cc];
                    Tb[r][cc] = acc;
                }
            }
        }
        __syncthreads();
        if (warp == 0 && lane < cw) {   // forward substitution, column `lane`
            for (int r = 0; r < bw; r++) {
                T v = Tb[r][lane];
                for (int k = 0; k < r; k++) v -= Lbb[r][k] * Tb[k][lane];
                Tb[r][lane] = v / Lbb[r][r];
            }
        }
        __syncthreads();
        for (int q = tid; q < bw * cw; q += blockDim.x) {
            const int r = q / cw, cc = q - r * cw;
            Qt[(long long)(b0 + r) * s + c0 + cc] = Tb[r][cc];
        }
        __syncthreads();
    }
}

// G = L21 L11^-1 of every front, as tiles of 64 x 64 entries (rows i of the
// structure part, columns k): a 256-thread block per tile, the product over
// m in 32-wide slabs of L21 (64 x 32) and L11^-1 (32 x 64) staged in shared
// memory, 4 x 4 outputs per thread.  L11^-1 is lower triangular and only
// its blocks on or below the diagonal are stored, so entries with m < k are
// read as zero.  Tiles: {level-order front index, first row, first column}.
constexpr int kGmT = 64, kGmK = 32;

template <typename T>
__global__ void __launch_bounds__(256) k_mf_gmat(MfDev m, const int4 *tiles, long long ntiles, const T *L, T *Q) {
    __shared__ T As[kGmK][kGmT + 1];   // As[mm][i]
    __shared__ T Bs[kGmK][kGmT + 1];   // Bs[mm][k]
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;   // 16 x 16 threads, 4 x 4 outputs each
    for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const int4 tl = tiles[t];
        const FoNode nd = m.node[m.lvl_nodes[tl.x]];
        const int s = nd.s, sc = nd.f - nd.s, i0 = tl.y, k0 = tl.z;
        const T *L21 = L + nd.L_off + (long long)s * s;   // row i of the structure part: L21 + i * s
        const T *Qt = Q + nd.L_off;
        T acc[4][4];
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int b = 0; b < 4; b++) acc[a][b] = T(0);
        for (int m0 = k0; m0 < s; m0 += kGmK) {
            for (int q = threadIdx.x; q < kGmK * kGmT; q += 256) {
                const int mm = q % kGmK, ii = q / kGmK;   // A: consecutive threads along m (row-major L21)
                const int gi = i0 + ii, gm = m0 + mm;
                As[mm][ii] = (gi < sc && gm < s) ? L21[(long long)gi * s + gm] : T(0);
                const int kk = q % kGmT, m2 = q / kGmT;    // B: consecutive threads along k (row-major Q)
                const int gk = k0 + kk, gm2 = m0 + m2;
                Bs[m2][kk] = (gk < s && gm2 < s && gm2 >= gk) ? Qt[(long long)gm2 * s + gk] : T(0);
            }
            __syncthreads();
#pragma unroll 8
            for (int mm = 0; mm < kGmK; mm++) {
                T av[4], bv[4];
#pragma unroll
                for (int a = 0; a < 4; a++) av[a] = As[mm][ty * 4 + a];
#pragma unroll
                for (int b = 0; b < 4; b++) bv[b] = Bs[mm][tx * 4 + b];
#pragma unroll
                for (int a = 0; a < 4; a++)
#pragma unroll
                    for (int b = 0; b < 4; b++) acc[a][b] += av[a] * bv[b];
            }
            __syncthreads();
        }
#pragma unroll
        for (int a = 0; a < 4; a++) {
            const int gi = i0 + ty * 4 + a;
            if (gi >= sc) continue;
#pragma unroll
            for (int b = 0; b < 4; b++) {
                const int gk = k0 + tx * 4 + b;
                if (gk < s) Q[nd.L_off + (long long)(s + gi) * s + gk] = acc[a][b];
            }
        }
    }
}

// A solve's work items are tiles of one front: {front, first row, last row + 1}
// going up, {front, first of 32 columns} going down.  A block first puts the
// part of the vector that its tile multiplies into shared memory -- going up
// the own entries minus what the children pass up (src names those entries,
// so a tile gathers for itself and needs no launch or barrier before it) --
// and then reads its part of Q once, coalesced.  526k DoFs, 16 levels: with a
// gather launch per level, a warp per row of Q that searched its front and
// gathered the vector through two indices per entry, and 1,024-thread column
// tiles doing the same, 3.6 ms per application; Q is 295 MB and read twice.
template <int NT>
__global__ void __launch_bounds__(NT) k_fq_fwd(FoDev m, const int4 *tiles, const float *Q, float *uv, const float *w,
                                               float *wy) {
    extern __shared__ float fq_smem[];
    float *b = fq_smem;
    const int4 t = tiles[blockIdx.x];
    const FoNode nd = m.node[t.x];
    const int s = nd.s, tid = threadIdx.x;
    const int32_t *fr = m.front + nd.front_off;
    const int2 *src = m.src + nd.front_off;
    auto up = [&](int k) {
        const int2 q = src[k];
        return (q.x >= 0 ? uv[q.x] : 0.f) + (q.y >= 0 ? uv[q.y] : 0.f);
    };
    for (int k = tid; k < s; k += NT) b[k] = w[fr[k]] - up(k);
    __syncthreads();
    const float *Qt = Q + nd.L_off;
    // 8 lanes per row of short rows, a warp otherwise, two rows at a time (the
    // entries above a row's diagonal are stored as zeros within its 32 x 32
    // block and not at all beyond it)
    const int lp = s <= 64 ? 8 : 32, lane = tid & (lp - 1), rows = NT / lp;
    const int span = (t.z - t.y + 2 * rows - 1) / (2 * rows) * (2 * rows);
    for (int o = tid / lp; o < span; o += 2 * rows) {
        const int r0 = t.y + o, r1 = r0 + rows;
        const int e0 = r0 < t.z ? (r0 < s ? r0 + 1 : s) : 0, e1 = r1 < t.z ? (r1 < s ? r1 + 1 : s) : 0;
        const float *Q0 = Qt + (long long)r0 * s, *Q1 = Qt + (long long)r1 * s;
        float a0 = 0.f, a1 = 0.f;
        const int both = min(e0, e1);
        int k = lane;
#pragma unroll 4
        for (; k < both; k += lp) {
            const float bk = b[k];
            a0 += Q0[k] * bk;
            a1 += Q1[k] * bk;
        }
        for (int q = k; q < e0; q += lp) a0 += Q0[q] * b[q];
        for (int q = k; q < e1; q += lp) a1 += Q1[q] * b[q];
        for (int d = lp / 2; d > 0; d >>= 1) {
            a0 += __shfl_xor_sync(0xffffffffu, a0, d);
            a1 += __shfl_xor_sync(0xffffffffu, a1, d);
        }
        if (lane == 0) {
            if (r0 < t.z) {
                if (r0 < s) wy[fr[r0]] = a0;
                else uv[nd.uv_off + r0 - s] = up(r0) + a0;
            }
            if (r1 < t.z) {
                if (r1 < s) wy[fr[r1]] = a1;
                else uv[nd.uv_off + r1 - s] = up(r1) + a1;
            }
        }
    }
}

template <int NT>
__global__ void __launch_bounds__(NT) k_fq_bwd(FoDev m, const int4 *tiles, const float *Q, const float *wy, float *wx) {
    extern __shared__ float fq_smem[];
    float *part = fq_smem, *v = part + NT;
    const int4 t = tiles[blockIdx.x];
    const FoNode nd = m.node[t.x];
    const int s = nd.s, f = nd.f, kb = t.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NW = NT / 32;
    const int32_t *fr = m.front + nd.front_off;
    for (int j = kb + tid; j < f; j += NT) v[j - kb] = j < s ? wy[fr[j]] : -wx[fr[j]];
    __syncthreads();
    const int k = kb + lane;
    float acc = 0.f;
    if (k < s) {
        const float *Qk = Q + nd.L_off + k;
#pragma unroll 8
        for (int j = kb + warp; j < f; j += NW) acc += Qk[(long long)j * s] * v[j - kb];
    }
    part[tid] = acc;
    __syncthreads();
    if (warp == 0 && k < s) {
        float sum = 0.f;
        for (int g = 0; g < NW; g++) sum += part[g * 32 + lane];
        wx[fr[k]] = sum;
    }
}

// ---------------------------------------------------------------- vector kernels
// A x by 8 lanes per row (20-odd entries a row: a warp per row leaves lanes
// idle and adds five FP64 shuffle steps to three multiply-adds; 526k rows
// 0.34 ms before)
__device__ __forceinline__ double row_dot8(const int32_t *rowptr, const int32_t *cols, const double *vals,
                                           const double *x, int row, int lane) {
    double s = 0.0;
    for (int k = rowptr[row] + lane; k < rowptr[row + 1]; k += 8) s += vals[k] * x[cols[k]];
    return s;
}

// block's sum (256 threads, fixed order) in part[blockIdx.x]
__device__ __forceinline__ void block_part(double acc, double *part) {
    __shared__ double sh[32];
    acc = warp_sum_d(acc);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sh[w];
        part[blockIdx.x] = t;
    }
}

// sum of nb partials, the same in every thread of every block
__device__ __forceinline__ double all_parts(const double *part, int nb) {
    __shared__ double sh2[33];
    double a = 0.0;
    for (int i = threadIdx.x; i < nb; i += blockDim.x) a += part[i];
    a = warp_sum_d(a);
    if ((threadIdx.x & 31) == 0) sh2[threadIdx.x >> 5] = a;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sh2[w];
        sh2[32] = t;
    }
    __syncthreads();
    return sh2[32];
}

// r = b - A x (FP64), per-block partial sums of r^2 (fixed order)
__global__ void __launch_bounds__(kTB) k_resid(int n, const int32_t *rowptr, const int32_t *cols, const double *vals,
                                               const double *x, const double *b, double *r, double *part) {
    const int lane = threadIdx.x & 7, pad = (n + 3) & ~3;
    double acc = 0.0;
    for (int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 3; row < pad; row += (gridDim.x * blockDim.x) >> 3) {
        double s = row < n ? row_dot8(rowptr, cols, vals, x, row, lane) : 0.0;
        for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (row < n && lane == 0) {
            const double v = b[row] - s;
            r[row] = v;
            acc += v * v;
        }
    }
    block_part(acc, part);
}

// q = A p (FP64) and partial sums of p.q
__global__ void __launch_bounds__(kTB) k_apply_dot(int n, const int32_t *rowptr, const int32_t *cols, const double *vals,
                                                   const double *p, double *q, double *part) {
    const int lane = threadIdx.x & 7, pad = (n + 3) & ~3;
    double acc = 0.0;
    for (int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 3; row < pad; row += (gridDim.x * blockDim.x) >> 3) {
        double s = row < n ? row_dot8(rowptr, cols, vals, p, row, lane) : 0.0;
        for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (row < n && lane == 0) {
            q[row] = s;
            acc += p[row] * s;
        }
    }
    block_part(acc, part);
}

template <typename T>
__global__ void k_to(int n, const double *a, T *b) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) b[i] = (T)a[i];
}

// x += alpha p, r -= alpha q with alpha = rz / (p, q) from the partial sums,
// the new residual rounded to FP32 for the preconditioner, partial sums of r^2;
// *bad when (p, q) is not positive
__global__ void __launch_bounds__(kTB) k_cg_update(int n, const double *pqpart, int nb, const double *rz, const double *p,
                                                   const double *q, double *x, double *r, float *w, double *part,
                                                   int *bad) {
    const double pq = all_parts(pqpart, nb);
    const bool ok = pq > 0.0 && isfinite(pq);
    const double alpha = ok ? *rz / pq : 0.0;
    if (!ok && blockIdx.x == 0 && threadIdx.x == 0) *bad = 1;
    double acc = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        x[i] += alpha * p[i];
        const double ri = r[i] - alpha * q[i];
        r[i] = ri;
        w[i] = (float)ri;
        acc += ri * ri;
    }
    block_part(acc, part);
}

// p = z + (rz_new / rz_old) p with rz_new from the partial sums (first: p = z)
__global__ void __launch_bounds__(kTB) k_xpby(int n, const double *zpart, int nb, const double *rz_old, double *rz_new,
                                              int first, const double *z, double *p) {
    const double rz = all_parts(zpart, nb);
    if (blockIdx.x == 0 && threadIdx.x == 0) *rz_new = rz;
    const double beta = first ? 0.0 : rz / *rz_old;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        p[i] = first ? z[i] : z[i] + beta * p[i];
}

// z = (double) zf, partial sums of r.z
template <typename T>
__global__ void k_from_dot(int n, const T *zf, const double *r, double *z, double *part) {
    __shared__ double sh[32];
    double acc = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double zi = (double)zf[i];
        z[i] = zi;
        acc += r[i] * zi;
    }
    acc = warp_sum_d(acc);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sh[w];
        part[blockIdx.x] = t;
    }
}

// partial sums of a.b
__global__ void k_dot(int n, const double *a, const double *b, double *part) {
    __shared__ double sh[32];
    double acc = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) acc += a[i] * b[i];
    acc = warp_sum_d(acc);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sh[w];
        part[blockIdx.x] = t;
    }
}

// per-block maxima of the row sums of |A| (||A||_inf)
__global__ void k_rownorm(int n, const int32_t *rowptr, const double *vals, double *part) {
    __shared__ double sh[32];
    double mx = 0.0;
    for (int row = blockIdx.x * blockDim.x + threadIdx.x; row < n; row += gridDim.x * blockDim.x) {
        double s = 0.0;
        for (int k = rowptr[row]; k < rowptr[row + 1]; k++) s += fabs(vals[k]);
        mx = fmax(mx, s);
    }
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t = fmax(t, sh[w]);
        part[blockIdx.x] = t;
    }
}

template <typename T>
__global__ void k_add_from(int n, const T *w, double *x) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] += (double)w[i];
}

}  // namespace

// ---------------------------------------------------------------- host side

struct MfCache {
    NdSymbolic S;
    MfForest *F = nullptr;          // of the precision last used
    int esize = 0;
    int *err = nullptr;
    // inverse-based FP32 preconditioner: Q = [L11^-1; L21 L11^-1] per front and
    // three vectors
    std::vector<std::pair<void *, size_t>> bufs;
    MfDev dev{};
    float *Q = nullptr, *w = nullptr, *wy = nullptr, *wx = nullptr;
    const long long *bcol = nullptr;   // prefix of 32-column tiles per front in level order
    const int4 *gtiles = nullptr;      // 64 x 64 tiles of every front's L21 L11^-1
    const int4 *tiles = nullptr;       // tiles of the solves
    struct Lv {
        int fwd, nfwd, fwdb, nfwdb, bwd, nbwd, bwdb, nbwdb, maxf;   // first tile and count: up and down, small and large fronts
    };
    std::vector<Lv> lv;
    long long total_gtiles = 0, total_bcols = 0;
    // the preconditioner's level launches (w -> wx), captured once
    cudaGraphExec_t apply_graph = nullptr;
    int apply_kernels = 0;
};

namespace {

constexpr int kFwdSmall = 64;    // own DoFs up to which a tile going up is 128 rows by 128 threads, else 32 rows by 512
constexpr int kBwdSmall = 256;   // fronts up to this size take 128 threads per column tile, larger ones 512

template <typename V>
int mf_take(grmp_context ctx, MfCache &C, size_t count, V **out) {
    const size_t bytes = std::max<size_t>(1, count) * sizeof(V);
    int rc = grmp_alloc(ctx, (void **)out, bytes);
    if (!rc) C.bufs.push_back({(void *)*out, bytes});
    return rc;
}

template <typename V>
int mf_upload(grmp_context ctx, MfCache &C, const std::vector<V> &v, const V **out) {
    V *p = nullptr;
    int rc = mf_take(ctx, C, v.size(), &p);
    if (rc) return rc;
    *out = p;
    if (v.empty()) return GRMP_OK;
    cudaError_t e = cudaMemcpyAsync(p, v.data(), v.size() * sizeof(V), cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    return e == cudaSuccess ? GRMP_OK : grmp_cuda_fail(ctx, e, "multifrontal upload");
}

// device arrays of the precision in use
void mf_free_numeric(grmp_context ctx, MfCache &C) {
    if (C.apply_graph) cudaGraphExecDestroy(C.apply_graph);
    C.apply_graph = nullptr;
    grmp_forest_free(ctx, C.F);
    C.F = nullptr;
    for (auto &b : C.bufs) grmp_free(ctx, b.first, b.second);
    C.bufs.clear();
    C.Q = C.w = C.wy = C.wx = nullptr;
    C.err = nullptr;
    C.esize = 0;
}

int mf_build(grmp_matrix A) {
    grmp_context ctx = A->space->mesh->ctx;
    const int n = A->nrows;
    std::vector<int32_t> rp(n + 1), ci((size_t)A->nnz);
    cudaError_t e = cudaMemcpyAsync(rp.data(), A->d_rowptr, (size_t)(n + 1) * 4, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(ci.data(), A->d_cols, (size_t)A->nnz * 4, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return grmp_cuda_fail(ctx, e, "multifrontal: pattern download");
    // separators in the graph of the mesh's cells, which has to cover the pattern:
    // face terms couple across its separators, their matrices use the pattern itself
    grmp_space s = A->space;
    NdGraph G;
    bool mesh_graph = false;
    if (!A->imported && !A->face_coupled && s->d_celldofs && (s->fe == GRMP_FE_H1P1 || s->fe == GRMP_FE_H1P2)) {
        std::vector<int32_t> cd((size_t)s->mesh->ncells * s->ldofs);
        e = cudaMemcpyAsync(cd.data(), s->d_celldofs, cd.size() * 4, cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) return grmp_cuda_fail(ctx, e, "multifrontal: cell DoFs");
        mesh_graph = nd_cell_graph(n, s->mesh->ncells, s->ldofs, s->ncomp, cd.data(), &G) == 0;
    }
    MfCache *C = new MfCache;
    const int src = nd_symbolic_build(n, rp.data(), ci.data(), &C->S, mesh_graph ? &G : nullptr);
    if (src) {
        delete C;
        return grmp_fail(ctx, GRMP_ERR_INVALID_ARG, "multifrontal: symbolic analysis failed (%d)", src);
    }
    A->mf = C;
    return GRMP_OK;
}

// forest, and for FP32 the inverse's arrays and tile lists
int mf_numeric_arrays(grmp_matrix A, int esize) {
    grmp_context ctx = A->space->mesh->ctx;
    MfCache &C = *A->mf;
    if (C.esize == esize) return GRMP_OK;
    mf_free_numeric(ctx, C);
    const NdSymbolic &S = C.S;
    // shared memory of the solve kernels: the front's vector
    if ((esize == 8 ? (size_t)(S.max_f + 512) * 8 : (size_t)(S.max_f + 512) * 4) > 220 * 1024)
        return grmp_fail(ctx, GRMP_ERR_UNSUPPORTED, "direct solve: front of %d DoFs exceeds shared memory", S.max_f);
    int rc = grmp_forest_create(ctx, {&S}, {FoProblem{0, 0, 0}}, esize, &C.F);
    if (!rc) rc = mf_take(ctx, C, 1, &C.err);
    const size_t n = (size_t)A->nrows;
    if (!rc && esize == 8) {
        double *w = nullptr;
        rc = mf_take(ctx, C, n, &w);
        C.w = (float *)w;
    } else if (!rc) {
        const int nl = (int)S.level_ptr.size() - 1;
        std::vector<long long> bcol(S.nnodes + 1, 0);
        std::vector<int4> gtiles, tiles;
        for (int i = 0; i < S.nnodes; i++) {
            const NdNode &q = S.node[S.level_nodes[i]];
            bcol[i + 1] = bcol[i] + (q.s + 31) / 32;
            for (int i0 = 0; i0 < q.f - q.s; i0 += kGmT)
                for (int k0 = 0; k0 < q.s; k0 += kGmT) gtiles.push_back(make_int4(i, i0, k0, 0));
        }
        C.lv.assign(nl, {});
        for (int l = 0; l < nl; l++) {
            MfCache::Lv &v = C.lv[l];
            v.maxf = S.level_maxf[l];
            v.fwd = (int)tiles.size();
            for (int i = S.level_ptr[l]; i < S.level_ptr[l + 1]; i++) {
                const int t = S.level_nodes[i];
                const NdNode &q = S.node[t];
                if (q.s <= kFwdSmall)
                    for (int r = 0; r < q.f; r += 128) tiles.push_back(make_int4(t, r, std::min(q.f, r + 128), 0));
            }
            v.nfwd = (int)tiles.size() - v.fwd;
            v.fwdb = (int)tiles.size();
            for (int i = S.level_ptr[l]; i < S.level_ptr[l + 1]; i++) {
                const int t = S.level_nodes[i];
                const NdNode &q = S.node[t];
                if (q.s > kFwdSmall)   // every tile gathers all s own entries
                    for (int r = 0; r < q.f; r += 32) tiles.push_back(make_int4(t, r, std::min(q.f, r + 32), 0));
            }
            v.nfwdb = (int)tiles.size() - v.fwdb;
            for (int big = 0; big < 2; big++) {
                const int b = (int)tiles.size();
                for (int i = S.level_ptr[l]; i < S.level_ptr[l + 1]; i++) {
                    const int t = S.level_nodes[i];
                    if ((S.node[t].f > kBwdSmall) == (big == 1))
                        for (int k = 0; k < S.node[t].s; k += 32) tiles.push_back(make_int4(t, k, 0, 0));
                }
                (big ? v.bwdb : v.bwd) = b;
                (big ? v.nbwdb : v.nbwd) = (int)tiles.size() - b;
            }
        }
        C.total_gtiles = (long long)gtiles.size();
        C.total_bcols = bcol[S.nnodes];
        C.dev.node = C.F->dev.node;
        rc = mf_upload(ctx, C, S.level_nodes, &C.dev.lvl_nodes);
        if (!rc) rc = mf_upload(ctx, C, bcol, &C.bcol);
        if (!rc) rc = mf_upload(ctx, C, gtiles, &C.gtiles);
        if (!rc) rc = mf_upload(ctx, C, tiles, &C.tiles);
        if (!rc) rc = mf_take(ctx, C, (size_t)S.L_size, &C.Q);
        if (!rc) rc = mf_take(ctx, C, n, &C.w);
        if (!rc) rc = mf_take(ctx, C, n, &C.wy);
        if (!rc) rc = mf_take(ctx, C, n, &C.wx);
    }
    if (rc) {
        mf_free_numeric(ctx, C);
        return rc;
    }
    C.esize = esize;
    return GRMP_OK;
}

int mf_numeric(grmp_matrix A, bool mixed) {
    grmp_context ctx = A->space->mesh->ctx;
    int rc = mf_numeric_arrays(A, mixed ? 4 : 8);
    if (rc) return rc;
    MfCache &C = *A->mf;
    rc = mixed ? grmp_forest_factor32(ctx, C.F, A->d_vals64, C.err) : grmp_forest_factor64(ctx, C.F, A->d_vals64, C.err);
    if (rc) return rc;
    int herr = 0;
    cudaError_t e = cudaMemcpyAsync(&herr, C.err, 4, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return grmp_cuda_fail(ctx, e, "multifrontal factorisation");
    if (herr)
        return grmp_fail(ctx, GRMP_ERR_NAN, "multifrontal %s factorisation: non-positive pivot in front %d",
                         mixed ? "FP32" : "FP64", herr - 1);
    if (!mixed) return GRMP_OK;
    // Q = [L11^-1; L21 L11^-1] of every front
    if (C.total_bcols > 0) {
        k_mf_invert<float><<<(unsigned)C.total_bcols, kTB, 0, ctx->stream>>>(C.dev, C.bcol, C.S.nnodes,
                                                                            (const float *)C.F->L, C.Q);
        GRMP_LAUNCHED(ctx);
    }
    if (C.total_gtiles > 0) {
        const int gg = (int)std::min<long long>(C.total_gtiles, 8LL * ctx->num_sms);
        k_mf_gmat<float><<<gg, 256, 0, ctx->stream>>>(C.dev, C.gtiles, C.total_gtiles, (const float *)C.F->L, C.Q);
        GRMP_LAUNCHED(ctx);
    }
    e = cudaGetLastError();
    return e == cudaSuccess ? GRMP_OK : grmp_cuda_fail(ctx, e, "multifrontal inverse");
}

// wx <- A^{-1} w with the inverse-based factor: the level launches, in order
int mf_enqueue_inverse(grmp_matrix A) {
    grmp_context ctx = A->space->mesh->ctx;
    MfCache &C = *A->mf;
    float *uv = (float *)C.F->uv;
    const size_t sf = (size_t)C.S.max_s * 4;
    grmp_allow_smem(k_fq_fwd<512>);
    grmp_allow_smem(k_fq_bwd<512>);
    int k = 0;
    for (const MfCache::Lv &v : C.lv) {
        if (v.nfwdb) {
            k_fq_fwd<512><<<v.nfwdb, 512, sf, ctx->stream>>>(C.F->dev, C.tiles + v.fwdb, C.Q, uv, C.w, C.wy);
            k++;
        }
        if (v.nfwd) {
            k_fq_fwd<128><<<v.nfwd, 128, (size_t)kFwdSmall * 4, ctx->stream>>>(C.F->dev, C.tiles + v.fwd, C.Q, uv, C.w, C.wy);
            k++;
        }
    }
    for (size_t l = C.lv.size(); l-- > 0;) {
        const MfCache::Lv &v = C.lv[l];
        if (v.nbwdb) {
            k_fq_bwd<512><<<v.nbwdb, 512, (size_t)(512 + v.maxf) * 4, ctx->stream>>>(C.F->dev, C.tiles + v.bwdb, C.Q, C.wy,
                                                                                    C.wx);
            k++;
        }
        if (v.nbwd) {
            k_fq_bwd<128><<<v.nbwd, 128, (size_t)(128 + kBwdSmall) * 4, ctx->stream>>>(C.F->dev, C.tiles + v.bwd, C.Q,
                                                                                      C.wy, C.wx);
            k++;
        }
    }
    return k;
}

// The sequence is replayed once per CG iteration with the same buffers, so it
// is captured into a CUDA graph at the first application after the numeric
// storage was (re)allocated and replayed from then on.
int mf_apply_inverse(grmp_matrix A) {
    grmp_context ctx = A->space->mesh->ctx;
    MfCache &C = *A->mf;
    if (!C.apply_graph) {
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            C.apply_kernels = mf_enqueue_inverse(A);
            e = cudaStreamEndCapture(ctx->stream, &g);
        }
        if (e == cudaSuccess) e = cudaGraphInstantiate(&C.apply_graph, g, 0);
        if (g) cudaGraphDestroy(g);
        if (e != cudaSuccess) {
            C.apply_graph = nullptr;
            return grmp_cuda_fail(ctx, e, "preconditioner graph capture");
        }
    }
    cudaError_t e = cudaGraphLaunch(C.apply_graph, ctx->stream);
    ctx->launches += (uint64_t)C.apply_kernels;
    if (e != cudaSuccess) return grmp_cuda_fail(ctx, e, "preconditioner graph launch");
    return GRMP_OK;
}

double host_sum(grmp_context ctx, const double *dpart, int nb, cudaError_t *e) {
    std::vector<double> h(nb);
    *e = cudaMemcpyAsync(h.data(), dpart, (size_t)nb * 8, cudaMemcpyDeviceToHost, ctx->stream);
    if (*e == cudaSuccess) *e = cudaStreamSynchronize(ctx->stream);
    double s = 0.0;
    for (double v : h) s += v;   // fixed order
    return s;
}

}  // namespace

void grmp_mf_cache_free(grmp_matrix A) {
    if (!A || !A->mf) return;
    mf_free_numeric(A->space->mesh->ctx, *A->mf);
    delete A->mf;
    A->mf = nullptr;
}

// grmp_solve for the direct modes; called with the context locked.
int grmp_mf_solve(grmp_matrix A, grmp_vector b, grmp_vector x, const grmp_solve_params *p, grmp_solve_stats *st) {
    grmp_context ctx = A->space->mesh->ctx;
    const int n = A->nrows;
    const bool mixed = p->mode == GRMP_SOLVE_MIXED_DIRECT;
    if (!A->has64) return grmp_fail(ctx, GRMP_ERR_INVALID_ARG, "solve: FP64 values not assembled");
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, ctx->stream);
    int rc = A->mf ? GRMP_OK : mf_build(A);
    if (!rc) rc = mf_numeric(A, mixed);
    const int nb = 2 * ctx->num_sms, tb = 256;
    double *r = nullptr, *z = nullptr, *pp = nullptr, *q = nullptr, *part = nullptr;
    const size_t vb = (size_t)n * 8;
    if (!rc) rc = grmp_alloc(ctx, (void **)&r, vb);
    if (!rc) rc = grmp_alloc(ctx, (void **)&z, vb);
    if (!rc) rc = grmp_alloc(ctx, (void **)&pp, vb);
    if (!rc) rc = grmp_alloc(ctx, (void **)&q, vb);
    // partial sums: r.r, p.q, r.z; then the two r.z scalars and the breakdown flag
    if (!rc) rc = grmp_alloc(ctx, (void **)&part, (size_t)(3 * nb + 4) * 8);
    auto cleanup = [&]() {
        grmp_free(ctx, r, vb);
        grmp_free(ctx, z, vb);
        grmp_free(ctx, pp, vb);
        grmp_free(ctx, q, vb);
        grmp_free(ctx, part, (size_t)(3 * nb + 4) * 8);
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
    };
    if (rc) {
        cleanup();
        return rc;
    }
    MfCache &C = *A->mf;
    cudaError_t e = cudaSuccess;
    const int gv = (n + tb - 1) / tb;
    if (!p->use_initial_guess) cudaMemsetAsync(x->d, 0, vb, ctx->stream);
    k_dot<<<nb, tb, 0, ctx->stream>>>(n, b->d, b->d, part);
    GRMP_LAUNCHED(ctx);
    const double bn = sqrt(host_sum(ctx, part, nb, &e));
    const double tol = std::max(p->abstol, p->reltol * bn);
    int it = 0, status = GRMP_ERR_NOT_CONVERGED;
    double rn = 0.0;
    if (!mixed) {
        // FP64 factor: x += A^{-1} (b - A x) until reltol or the residual stops falling
        double prev = INFINITY;
        for (;; it++) {
            k_resid<<<nb, tb, 0, ctx->stream>>>(n, A->d_rowptr, A->d_cols, A->d_vals64, x->d, b->d, r, part);
            GRMP_LAUNCHED(ctx);
            rn = sqrt(host_sum(ctx, part, nb, &e));
            if (e != cudaSuccess) break;
            if (rn <= tol || bn == 0.0) {
                status = GRMP_OK;
                break;
            }
            if ((it > 0 && rn > 0.5 * prev) || it >= std::min(p->maxiter, 8)) {
                // the residual stopped falling (FP64 floor of an ill-conditioned system):
                // accept when the normwise backward error ||r|| / (||A|| ||x|| + ||b||) is at rounding level
                k_rownorm<<<nb, tb, 0, ctx->stream>>>(n, A->d_rowptr, A->d_vals64, part);
                GRMP_LAUNCHED(ctx);
                std::vector<double> hm(nb);
                if (e == cudaSuccess) e = cudaMemcpyAsync(hm.data(), part, (size_t)nb * 8, cudaMemcpyDeviceToHost, ctx->stream);
                if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
                double anorm = 0.0;
                for (double v : hm) anorm = std::max(anorm, v);
                k_dot<<<nb, tb, 0, ctx->stream>>>(n, x->d, x->d, part);
                GRMP_LAUNCHED(ctx);
                const double xn = sqrt(host_sum(ctx, part, nb, &e));
                const double eta = rn / (anorm * xn + bn + 1e-300);
                status = (it > 0 && rn > 0.5 * prev && eta <= 1e-13) ? GRMP_OK : GRMP_ERR_NOT_CONVERGED;
                break;
            }
            prev = rn;
            cudaMemcpyAsync((double *)C.w, r, vb, cudaMemcpyDeviceToDevice, ctx->stream);
            grmp_forest_solve64(ctx, C.F, (double *)C.w, nullptr);
            k_add_from<double><<<gv, tb, 0, ctx->stream>>>(n, (const double *)C.w, x->d);
            GRMP_LAUNCHED(ctx);
        }
    } else {
        // FP64 conjugate gradients preconditioned by the FP32 factorisation
        k_resid<<<nb, tb, 0, ctx->stream>>>(n, A->d_rowptr, A->d_cols, A->d_vals64, x->d, b->d, r, part);
        GRMP_LAUNCHED(ctx);
        rn = sqrt(host_sum(ctx, part, nb, &e));
        double *pqpart = part + nb, *zpart = part + 2 * nb, *rz = part + 3 * nb;
        int *bad = (int *)(rz + 2);
        cudaMemsetAsync(bad, 0, 4, ctx->stream);
        int cur = 0;
        // z = M^{-1} r and p = z + beta p (w holds r in FP32); the scalars stay on the device
        auto direction = [&](bool first) {
            if (mf_apply_inverse(A)) e = cudaErrorUnknown;
            k_from_dot<float><<<nb, tb, 0, ctx->stream>>>(n, C.wx, r, z, zpart);
            k_xpby<<<nb, tb, 0, ctx->stream>>>(n, zpart, nb, rz + cur, rz + (cur ^ 1), first ? 1 : 0, z, pp);
            ctx->launches += 2;
            cur ^= 1;
        };
        // CG with restarts from the true FP64 residual: when the recurrence
        // residual has converged but b - A x has not, restart from x (at most
        // 3 times); a residual that no longer falls is accepted when its
        // normwise backward error is at FP64 rounding level.
        double prev_true = INFINITY;
        for (int restart = 0; restart < 4 && e == cudaSuccess; restart++) {
            if (rn > tol) {
                k_to<float><<<gv, tb, 0, ctx->stream>>>(n, r, C.w);
                GRMP_LAUNCHED(ctx);
                direction(true);
            }
            status = GRMP_ERR_NOT_CONVERGED;
            while (e == cudaSuccess) {
                if (rn <= tol || bn == 0.0) {
                    status = GRMP_OK;
                    break;
                }
                if (it >= p->maxiter) break;
                k_apply_dot<<<nb, tb, 0, ctx->stream>>>(n, A->d_rowptr, A->d_cols, A->d_vals64, pp, q, pqpart);
                k_cg_update<<<nb, tb, 0, ctx->stream>>>(n, pqpart, nb, rz + cur, pp, q, x->d, r, C.w, part, bad);
                ctx->launches += 2;
                int hbad = 0;
                cudaError_t eb = cudaMemcpyAsync(&hbad, bad, 4, cudaMemcpyDeviceToHost, ctx->stream);
                rn = sqrt(host_sum(ctx, part, nb, &e));
                if (e == cudaSuccess) e = eb;
                if (hbad || !std::isfinite(rn)) {
                    status = GRMP_ERR_NAN;
                    break;
                }
                it++;
                if (rn <= tol) continue;
                direction(false);
            }
            if (e != cudaSuccess || status == GRMP_ERR_NAN) break;
            // the true FP64 residual of the iterate (r becomes b - A x)
            k_resid<<<nb, tb, 0, ctx->stream>>>(n, A->d_rowptr, A->d_cols, A->d_vals64, x->d, b->d, r, part);
            GRMP_LAUNCHED(ctx);
            rn = sqrt(host_sum(ctx, part, nb, &e));
            if (rn <= 2.0 * tol) {
                status = GRMP_OK;
                break;
            }
            if (rn > 0.5 * prev_true || it >= p->maxiter) {
                k_rownorm<<<nb, tb, 0, ctx->stream>>>(n, A->d_rowptr, A->d_vals64, part);
                GRMP_LAUNCHED(ctx);
                std::vector<double> hm(nb);
                if (e == cudaSuccess) e = cudaMemcpyAsync(hm.data(), part, (size_t)nb * 8, cudaMemcpyDeviceToHost, ctx->stream);
                if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
                double anorm = 0.0;
                for (double v : hm) anorm = std::max(anorm, v);
                k_dot<<<nb, tb, 0, ctx->stream>>>(n, x->d, x->d, part);
                GRMP_LAUNCHED(ctx);
                const double xn = sqrt(host_sum(ctx, part, nb, &e));
                status = rn / (anorm * xn + bn + 1e-300) <= 1e-13 ? GRMP_OK : GRMP_ERR_NOT_CONVERGED;
                break;
            }
            prev_true = rn;
            status = GRMP_ERR_NOT_CONVERGED;
        }
    }
    cudaEventRecord(e1, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    float ms = 0.0f;
    if (e == cudaSuccess) cudaEventElapsedTime(&ms, e0, e1);
    cleanup();
    if (e != cudaSuccess) return grmp_cuda_fail(ctx, e, "multifrontal solve");
    st->status = status;
    st->iterations = it;
    st->outer_iterations = 0;
    st->spmv_config = 0;
    st->grid_blocks = nb;
    st->final_relres = bn > 0 ? rn / bn : 0.0;
    st->solve_ms = ms;
    if (status == GRMP_ERR_NOT_CONVERGED)
        return grmp_fail(ctx, status, "direct solve: relative residual %.3e after %d steps", st->final_relres, it);
    if (status == GRMP_ERR_NAN) return grmp_fail(ctx, status, "direct solve: breakdown of the preconditioned CG");
    return status;
}
