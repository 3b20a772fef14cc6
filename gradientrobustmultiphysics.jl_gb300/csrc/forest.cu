// Multifrontal Cholesky over a forest of assembly trees: the direct solver of
// one large matrix (multifrontal.cu) and of a batch of Stokes problems
// (batch.cu).
//
// All fronts of one level (height above the leaves) of all problems are one
// set of independent work items, a level is a few launches:
//  * fronts that fit shared memory (150 rows FP64, 212 FP32) by one block
//    each: assembled, factored and taken apart there, global memory sees
//    entries, children's update matrices, factor columns and the update
//    matrix once;
//  * larger fronts by groups of blocks (one cooperative launch a level, each
//    group its own bounded barrier) in 64-column panels.
// GB300 issues two FP64 FMAs a clock per SM, so the FP64 kernels are built
// around giving every lane its own entry: panels of 16 in registers, 4 x 4
// register tiles, triangular solves against inverted diagonal blocks, solves
// with a thread per row or per column instead of shuffle sums.
// One problem per block (the form before this one) left the large problems of
// a batch on one SM each: 160 squares of 8..96, 494 ms.
// Which code handles a front depends on its size alone and every entry's sum
// has a fixed order, so a problem's bits do not depend on the batch it is in.
#include <algorithm>
#include <cmath>

#include "forest.h"

namespace {

constexpr int kPan = 16;          // panel of the shared-memory fronts
constexpr int kWide = 64, kWs = kWide + 1;
constexpr int kBigT = 256;

template <typename T>
constexpr int small_limit() {
    return sizeof(T) == 8 ? 150 : 212;
}
inline int class_limit(int esize, int k) {
    const int l64[4] = {48, 72, 104, 150}, l32[4] = {48, 88, 140, 212};
    return esize == 8 ? l64[k] : l32[k];
}

struct CoopState {
    GridBarrier bar;
    int status, abort;
};

// Cholesky of a 16 x 16 block (kw x kw used) of a row-major matrix by one
// warp, a lane per row, rows in registers; inv gets the reciprocals of the
// diagonal.  False (all lanes alike): non-positive pivot.
template <typename T>
__device__ __forceinline__ bool chol16(T *A, int ld, int kw, T *inv) {
    const int lane = threadIdx.x & 31;
    T a[kPan];
#pragma unroll
    for (int j = 0; j < kPan; j++) a[j] = lane < kw && j <= lane ? A[lane * ld + j] : T(0);
    bool ok = true;
#pragma unroll
    for (int c = 0; c < kPan; c++) {
        if (c < kw && ok) {
            const T piv = __shfl_sync(0xffffffffu, a[c], c);
            if (!(piv > T(0)) || !isfinite((double)piv)) {
                ok = false;
            } else {
                const T iv = rsqrt(piv);   // one dependent chain instead of a square root and a division
                a[c] *= iv;
                if (lane == 0) inv[c] = iv;
#pragma unroll
                for (int j = c + 1; j < kPan; j++) {
                    const T l = __shfl_sync(0xffffffffu, a[c], j);
                    if (lane >= j) a[j] -= a[c] * l;
                }
            }
        }
    }
#pragma unroll
    for (int j = 0; j < kPan; j++)
        if (lane < kw && j <= lane) A[lane * ld + j] = a[j];
    return ok;
}

// one row against the factored 16 x 16 block D: x L^T = row
template <typename T>
__device__ __forceinline__ void row16(T *row, const T *D, int ld, int kw, const T *inv) {
    T x[kPan];
#pragma unroll
    for (int j = 0; j < kPan; j++) x[j] = j < kw ? row[j] : T(0);
    // right-looking: the updates of one step are independent of each other
#pragma unroll
    for (int j = 0; j < kPan; j++)
        if (j < kw) {
            x[j] *= inv[j];
#pragma unroll
            for (int l = j + 1; l < kPan; l++)
                if (l < kw) x[l] -= x[j] * D[l * ld + j];
        }
#pragma unroll
    for (int j = 0; j < kPan; j++)
        if (j < kw) row[j] = x[j];
}

// lower tile (bi, bj) of a linear index
__device__ __forceinline__ void tile_of(int q, int &bi, int &bj) {
    bi = (int)((sqrtf(8.0f * (float)q + 1.0f) - 1.0f) * 0.5f);
    while ((bi + 1) * (bi + 2) / 2 <= q) bi++;
    while (bi * (bi + 1) / 2 > q) bi--;
    bj = q - bi * (bi + 1) / 2;
}

// inverses of the nb x nb (<= 32) lower triangular blocks at rows b, b + 32, ...
// of L11 into their place in Lt: a warp per block, a lane per column
template <typename T>
__device__ __forceinline__ void invert_blocks(const T *A, int ld, int s, T *Lt, int warp, int nw) {
    const int lane = threadIdx.x & 31;
    for (int b = warp * 32; b < s; b += nw * 32) {
        const int nb = min(32, s - b);
        const T *D = A + (long long)b * ld + b;
        T w[32];
#pragma unroll
        for (int r = 0; r < 32; r++) {
            w[r] = T(0);
            if (r < nb) {
                T sum = T(0);
#pragma unroll
                for (int k = 0; k < r; k++) sum += D[r * ld + k] * w[k];
                const T iv = T(1) / D[r * ld + r];
                w[r] = r == lane ? iv : (r > lane ? -sum * iv : T(0));
                if (lane < nb) Lt[(long long)(b + r) * s + b + lane] = w[r];
            }
        }
    }
}

// ------------------------------------------------------------------ fronts in shared memory
template <typename T, int NT, bool WB>
__global__ void __launch_bounds__(NT) k_ff_small(FoDev m, const int2 *items, const double *vals, T *L, T *U, int *err) {
    extern __shared__ __align__(16) unsigned char fo_smem[];
    T *A = reinterpret_cast<T *>(fo_smem);
    __shared__ T inv[kPan];
    __shared__ int bad;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NW = NT / 32;
    const int2 it = items[blockIdx.x];
    const FoNode nd = m.node[it.y];
    const FoProb pr = m.prob[it.x];
    const int f = nd.f, s = nd.s, ld = f | 1;
    if (tid == 0) bad = *(volatile int *)(err + it.x);   // a lower level of this problem failed
    for (int k = tid; k < f * ld; k += NT) A[k] = T(0);
    __syncthreads();
    if (bad) return;
    for (int e = tid; e < nd.nentry; e += NT) {
        const int pos = m.ent_pos[nd.entry_off + e], r = pos / f;
        A[r * ld + pos - r * f] = (T)vals[pr.nnz0 + m.ent_rel[nd.entry_off + e]];
    }
    __syncthreads();
    for (int c = 0; c < nd.nchild; c++) {
        const FoNode cn = m.node[m.child[nd.child_off + c]];
        const int sc = cn.f - cn.s;
        const T *Uc = U + pr.Ub + cn.U_off;
        const int32_t *ex = m.ext + cn.ext_off;
        for (int a = warp; a < sc; a += NW) {
            const int pa = ex[a] * ld;
            for (int b = lane; b <= a; b += 32) A[pa + ex[b]] += Uc[(long long)a * sc + b];
        }
        __syncthreads();
    }
    for (int k0 = 0; k0 < s; k0 += kPan) {
        const int kw = min(kPan, s - k0), k1 = k0 + kw;
        T *D = A + k0 * ld + k0;
        if (warp == 0) {
            const bool ok = chol16(D, ld, kw, inv);
            if (lane == 0 && !ok) bad = 1;
        }
        __syncthreads();
        if (bad) {
            if (tid == 0) atomicCAS(err + it.x, 0, it.y + 1);
            return;
        }
        for (int i = k1 + tid; i < f; i += NT) row16(A + i * ld + k0, D, ld, kw, inv);
        __syncthreads();
        const int mm = f - k1, nt = (mm + 3) >> 2, ntiles = nt * (nt + 1) / 2;
        const T *Pt = A + k1 * ld + k0;
        for (int q = tid; q < ntiles; q += NT) {
            int bi, bj;
            tile_of(q, bi, bj);
            const int i0 = min(bi * 4, mm - 1), j0 = min(bj * 4, mm - 1);
            // rows past the end repeat the last one; they are not stored
            const T *xr[4], *yr[4];
#pragma unroll
            for (int a = 0; a < 4; a++) {
                xr[a] = Pt + min(i0 + a, mm - 1) * ld;
                yr[a] = Pt + min(j0 + a, mm - 1) * ld;
            }
            T acc[4][4];
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int b = 0; b < 4; b++) acc[a][b] = T(0);
            for (int t = 0; t < kw; t++) {
                T x[4], y[4];
#pragma unroll
                for (int a = 0; a < 4; a++) {
                    x[a] = xr[a][t];
                    y[a] = yr[a][t];
                }
#pragma unroll
                for (int a = 0; a < 4; a++)
#pragma unroll
                    for (int b = 0; b < 4; b++) acc[a][b] += x[a] * y[b];
            }
#pragma unroll
            for (int a = 0; a < 4; a++) {
                const int i = bi * 4 + a;
                T *Fi = A + (k1 + i) * ld + k1;
#pragma unroll
                for (int b = 0; b < 4; b++) {
                    const int j = bj * 4 + b;
                    if (i < mm && j <= i) Fi[j] -= acc[a][b];
                }
            }
        }
        __syncthreads();
    }
    T *Lt = L + pr.Lb + nd.L_off;
    if (WB) invert_blocks(A, ld, s, Lt, warp, NW);
    for (int i = warp; i < f; i += NW)
        for (int j = lane; j < s; j += 32)
            if (!WB || i >= s || (i >> 5) != (j >> 5)) Lt[(long long)i * s + j] = j <= i ? A[i * ld + j] : T(0);
    const int sc = f - s;
    T *Ut = U + pr.Ub + nd.U_off;
    for (int a = warp; a < sc; a += NW)
        for (int b = lane; b <= a; b += 32) Ut[(long long)a * sc + b] = A[(s + a) * ld + s + b];
}

// ------------------------------------------------------------------ fronts by groups of blocks
// One 64-column panel: (a) every block factors the diagonal block and its
// inverse W for itself in shared memory (the same arithmetic in every block:
// no barrier before (b)); (b) 32-row tiles of the rows below become A W^T;
// group barrier; (c) 64 x 64 tiles of the trailing lower triangle, 4 x 4
// entries a thread; group barrier.  With the diagonal block factored column
// by column by the whole block (three barriers a column) and a row of (b) a
// thread, a panel cost 80 us (FP32) to 250 us (FP64: 2,080 dependent FMAs a
// row on two blocks); now about 15 and 35 us.
template <typename T>
__device__ __forceinline__ bool diag64(T *Dg, T *W, T *tmp, T *inv, int *flag, int kw) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) *flag = 0;
    __syncthreads();
    for (int b = 0; b < kw; b += kPan) {
        const int bw = min(kPan, kw - b), b1 = b + bw;
        if (warp == 0) {
            const bool ok = chol16(Dg + b * kWs + b, kWs, bw, inv + b);
            if (lane == 0 && !ok) *flag = 1;
        }
        __syncthreads();
        if (*flag) return false;
        for (int i = b1 + tid; i < kw; i += kBigT) row16(Dg + i * kWs + b, Dg + b * kWs + b, kWs, bw, inv + b);
        __syncthreads();
        const int r = kw - b1;
        for (int q = tid; q < r * r; q += kBigT) {
            const int i = b1 + q / r, j = b1 + q % r;
            if (j <= i) {
                T s = T(0);
                for (int t = 0; t < bw; t++) s += Dg[i * kWs + b + t] * Dg[j * kWs + b + t];
                Dg[i * kWs + j] -= s;
            }
        }
        __syncthreads();
    }
    // W = L^-1: diagonal 16 x 16 blocks (a warp each, a lane per column), then
    // W_ij = -W_ii sum_k L_ik W_kj by block diagonals
    for (int q = tid; q < kWide * kWs; q += kBigT) W[q] = T(0);
    __syncthreads();
    const int nb = (kw + kPan - 1) / kPan;
    if (warp < nb && lane < kPan) {
        const int b = warp * kPan, bw = min(kPan, kw - b);
        T w[kPan];
#pragma unroll
        for (int r = 0; r < kPan; r++) {
            w[r] = T(0);
            if (r < bw) {
                T sum = T(0);
#pragma unroll
                for (int k = 0; k < r; k++) sum += Dg[(b + r) * kWs + b + k] * w[k];
                w[r] = r == lane ? inv[b + r] : (r > lane ? -sum * inv[b + r] : T(0));
                if (lane < bw) W[(b + r) * kWs + b + lane] = w[r];
            }
        }
    }
    __syncthreads();
    const int r = tid >> 4, c = tid & 15;   // 256 threads: one entry of a 16 x 16 block each
    for (int d = 1; d < nb; d++)
        for (int j = 0; j + d < nb; j++) {
            const int i = j + d;
            T s = T(0);
            for (int k = j * kPan; k < i * kPan; k++) s += Dg[(i * kPan + r) * kWs + k] * W[k * kWs + j * kPan + c];
            tmp[r * 17 + c] = s;
            __syncthreads();
            T w = T(0);
            for (int k = 0; k <= r; k++) w -= W[(i * kPan + r) * kWs + i * kPan + k] * tmp[k * 17 + c];
            W[(i * kPan + r) * kWs + j * kPan + c] = w;
            __syncthreads();
        }
    return true;
}

template <typename T, bool WB, typename Sync>
__device__ bool big_front(const FoDev &m, int2 it, const double *vals, T *L, T *U, T *F, T *P, int grank, int gblocks,
                          Sync sync, int *err, T *sm) {
    T *Dg = sm, *W = Dg + kWide * kWs, *At = W + kWide * kWs, *tmp = At + 32 * kWs, *inv = tmp + 16 * 17;
    __shared__ int flag;
    const int tid = threadIdx.x, lane = tid & 31;
    const long long gtid = (long long)grank * kBigT + tid, gsz = (long long)gblocks * kBigT;
    const long long gwarp = gtid >> 5, nwarps = gsz >> 5;
    const FoNode nd = m.node[it.y];
    const FoProb pr = m.prob[it.x];
    const int f = nd.f, s = nd.s;
    T *Lt = L + pr.Lb + nd.L_off;
    // a warp per row: zero it and add the rows of the children's update matrices
    // that fall on it (src names them), then the matrix entries
    const int2 *src = m.src + nd.front_off;
    for (long long i = gwarp; i < f; i += nwarps) {
        T *Fi = F + i * f;
        for (int j = lane; j <= i; j += 32) Fi[j] = T(0);
        __syncwarp();
        const int2 q = src[i];
        for (int c = 0; c < nd.nchild; c++) {
            const FoNode cn = m.node[m.child[nd.child_off + c]];
            const int sc = cn.f - cn.s;
            const long long ax = q.x - cn.uv_off, ay = q.y - cn.uv_off;
            const long long a = q.x >= 0 && ax >= 0 && ax < sc ? ax : (q.y >= 0 && ay >= 0 && ay < sc ? ay : -1);
            if (a < 0) continue;
            const T *Uc = U + pr.Ub + cn.U_off + a * sc;
            const int32_t *ex = m.ext + cn.ext_off;
            for (int b = lane; b <= a; b += 32) Fi[ex[b]] += Uc[b];
            __syncwarp();
        }
    }
    if (!sync()) return false;
    for (long long e = gtid; e < nd.nentry; e += gsz)
        F[m.ent_pos[nd.entry_off + e]] += (T)vals[pr.nnz0 + m.ent_rel[nd.entry_off + e]];
    if (!sync()) return false;
    for (int k0 = 0; k0 < s; k0 += kWide) {
        const int kw = min(kWide, s - k0), k1 = k0 + kw, mrows = f - k1;
        for (int q = tid; q < kWide * kWide; q += kBigT) {
            const int r = q / kWide, c = q - r * kWide;
            Dg[r * kWs + c] = (r < kw && c <= r) ? F[(long long)(k0 + r) * f + k0 + c] : T(0);
        }
        __syncthreads();
        if (!diag64(Dg, W, tmp, inv, &flag, kw)) {   // the same in every block of the group
            if (tid == 0) atomicCAS(err + it.x, 0, it.y + 1);
            return sync();
        }
        // (b) rows below: A W^T, written to F and to the panel P
        for (int i0 = k1 + grank * 32; i0 < f; i0 += gblocks * 32) {
            for (int q = tid; q < 32 * kWide; q += kBigT) {
                const int r = q / kWide, c = q - r * kWide;
                At[r * kWs + c] = (i0 + r < f && c < kw) ? F[(long long)(i0 + r) * f + k0 + c] : T(0);
            }
            __syncthreads();
            const int r = tid >> 3, c = tid & 7;
            T acc[8];
#pragma unroll
            for (int q = 0; q < 8; q++) {
                acc[q] = T(0);
                const int j = c + 8 * q;
                for (int l = 0; l <= j; l++) acc[q] += At[r * kWs + l] * W[j * kWs + l];
            }
            if (i0 + r < f) {
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const int j = c + 8 * q;
                    if (j < kw) {
                        F[(long long)(i0 + r) * f + k0 + j] = acc[q];
                        P[(long long)(i0 + r - k1) * kWs + j] = acc[q];
                    }
                }
            }
            __syncthreads();
        }
        if (!sync()) return false;
        // the factored diagonal block (and the inverses of its 32 x 32 blocks)
        // go out only now: before the barrier other blocks may still read the
        // unfactored one
        if (grank == 0)
            for (int q = tid; q < kw * kw; q += kBigT) {
                const int r = q / kw, c = q - r * kw;
                if (c <= r) F[(long long)(k0 + r) * f + k0 + c] = Dg[r * kWs + c];
                if (WB && (r >> 5) == (c >> 5)) Lt[(long long)(k0 + r) * s + k0 + c] = W[r * kWs + c];
            }
        __syncthreads();
        // (c) trailing update
        constexpr int TS = sizeof(T) == 8 ? 32 : 64, R = TS / 16;
        T *Ta = Dg, *Tb = W;
        const int nt = (mrows + TS - 1) / TS, ntiles = nt * (nt + 1) / 2;
        const int ty = tid >> 4, tx = tid & 15;
        for (int q = grank; q < ntiles; q += gblocks) {
            int bi, bj;
            tile_of(q, bi, bj);
            for (int e = tid; e < TS * kWide; e += kBigT) {
                const int r = e / kWide, c = e - r * kWide;
                const int ia = bi * TS + r, ib = bj * TS + r;
                Ta[r * kWs + c] = (ia < mrows && c < kw) ? P[(long long)ia * kWs + c] : T(0);
                Tb[r * kWs + c] = (ib < mrows && c < kw) ? P[(long long)ib * kWs + c] : T(0);
            }
            __syncthreads();
            T acc[R][R];
#pragma unroll
            for (int a = 0; a < R; a++)
#pragma unroll
                for (int b = 0; b < R; b++) acc[a][b] = T(0);
#pragma unroll 2
            for (int t = 0; t < kw; t++) {
                T x[R], y[R];
#pragma unroll
                for (int a = 0; a < R; a++) {
                    x[a] = Ta[(ty + 16 * a) * kWs + t];
                    y[a] = Tb[(tx + 16 * a) * kWs + t];
                }
#pragma unroll
                for (int a = 0; a < R; a++)
#pragma unroll
                    for (int b = 0; b < R; b++) acc[a][b] += x[a] * y[b];
            }
#pragma unroll
            for (int a = 0; a < R; a++) {
                const int i = bi * TS + ty + 16 * a;
                T *Fi = F + (long long)(k1 + i) * f + k1;
#pragma unroll
                for (int b = 0; b < R; b++) {
                    const int j = bj * TS + tx + 16 * b;
                    if (i < mrows && j <= i) Fi[j] -= acc[a][b];
                }
            }
            __syncthreads();
        }
        if (!sync()) return false;
    }
    for (long long i = gwarp; i < f; i += nwarps)
        for (int j = lane; j < s; j += 32) {
            const bool blk = i < s && (i >> 5) == (j >> 5);
            if (!WB || !blk) Lt[i * s + j] = j <= i ? F[i * f + j] : T(0);
            else if (j > i) Lt[i * s + j] = T(0);
        }
    const int sc = f - s;
    T *Ut = U + pr.Ub + nd.U_off;
    for (long long a = gwarp; a < sc; a += nwarps)
        for (int b = lane; b <= a; b += 32) Ut[a * sc + b] = F[(s + a) * f + s + b];
    return sync();   // F and P are reused by the group's next front
}

template <typename T, bool WB>
__global__ void __launch_bounds__(kBigT, 2) k_ff_big(FoDev m, const int2 *items, int count, const int4 *blocks, int slots,
                                                     const double *vals, T *L, T *U, T *pool, long long fslot,
                                                     long long pslot, CoopState *cs, int *err, long long spin) {
    const int4 b = blocks[blockIdx.x];
    // group b.x takes fronts b.x, b.x + groups, ...; its buffers are slot b.x (slots < groups only when
    // memory is short: then the groups of the later slots leave their fronts to the first ones)
    if (b.x >= slots) return;
    const int step = min(b.w, slots);
    CoopState *c = cs + b.x;
    extern __shared__ __align__(16) unsigned char fo_bsmem[];
    T *sm = reinterpret_cast<T *>(fo_bsmem);
    T *F = pool + (long long)b.x * (fslot + pslot), *P = F + fslot;
    auto sync = [&]() { return grid_barrier(&c->bar, b.z, &c->status, spin); };
    for (int q = b.x; q < count; q += step)
        if (!big_front<T, WB>(m, items[q], vals, L, U, F, P, b.y, b.z, sync, err, sm)) return;
}

// ------------------------------------------------------------------ FP64 solves
// 32 columns of L (rows i0 + 8 k) times 32 values, 8 rows a warp: four lanes a
// row, eight consecutive columns each, two shuffle additions a row.  FP64 pipe
// time 1.25 of the multiply-adds alone; a lane per row needs the tile staged
// through shared memory first (3 times slower on 100 to 500 rows), a warp per
// row spends five shuffle additions a row.
__device__ __forceinline__ double rows8(const double *Lt, int s, int i, bool in, int kb, int nb, const double *v) {
    const int c0 = (threadIdx.x & 3) * 8;
    double l[8];
    const double *r = Lt + (long long)i * s + kb + c0;
#pragma unroll
    for (int j = 0; j < 8; j++) l[j] = in && c0 + j < nb ? r[j] : 0.0;
    double a = 0.0;
#pragma unroll
    for (int j = 0; j < 8; j++)
        if (c0 + j < nb) a += l[j] * v[kb + c0 + j];   // beyond nb: structure rows, which other warps write meanwhile
    a += __shfl_xor_sync(0xffffffffu, a, 1);
    a += __shfl_xor_sync(0xffffffffu, a, 2);
    return a;
}

// Forward: the front's vector is its own entries of w minus the children's
// update entries, and their sum for its structure (gathered: src names the
// entries of each row); per 32 columns y = W v, then the remaining rows
// subtract (own) or add (structure) L y.  The structure part is the front's
// update vector.
template <int NT>
__global__ void __launch_bounds__(NT) k_fs_fwd(FoDev m, const int2 *items, const double *L, double *uv, double *w,
                                               const int *active) {
    extern __shared__ __align__(16) unsigned char fo_ssmem[];
    double *v = reinterpret_cast<double *>(fo_ssmem);   // f
    const int2 it = items[blockIdx.x];
    if (active && !active[it.x]) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NW = NT / 32;
    const FoNode nd = m.node[it.y];
    const FoProb pr = m.prob[it.x];
    const int f = nd.f, s = nd.s;
    const int32_t *fr = m.front + nd.front_off;
    const int2 *src = m.src + nd.front_off;
    const double *Lt = L + pr.Lb + nd.L_off;
    double *u = uv + pr.uvb;
    for (int k = tid; k < f; k += NT) {
        const int2 q = src[k];
        const double c = (q.x >= 0 ? u[q.x] : 0.0) + (q.y >= 0 ? u[q.y] : 0.0);
        v[k] = k < s ? w[pr.row0 + fr[k]] - c : c;
    }
    __syncthreads();
    for (int kb = 0; kb < s; kb += 32) {
        const int nb = min(32, s - kb);
        // y = W v: every warp its rows, written after all have read v
        constexpr int NY = 8 * NW < 32 ? 32 / (8 * NW) : 1;   // warps from 4 on have no row of these
        double y[NY];
#pragma unroll
        for (int q = 0; q < NY; q++) {
            const int r = (q * NW + warp) * 8 + (lane >> 2);
            y[q] = r < 32 ? rows8(Lt, s, kb + r, r < nb, kb, nb, v) : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < NY; q++) {
            const int r = (q * NW + warp) * 8 + (lane >> 2);
            if (r < nb && (lane & 3) == 0) v[kb + r] = y[q];
        }
        __syncthreads();
#pragma unroll 2
        for (int i0 = kb + nb + warp * 8; i0 < f; i0 += NW * 8) {
            const int i = i0 + (lane >> 2);
            const double a = rows8(Lt, s, i, i < f, kb, nb, v);
            if (i < f && (lane & 3) == 0) v[i] = i < s ? v[i] - a : v[i] + a;
        }
        __syncthreads();
    }
    for (int k = tid; k < s; k += NT) w[pr.row0 + fr[k]] = v[k];
    double *out = u + nd.uv_off;
    for (int k = s + tid; k < f; k += NT) out[k - s] = v[k];
}

// Backward: per 32 columns from the last, z = y - L^T x over the rows below
// (a lane per column, the warps split the rows), x = W^T z (warp 0, its part of
// W loaded before the sums are ready).
template <int NT>
__global__ void __launch_bounds__(NT) k_fs_bwd(FoDev m, const int2 *items, const double *L, double *w, const int *active) {
    extern __shared__ __align__(16) unsigned char fo_ssmem[];
    double *part = reinterpret_cast<double *>(fo_ssmem);   // NT / 32 x 32
    double *v = part + NT;
    const int2 it = items[blockIdx.x];
    if (active && !active[it.x]) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NW = NT / 32;
    const FoNode nd = m.node[it.y];
    const FoProb pr = m.prob[it.x];
    const int f = nd.f, s = nd.s;
    const int32_t *fr = m.front + nd.front_off;
    const double *Lt = L + pr.Lb + nd.L_off;
    for (int k = tid; k < f; k += NT) v[k] = w[pr.row0 + fr[k]];
    __syncthreads();
    for (int kb = ((s + 31) / 32 - 1) * 32; kb >= 0; kb -= 32) {
        const int nb = min(32, s - kb);
        const double *Lk = Lt + kb + lane;
        double wr[32];
        if (warp == 0) {
#pragma unroll
            for (int r = 0; r < 32; r++) wr[r] = r < nb && lane < nb ? Lk[(long long)(kb + r) * s] : 0.0;
        }
        double a = 0.0;
        if (lane < nb) {
#pragma unroll 8
            for (int i = kb + nb + warp; i < f; i += NW) a += Lk[(long long)i * s] * v[i];
        }
        part[tid] = a;
        __syncthreads();
        if (warp == 0) {
            double z = 0.0;
            if (lane < nb) {
                z = v[kb + lane];
                for (int g = 0; g < NW; g++) z -= part[g * 32 + lane];
            }
            double x = 0.0;
#pragma unroll
            for (int r = 0; r < 32; r++) x += wr[r] * __shfl_sync(0xffffffffu, z, r);
            if (lane < nb) v[kb + lane] = x;
        }
        __syncthreads();
    }
    for (int k = tid; k < s; k += NT) w[pr.row0 + fr[k]] = v[k];
}

template <typename V>
int fo_upload(grmp_context ctx, MfForest &F, const std::vector<V> &v, const V **out) {
    V *p = nullptr;
    const size_t bytes = std::max<size_t>(1, v.size()) * sizeof(V);
    int rc = grmp_alloc(ctx, (void **)&p, bytes);
    if (rc) return rc;
    F.bufs.push_back({p, bytes});
    *out = p;
    if (v.empty()) return GRMP_OK;
    cudaError_t e = cudaMemcpyAsync(p, v.data(), v.size() * sizeof(V), cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);   // the host vector is gone after the call
    return e == cudaSuccess ? GRMP_OK : grmp_cuda_fail(ctx, e, "multifrontal upload");
}

// groups of a level's large fronts with buffers of their own
constexpr size_t kPoolBound = (size_t)3 << 30;
constexpr int kMaxGroups = 160;
inline long long slot_elems(int maxf) { return (long long)maxf * maxf + (long long)maxf * kWs; }
inline int big_slots(const FoLevel &l, int num_sms, size_t poolb, int esize) {
    const long long fit = std::max<long long>(1, (long long)(poolb / (slot_elems(l.big.maxf) * esize)));
    return (int)std::min<long long>({(long long)l.big.count, fit, (long long)num_sms, (long long)kMaxGroups});
}

size_t pool_bytes(const MfForest &F, int num_sms, int esize) {
    size_t b = 0;
    for (const FoLevel &l : F.level)
        if (l.big.count)
            b = std::max<size_t>(b, (size_t)big_slots(l, num_sms, kPoolBound, esize) * slot_elems(l.big.maxf) * esize);
    return b;
}

int fo_storage(grmp_context ctx, MfForest *F, int esize) {
    if (F->esize == esize) return GRMP_OK;
    F->Lb = std::max<size_t>(1, F->L_size) * esize;
    F->Ub = std::max<size_t>(1, F->U_size) * esize;
    F->uvb = std::max<size_t>(1, F->uv_size) * esize;
    int rc = grmp_alloc(ctx, &F->L, F->Lb);
    if (!rc) rc = grmp_alloc(ctx, &F->U, F->Ub);
    if (!rc) rc = grmp_alloc(ctx, &F->uv, F->uvb);
    if (!rc) rc = grmp_alloc(ctx, &F->cs, kMaxGroups * sizeof(CoopState));
    if (rc) {
        grmp_free(ctx, F->L, F->Lb);
        grmp_free(ctx, F->U, F->Ub);
        grmp_free(ctx, F->uv, F->uvb);
        F->L = F->U = F->uv = F->cs = nullptr;
        return rc;
    }
    F->esize = esize;
    return GRMP_OK;
}

// Buffers of the large fronts, for one factorisation (nothing else needs them,
// and they can be larger than the factor).  Short of memory or budget: fewer
// groups of blocks, down to one front's.
int fo_pool(grmp_context ctx, MfForest *F, int esize) {
    size_t one = 256;
    for (const FoLevel &l : F->level)
        if (l.big.count) one = std::max<size_t>(one, (size_t)slot_elems(l.big.maxf) * esize);
    F->poolb = std::max<size_t>(one, pool_bytes(*F, ctx->num_sms, esize));
    int rc;
    while ((rc = F->poolb > one ? grmp_alloc_spare(ctx, &F->pool, F->poolb) : grmp_alloc(ctx, &F->pool, F->poolb)) &&
           F->poolb > one) {
        cudaGetLastError();
        F->poolb = std::max(one, F->poolb / 2);
    }
    if (!rc) ctx->last_error.clear();
    return rc;
}

template <typename T, int NT, bool WB>
void launch_small(grmp_context ctx, MfForest *F, const FoItems &it, const double *vals, int *err) {
    const size_t smem = (size_t)it.maxf * (it.maxf | 1) * sizeof(T);
    cudaFuncSetAttribute(k_ff_small<T, NT, WB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)((size_t)small_limit<T>() * (small_limit<T>() | 1) * sizeof(T)));
    k_ff_small<T, NT, WB><<<it.count, NT, smem, ctx->stream>>>(F->dev, it.d, vals, (T *)F->L, (T *)F->U, err);
    GRMP_LAUNCHED(ctx);
}

template <typename T, bool WB>
int fo_factor_levels(grmp_context ctx, MfForest *F, const double *vals, int *err) {
    cudaMemsetAsync(err, 0, (size_t)F->nprob * 4, ctx->stream);
    const size_t bsmem = ((size_t)2 * kWide * kWs + 32 * kWs + 16 * 17 + kWide) * sizeof(T);
    int coop = 0;
    cudaError_t e = cudaSuccess;
    for (const FoLevel &l : F->level) {
        for (int k = 0; k < 4; k++)
            if (l.small_[k].count) {
                if (k < 2) launch_small<T, 128, WB>(ctx, F, l.small_[k], vals, err);
                else launch_small<T, 256, WB>(ctx, F, l.small_[k], vals, err);
            }
        if (!l.big.count) continue;
        if (!coop) {
            cudaFuncSetAttribute(k_ff_big<T, WB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bsmem);
            coop = 1;
        }
        int slots = big_slots(l, ctx->num_sms, F->poolb, sizeof(T)), count = l.big.count;
        const int ng = slots;
        const int4 *blocks = l.blocks;
        cudaMemsetAsync(F->cs, 0, kMaxGroups * sizeof(CoopState), ctx->stream);
        FoDev dv = F->dev;
        const int2 *items = l.big.d;
        T *Lp = (T *)F->L, *Up = (T *)F->U, *pool = (T *)F->pool;
        long long fs = (long long)l.big.maxf * l.big.maxf, ps = (long long)l.big.maxf * kWs, spin = ctx->wait_limit;
        CoopState *cs = (CoopState *)F->cs;
        void *args[] = {&dv, &items, &count, &blocks, &slots, &vals, &Lp, &Up, &pool, &fs, &ps, &cs, &err, &spin};
        e = cudaLaunchCooperativeKernel((void *)k_ff_big<T, WB>, l.nblocks, kBigT, args, bsmem, ctx->stream);
        GRMP_LAUNCHED(ctx);
        std::vector<CoopState> hc(ng);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(hc.data(), cs, (size_t)ng * sizeof(CoopState), cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) break;
        for (auto &h : hc)
            if (h.status)
                return grmp_fail(ctx, GRMP_ERR_TIMEOUT, "multifrontal factorisation: a grid barrier wait timed out");
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    return e == cudaSuccess ? GRMP_OK : grmp_cuda_fail(ctx, e, "multifrontal factorisation");
}

template <typename T, bool WB>
int fo_factor(grmp_context ctx, MfForest *F, const double *vals, int *err) {
    int rc = fo_storage(ctx, F, sizeof(T));
    if (!rc) rc = fo_pool(ctx, F, sizeof(T));
    if (rc) return rc;
    rc = fo_factor_levels<T, WB>(ctx, F, vals, err);
    grmp_free(ctx, F->pool, F->poolb);
    F->pool = nullptr;
    return rc;
}

}  // namespace

FoNeed::FoNeed(const std::vector<const NdSymbolic *> &groups, int esize) {
    const int large = class_limit(esize, 3);
    for (const NdSymbolic *S : groups) {
        Group g{(size_t)(S->L_size + S->U_size + S->uv_size) * esize, 0, 0};
        for (size_t l = 0; l + 1 < S->level_ptr.size(); l++) {
            size_t level = 0;
            for (int q = S->level_ptr[l]; q < S->level_ptr[l + 1]; q++) {
                const int f = S->node[S->level_nodes[q]].f;
                if (f <= large) continue;
                level += (size_t)slot_elems(f) * esize;
                g.slot = std::max(g.slot, (size_t)slot_elems(f) * esize);
            }
            g.pool = std::max(g.pool, level);
        }
        of.push_back(g);
        tree += S->node.size() * sizeof(FoNode) + S->front.size() * 12 + (S->child.size() + S->ext.size()) * 4 + S->ent_rel.size() * 8;
    }
}
void FoNeed::add(int group) {
    fac += of[group].fac;
    pool += of[group].pool;
    slot = std::max(slot, of[group].slot);
}
size_t FoNeed::with(int group) const {
    return total(fac + of[group].fac, pool + of[group].pool, std::max(slot, of[group].slot));
}
size_t FoNeed::total(size_t fac, size_t pool, size_t slot) { return fac + std::max(slot, std::min(pool, kPoolBound / 4)); }

int grmp_forest_create(grmp_context ctx, const std::vector<const NdSymbolic *> &groups, const std::vector<FoProblem> &probs,
                       int esize, MfForest **out) {
    MfForest *F = new MfForest;
    *out = F;
    F->nprob = (int)probs.size();
    const int ng = (int)groups.size();
    std::vector<FoNode> node;
    std::vector<int32_t> front, child, ent_rel, ent_pos, ext;
    std::vector<int2> src;
    std::vector<int> node0(ng);
    std::vector<char> used(ng, 0);   // a part of a batch holds the trees of its own problems only
    for (const FoProblem &p : probs) used[p.group] = 1;
    size_t nlev = 0;
    for (int g = 0; g < ng; g++) {
        if (!used[g]) continue;
        const NdSymbolic &S = *groups[g];
        const int nb = (int)node.size(), fb = (int)front.size(), cb = (int)child.size(), eb = (int)ent_rel.size(),
                  xb = (int)ext.size();
        node0[g] = nb;
        for (int t = 0; t < S.nnodes; t++) {
            const NdNode &q = S.node[t];
            node.push_back(FoNode{q.s, q.f, q.front_off + fb, q.child_off + cb, q.nchild, q.entry_off + eb, q.nentry,
                                  q.ext_off + xb, (long long)q.L_off, (long long)q.U_off, (long long)S.uv_off[t]});
        }
        src.resize(src.size() + S.front.size(), make_int2(-1, -1));
        for (int t = 0; t < S.nnodes; t++) {
            const NdNode &q = S.node[t];
            for (int c = 0; c < q.nchild; c++) {
                const int ch = S.child[q.child_off + c];
                const NdNode &cn = S.node[ch];
                for (int a = 0; a < cn.f - cn.s; a++) {
                    int2 &d = src[(size_t)fb + q.front_off + S.ext[cn.ext_off + a]];
                    const int at = (int)(S.uv_off[ch] + a);
                    if (d.x < 0) d.x = at;
                    else if (d.y < 0) d.y = at;
                    else return grmp_fail(ctx, GRMP_ERR_UNSUPPORTED, "multifrontal: more than two children in a front");
                }
            }
        }
        front.insert(front.end(), S.front.begin(), S.front.end());
        for (int c : S.child) child.push_back(c + nb);
        ent_rel.insert(ent_rel.end(), S.ent_rel.begin(), S.ent_rel.end());
        ent_pos.insert(ent_pos.end(), S.ent_pos.begin(), S.ent_pos.end());
        ext.insert(ext.end(), S.ext.begin(), S.ext.end());
        F->max_f = std::max(F->max_f, S.max_f);
        F->max_s = std::max(F->max_s, S.max_s);
        nlev = std::max(nlev, S.level_ptr.size() - 1);
    }
    std::vector<FoProb> pr;
    for (const FoProblem &p : probs) {
        const NdSymbolic &S = *groups[p.group];
        pr.push_back(FoProb{p.row0, 0, p.nnz0, F->L_size, F->U_size, F->uv_size});
        F->L_size += S.L_size;
        F->U_size += S.U_size;
        F->uv_size += S.uv_size;
    }
    // items of each level and class, largest fronts first
    F->level.resize(nlev);
    int rc = GRMP_OK;
    for (size_t l = 0; l < nlev && !rc; l++) {
        std::vector<int2> cls[8];   // 0-3 small, 4 big, 5-7 solve classes
        int maxf[8] = {};
        for (int p = 0; p < F->nprob; p++) {
            const NdSymbolic &S = *groups[probs[p].group];
            if (l + 1 >= S.level_ptr.size()) continue;
            for (int q = S.level_ptr[l]; q < S.level_ptr[l + 1]; q++) {
                const int t = S.level_nodes[q], f = S.node[t].f;
                if (f == 0) continue;
                const int2 it = make_int2(p, node0[probs[p].group] + t);
                int k = 0;
                while (k < 4 && f > class_limit(esize, k)) k++;
                cls[k].push_back(it);
                maxf[k] = std::max(maxf[k], f);
                k = f <= kFoSolve[0] ? 5 : (f <= kFoSolve[1] ? 6 : 7);
                cls[k].push_back(it);
                maxf[k] = std::max(maxf[k], f);
            }
        }
        FoLevel &L = F->level[l];
        FoItems *to[8] = {&L.small_[0], &L.small_[1], &L.small_[2], &L.small_[3], &L.big, &L.solve[0], &L.solve[1], &L.solve[2]};
        for (int k = 0; k < 8; k++) {
            std::stable_sort(cls[k].begin(), cls[k].end(), [&](int2 a, int2 b) { return node[a.y].f > node[b.y].f; });
            to[k]->count = (int)cls[k].size();
            to[k]->maxf = maxf[k];
        }
        // few shared-memory fronts in the level: one launch for all classes (a class is a launch,
        // and one front's chain of panels is its time); largest first
        int nsmall = 0;
        for (int k = 0; k < 4; k++) nsmall += to[k]->count;
        if (nsmall <= 2 * ctx->num_sms)
            for (int k = 2; k >= 0; k--) {
                cls[3].insert(cls[3].end(), cls[k].begin(), cls[k].end());
                to[3]->count += to[k]->count;
                to[3]->maxf = std::max(to[3]->maxf, to[k]->maxf);
                to[k]->count = to[k]->maxf = 0;
                cls[k].clear();
            }
        for (int k = 0; k < 8 && !rc; k++)
            if (to[k]->count) rc = fo_upload(ctx, *F, cls[k], &to[k]->d);
        // large fronts: with at most one per SM each gets blocks in proportion to its flops (all run at
        // once, the largest is the level's time), else groups of two blocks take them in turn
        if (!rc && L.big.count) {
            const int nblk = 2 * ctx->num_sms, cnt = L.big.count;
            std::vector<int4> blk;
            if (cnt <= ctx->num_sms) {
                double tot = 0;
                std::vector<double> wt;
                for (int2 it : cls[4]) {
                    const FoNode &q = node[it.y];
                    wt.push_back((double)q.s * q.f * q.f);
                    tot += wt.back();
                }
                std::vector<int> nb(cnt, 1);
                int left = nblk - cnt;
                for (int i = 0; i < cnt; i++) {
                    const int add = std::min(left, (int)(wt[i] / tot * (nblk - cnt)));
                    nb[i] += add;
                }
                for (int b : nb) left -= b - 1;
                for (int i = 0; left > 0; i = (i + 1) % cnt, left--) nb[i]++;
                for (int i = 0; i < cnt; i++)
                    for (int r = 0; r < nb[i]; r++) blk.push_back(make_int4(i, r, nb[i], cnt));
            } else {
                const int g = nblk / 2;
                for (int i = 0; i < g; i++)
                    for (int r = 0; r < 2; r++) blk.push_back(make_int4(i, r, 2, g));
            }
            L.nblocks = (int)blk.size();
            rc = fo_upload(ctx, *F, blk, &L.blocks);
        }
    }
    if (!rc) rc = fo_upload(ctx, *F, node, &F->dev.node);
    if (!rc) rc = fo_upload(ctx, *F, front, &F->dev.front);
    if (!rc) rc = fo_upload(ctx, *F, child, &F->dev.child);
    if (!rc) rc = fo_upload(ctx, *F, ent_rel, &F->dev.ent_rel);
    if (!rc) rc = fo_upload(ctx, *F, ent_pos, &F->dev.ent_pos);
    if (!rc) rc = fo_upload(ctx, *F, ext, &F->dev.ext);
    if (!rc) rc = fo_upload(ctx, *F, src, &F->dev.src);
    if (!rc) rc = fo_upload(ctx, *F, pr, &F->dev.prob);
    return rc;
}

void grmp_forest_release(grmp_context ctx, MfForest *F) {
    if (!F->esize) return;
    grmp_free(ctx, F->L, F->Lb);
    grmp_free(ctx, F->U, F->Ub);
    grmp_free(ctx, F->uv, F->uvb);
    grmp_free(ctx, F->cs, kMaxGroups * sizeof(CoopState));
    F->L = F->U = F->uv = F->cs = nullptr;
    F->esize = 0;
}

void grmp_forest_free(grmp_context ctx, MfForest *F) {
    if (!F) return;
    for (auto &b : F->bufs) grmp_free(ctx, b.first, b.second);
    grmp_forest_release(ctx, F);
    delete F;
}

int grmp_forest_factor64(grmp_context ctx, MfForest *F, const double *vals, int *err) {
    return fo_factor<double, true>(ctx, F, vals, err);
}
int grmp_forest_factor32(grmp_context ctx, MfForest *F, const double *vals, int *err) {
    return fo_factor<float, false>(ctx, F, vals, err);
}

void grmp_forest_solve64(grmp_context ctx, MfForest *F, double *w, const int *active) {
    const double *L = (const double *)F->L;
    double *uv = (double *)F->uv;
    auto smem_f = [](int maxf) { return (size_t)maxf * 8; };
    auto smem_b = [](int nt, int maxf) { return ((size_t)nt + maxf) * 8; };
    grmp_allow_smem(k_fs_fwd<512>);
    grmp_allow_smem(k_fs_bwd<512>);
    for (size_t l = 0; l < F->level.size(); l++) {
        const FoItems *c = F->level[l].solve;
        if (c[2].count) k_fs_fwd<512><<<c[2].count, 512, smem_f(c[2].maxf), ctx->stream>>>(F->dev, c[2].d, L, uv, w, active);
        if (c[1].count) k_fs_fwd<128><<<c[1].count, 128, smem_f(c[1].maxf), ctx->stream>>>(F->dev, c[1].d, L, uv, w, active);
        if (c[0].count) k_fs_fwd<64><<<c[0].count, 64, smem_f(c[0].maxf), ctx->stream>>>(F->dev, c[0].d, L, uv, w, active);
        for (int k = 0; k < 3; k++) ctx->launches += c[k].count > 0;
    }
    for (size_t l = F->level.size(); l-- > 0;) {
        const FoItems *c = F->level[l].solve;
        if (c[2].count) k_fs_bwd<512><<<c[2].count, 512, smem_b(512, c[2].maxf), ctx->stream>>>(F->dev, c[2].d, L, w, active);
        if (c[1].count) k_fs_bwd<128><<<c[1].count, 128, smem_b(128, c[1].maxf), ctx->stream>>>(F->dev, c[1].d, L, w, active);
        if (c[0].count) k_fs_bwd<64><<<c[0].count, 64, smem_b(64, c[0].maxf), ctx->stream>>>(F->dev, c[0].d, L, w, active);
        for (int k = 0; k < 3; k++) ctx->launches += c[k].count > 0;
    }
}
