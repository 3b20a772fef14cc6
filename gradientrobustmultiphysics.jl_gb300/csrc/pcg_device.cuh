// Device building blocks of the persistent solvers: block and grid sums in a
// fixed order, the synchronisation policies (a cooperative grid or one
// thread-block cluster) and the CSR row loops.
#pragma once

#include <cooperative_groups.h>

#include <type_traits>

#include "grmp_internal.h"

namespace {

constexpr int PTPB = 256;   // threads per block of the persistent kernel
inline int nblk(long long n, int tpb = 256) { return (int)((n + tpb - 1) / tpb); }

struct WorkLayout {
    size_t vec, off_r64, off_part;
};

struct SolveState {
    GridBarrier bar;
    int status;
    int iters;
    int outer;
    int nearer;   // multilevel solves: x has a smaller residual than the start
    double relres;
};

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sum NV values over the block; result valid in all threads.  Warp sums,
// then warp 0 sums the per-warp values with the same fixed shuffle tree and
// publishes the totals: one thread's worth of additions per value instead of
// every thread re-adding all warps' values (on GB300 that redundant work lands
// on the narrow FP64 pipe).
template <int NV, typename T>
__device__ __forceinline__ void block_sum_t(T *v, T *sh /* [32*NV] */) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int k = 0; k < NV; k++) v[k] = warp_sum(v[k]);
    __syncthreads();
    if (lane == 0)
        for (int k = 0; k < NV; k++) sh[wid * NV + k] = v[k];
    __syncthreads();
    if (wid == 0) {
        T a[NV];
        for (int k = 0; k < NV; k++) a[k] = lane < nw ? sh[lane * NV + k] : T(0);
        for (int k = 0; k < NV; k++) a[k] = warp_sum(a[k]);
        if (lane == 0)
            for (int k = 0; k < NV; k++) sh[k] = a[k];
    }
    __syncthreads();
    for (int k = 0; k < NV; k++) v[k] = sh[k];
    __syncthreads();
}

template <int NV>
__device__ __forceinline__ void block_sum(double *v, double *sh /* [32*NV] */) {
    block_sum_t<NV, double>(v, sh);
}

// Write this block's partial sums, pass a grid barrier, then every block sums
// all partials in the same fixed order.  Returns false on a barrier timeout.
// The partial-sum area holds two buffers used alternately by successive
// reductions (`round` counts them): a block may start writing the next
// reduction's partials while a slower block still reads the previous ones,
// but it cannot reach the reduction after that before every block has left
// this one.
constexpr int kPartStride = 4 * 4096;   // doubles per buffer (4 values x up to 4096 blocks)

template <int NV>
__device__ __forceinline__ bool grid_sum(double *v, double *partial_area, double *sh, SolveState *st, int &round,
                                         long long spin) {
    double *partial = partial_area + (round++ & 1) * kPartStride;
    block_sum<NV>(v, sh);
    if (threadIdx.x == 0)
        for (int k = 0; k < NV; k++) partial[blockIdx.x * 4 + k] = v[k];
    if (!grid_barrier(&st->bar, gridDim.x, &st->status, spin)) return false;
    double acc[NV];
    for (int k = 0; k < NV; k++) acc[k] = 0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x)
        for (int k = 0; k < NV; k++) acc[k] += __ldcg(&partial[b * 4 + k]);
    block_sum<NV>(acc, sh);
    for (int k = 0; k < NV; k++) v[k] = acc[k];
    return true;
}

// FP32 versions for the inner iteration of the mixed solver: on GB300 the
// FP64 pipe issues about 2 operations per clock per SM, so double-precision
// shuffles and sums in every reduction of every iteration are not free.  The
// summation order is fixed as in the FP64 versions.
template <int NV>
__device__ __forceinline__ void block_sum_f(float *v, float *sh /* [32*NV] */) {
    block_sum_t<NV, float>(v, sh);
}

template <int NV>
__device__ __forceinline__ bool grid_sum_f(float *v, double *partial_area, float *sh, SolveState *st, int &round,
                                           long long spin) {
    float *partial = reinterpret_cast<float *>(partial_area + (round++ & 1) * kPartStride);
    block_sum_f<NV>(v, sh);
    if (threadIdx.x == 0)
        for (int k = 0; k < NV; k++) partial[blockIdx.x * 4 + k] = v[k];
    if (!grid_barrier(&st->bar, gridDim.x, &st->status, spin)) return false;
    float acc[NV];
    for (int k = 0; k < NV; k++) acc[k] = 0.f;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x)
        for (int k = 0; k < NV; k++) acc[k] += __ldcg(&partial[b * 4 + k]);
    block_sum_f<NV>(acc, sh);
    for (int k = 0; k < NV; k++) v[k] = acc[k];
    return true;
}

// Synchronisation policies of the persistent solvers.
//
// GridSync: a cooperative grid over the whole GPU; barriers and reductions
// through global memory (grid_barrier, grid_sum), every wait bounded.
//
// ClusterSync: the whole solve in ONE thread-block cluster (8 or 16 CTAs on
// one GPC) for problems whose matrix and vectors sit in L2: the barrier is
// the hardware cluster barrier (barrier.cluster.arrive.release / wait.acquire,
// the cluster's analogue of __syncthreads: it orders global and shared
// memory at cluster scope), and reductions read each CTA's partial sums out
// of that CTA's shared memory (distributed shared memory) instead of global
// memory.  Every CTA executes the same sequence of barriers -- all decisions
// come from sums that every CTA forms in the same fixed order -- so the
// barrier cannot wait on a CTA that took another path; finish() is a last
// barrier that keeps every CTA's shared memory alive until no CTA reads it.
struct GridSync {
    SolveState *st;
    double *part;
    long long spin;
    int round;
    __device__ __forceinline__ bool barrier() { return grid_barrier(&st->bar, gridDim.x, &st->status, spin); }
    template <int NV>
    __device__ __forceinline__ bool sum(double *v, double *sh) {
        return grid_sum<NV>(v, part, sh, st, round, spin);
    }
    template <int NV>
    __device__ __forceinline__ bool sumf(float *v, float *sh) {
        return grid_sum_f<NV>(v, part, sh, st, round, spin);
    }
    __device__ __forceinline__ void finish() {}
};

namespace cg = cooperative_groups;

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// Sum NV values (already block-summed, valid in every thread) over the CTAs
// of the cluster: thread 0 publishes them in `mine` (this reduction's buffer
// of two, used alternately as in grid_sum), the cluster barrier, then warp 0
// reads every CTA's copy in rank order and sums with a fixed shuffle tree.
template <int NV, typename T>
__device__ __forceinline__ void cluster_combine(T *v, T (*pub)[4], int par, T *sh) {
    if (threadIdx.x == 0)
        for (int k = 0; k < NV; k++) pub[par][k] = v[k];
    cluster_barrier();
    cg::cluster_group cl = cg::this_cluster();
    const int nb = (int)cl.num_blocks();
    if (threadIdx.x < 32) {
        T a[NV];
        for (int k = 0; k < NV; k++) a[k] = T(0);
        if ((int)threadIdx.x < nb) {
            const T *rp = cl.map_shared_rank(&pub[par][0], (unsigned)threadIdx.x);
            for (int k = 0; k < NV; k++) a[k] = rp[k];
        }
        for (int k = 0; k < NV; k++) a[k] = warp_sum(a[k]);
        if (threadIdx.x == 0)
            for (int k = 0; k < NV; k++) sh[k] = a[k];
    }
    __syncthreads();
    for (int k = 0; k < NV; k++) v[k] = sh[k];
    __syncthreads();
}

struct ClusterSync {
    SolveState *st;
    double *part;     // unused: partial sums live in shared memory
    long long spin;   // unused: the cluster barrier is a hardware barrier
    int round;
    __device__ __forceinline__ bool barrier() {
        cluster_barrier();
        return true;
    }
    template <int NV>
    __device__ __forceinline__ bool sum(double *v, double *sh) {
        __shared__ double pub[2][4];
        block_sum<NV>(v, sh);
        cluster_combine<NV, double>(v, pub, round++ & 1, sh);
        return true;
    }
    template <int NV>
    __device__ __forceinline__ bool sumf(float *v, float *sh) {
        __shared__ float pub[2][4];
        block_sum_f<NV>(v, sh);
        cluster_combine<NV, float>(v, pub, round++ & 1, sh);
        return true;
    }
    __device__ __forceinline__ void finish() { cluster_barrier(); }
};

template <bool CL>
using SyncOf = typename std::conditional<CL, ClusterSync, GridSync>::type;

constexpr int kClT = 1024;   // threads per CTA of the cluster solvers

// Row loop shared by the SpMV variants: groups of TPR lanes per row, each
// lane with U independent (column, value) loads per chunk.  With PIPE the
// loop is software pipelined over the grid-strided rows: while the gathers `x[col]` of the
// current row are in flight, the first chunk of the next row and the bounds
// of the row after it are already being loaded, so a warp keeps the matrix
// stream busy across the dependent gather.  Per-row summation order (chunk
// by chunk, u = 0..U-1 within a chunk, then the lane reduction) does not
// depend on the pipelining.  gather(c) returns x[c]; epi(r, s) consumes the
// row sum (lane 0 of the group).
// Matrix entry sources: CSR arrays (column indices and values apart), or
// the FP32 copy packed as (column, value bits) pairs, one 8-byte load each.
template <typename V>
struct CsrSource {
    const int32_t *__restrict__ cols;
    const V *__restrict__ vals;
    template <typename A>
    __device__ __forceinline__ void get(int idx, int &c, A &v) const {
        c = __ldg(cols + idx);
        v = (A)__ldg(vals + idx);
    }
};

struct PackedSource {
    const int2 *__restrict__ pack;
    __device__ __forceinline__ void get(int idx, int &c, float &v) const {
        const int2 p = __ldg(pack + idx);
        c = p.x;
        v = __int_as_float(p.y);
    }
};

template <int U, int TPR, typename A, typename S>
__device__ __forceinline__ void load_chunk(const S &src, int k, int e, int *c, A *v) {
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int idx = k + u * TPR;
        if (idx < e) {
            src.get(idx, c[u], v[u]);
        } else {
            c[u] = 0;
            v[u] = A(0);
        }
    }
}

template <int TPR, int U, bool PIPE, typename A, typename S, typename G, typename E>
__device__ __forceinline__ void spmv_rows(int n, const int32_t *__restrict__ rowptr, const S src, G gather, E epi) {
    constexpr int RPW = 32 / TPR;   // rows per warp per step
    constexpr int CH = TPR * U;
    const int lane = threadIdx.x & (TPR - 1);
    const int gin = (threadIdx.x & 31) / TPR;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int stride = ((gridDim.x * blockDim.x) >> 5) * RPW;
    if (!PIPE) {
        // plain: bounds, chunk loads and gathers of one row after another
        for (int base = warp * RPW; base < n; base += stride) {
            const int r = base + gin;
            A s = 0;
            if (r < n) {
                const int kb = __ldg(rowptr + r), e = __ldg(rowptr + r + 1);
                for (int k = kb + lane; k < e; k += CH) {
                    int c[U];
                    A v[U];
                    load_chunk<U, TPR>(src, k, e, c, v);
#pragma unroll
                    for (int u = 0; u < U; u++) s += v[u] * gather(c[u]);
                }
            }
#pragma unroll
            for (int o = TPR / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (r < n && lane == 0) epi(r, s);
        }
        return;
    }
    int r = warp * RPW + gin;
    int kb = 0, e = 0, kbn = 0, en = 0;
    if (r < n) {
        kb = __ldg(rowptr + r);
        e = __ldg(rowptr + r + 1);
    }
    if (r + stride < n) {
        kbn = __ldg(rowptr + r + stride);
        en = __ldg(rowptr + r + stride + 1);
    }
    int c[U];
    A v[U];
    load_chunk<U, TPR>(src, kb + lane, e, c, v);
    for (int base = warp * RPW; base < n; base += stride) {
        // next row: first chunk; the row after: bounds
        int cn[U];
        A vn[U];
        load_chunk<U, TPR>(src, kbn + lane, en, cn, vn);
        const int r2 = r + 2 * stride;
        int kb2 = 0, e2 = 0;
        if (r2 < n) {
            kb2 = __ldg(rowptr + r2);
            e2 = __ldg(rowptr + r2 + 1);
        }
        A s = 0;
#pragma unroll
        for (int u = 0; u < U; u++) s += v[u] * gather(c[u]);
        for (int k = kb + lane + CH; k < e; k += CH) {   // rows longer than one chunk
            int c2[U];
            A v2[U];
            load_chunk<U, TPR>(src, k, e, c2, v2);
#pragma unroll
            for (int u = 0; u < U; u++) s += v2[u] * gather(c2[u]);
        }
#pragma unroll
        for (int o = TPR / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (r < n && lane == 0) epi(r, s);
        r += stride;
        kb = kbn;
        e = en;
        kbn = kb2;
        en = e2;
#pragma unroll
        for (int u = 0; u < U; u++) {
            c[u] = cn[u];
            v[u] = vn[u];
        }
    }
}

// y = A x over the rows of this grid.  If DOT, returns this thread's share
// of sum_r w[r]*y[r].  If RESID, y = b - A x (and DOT gives sum y^2).  The
// matrix is read-only for the whole solve (non-coherent path); x is written
// by other blocks between barriers (coherent loads).
template <int TPR, int U, bool PIPE, typename V, typename X, typename Y, bool DOT, bool RESID>
__device__ __forceinline__ double spmv_grid(int n, const int32_t *__restrict__ rowptr, const int32_t *__restrict__ cols,
                                            const V *__restrict__ vals, const X *x, Y *y, const Y *w,
                                            const double *b) {
    using A = typename std::conditional<sizeof(V) == 8, double, float>::type;
    double dot = 0;
    A dacc = 0;
    spmv_rows<TPR, U, PIPE, A>(
        n, rowptr, CsrSource<V>{cols, vals}, [&](int c) { return (A)x[c]; },
        [&](int r, A s) {
            if (RESID) {
                double v = b[r] - (double)s;
                y[r] = (Y)v;
                if (DOT) dot += v * v;
            } else {
                y[r] = (Y)s;
                if (DOT) dacc += (A)w[r] * s;   // FP32 partial in the FP32 path
            }
        });
    return dot + (double)dacc;
}

}  // namespace
