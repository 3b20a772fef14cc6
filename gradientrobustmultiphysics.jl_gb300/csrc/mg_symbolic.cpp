// Patterns of the multilevel preconditioner's hierarchy (mg.cu), built once
// per matrix pattern on the host cores.
//
// Step 0 of a P2 space interpolates from the vertices: the P1 functions are
// in the P2 space, with values 1 at their vertex and 1/2 at the midpoints of
// its edges.  Every other step aggregates: a row whose neighbours are all
// free takes them as one aggregate, rows left over join an aggregate next to
// them (Vanek, Mandel, Brezina 1996).  The vertex level keeps only couplings
// that P1 stiffness has on some cell: on right angles (squares split in triangles, Kuhn
// cubes) half of the neighbours do not couple, and aggregates that take them
// in span two couplings where the smoothed prolongation reaches one (128 x
// 128: 56 iterations with them, about half without).  Patterns include the DoFs that a call
// fixes later (they are masked by values), so one hierarchy serves every set
// of boundary DoFs.
#include <algorithm>
#include <cmath>
#include <thread>

#include "mg_symbolic.h"

namespace {

int host_threads(int n) {
    const int hw = std::max(1, (int)std::thread::hardware_concurrency());
    return std::max(1, std::min({hw, 16, n / 4096}));
}

// out row i = sorted distinct columns that fn(i, add) names; rows in parallel
template <typename F>
void build_rows(int n, int ncols, MgCsr *out, F fn) {
    const int nt = host_threads(n);
    std::vector<std::vector<int32_t>> part(nt);
    out->rp.assign((size_t)n + 1, 0);
    auto work = [&](int t) {
        const int i0 = (int)((long long)n * t / nt), i1 = (int)((long long)n * (t + 1) / nt);
        std::vector<int> mark(ncols, -1);
        std::vector<int32_t> &c = part[t];
        for (int i = i0; i < i1; i++) {
            const size_t b = c.size();
            fn(i, [&](int j) {
                if (mark[j] != i) {
                    mark[j] = i;
                    c.push_back(j);
                }
            });
            std::sort(c.begin() + b, c.end());
            out->rp[(size_t)i + 1] = (int32_t)(c.size() - b);
        }
    };
    std::vector<std::thread> pool;
    for (int t = 1; t < nt; t++) pool.emplace_back(work, t);
    work(0);
    for (auto &t : pool) t.join();
    for (int i = 0; i < n; i++) out->rp[i + 1] += out->rp[i];
    out->ci.resize(out->rp[n]);
    for (int t = 0; t < nt; t++)
        std::copy(part[t].begin(), part[t].end(), out->ci.begin() + out->rp[(size_t)((long long)n * t / nt)]);
}

void transpose(int n, int nc, const MgCsr &A, MgCsr *T, std::vector<int32_t> *perm) {
    T->rp.assign((size_t)nc + 1, 0);
    for (int32_t c : A.ci) T->rp[(size_t)c + 1]++;
    for (int c = 0; c < nc; c++) T->rp[c + 1] += T->rp[c];
    T->ci.resize(A.ci.size());
    perm->resize(A.ci.size());
    std::vector<int32_t> at(T->rp.begin(), T->rp.end() - 1);
    for (int i = 0; i < n; i++)
        for (int k = A.rp[i]; k < A.rp[i + 1]; k++) {
            const int q = at[A.ci[k]]++;
            T->ci[q] = i;
            (*perm)[q] = k;
        }
}

// aggregates in row order; returns their number
int aggregate(int n, const int32_t *rp, const int32_t *ci, std::vector<int32_t> *agg) {
    std::vector<int32_t> &a = *agg;
    a.assign(n, -1);
    int na = 0;
    for (int i = 0; i < n; i++) {
        if (a[i] >= 0) continue;
        bool free_ = true;
        for (int k = rp[i]; k < rp[i + 1] && free_; k++) free_ = a[ci[k]] < 0;
        if (!free_) continue;
        for (int k = rp[i]; k < rp[i + 1]; k++) a[ci[k]] = na;
        a[i] = na++;
    }
    // a leftover row joins the aggregate that most of its neighbours are in
    // (of the first pass; the lowest of equals)
    std::vector<int32_t> second(n, -1);
    std::vector<int> cnt(na, 0);
    for (int i = 0; i < n; i++) {
        if (a[i] >= 0) continue;
        int best = -1;
        for (int k = rp[i]; k < rp[i + 1]; k++) {
            const int g = a[ci[k]];
            if (g < 0) continue;
            cnt[g]++;
            if (best < 0 || cnt[g] > cnt[best] || (cnt[g] == cnt[best] && g < best)) best = g;
        }
        for (int k = rp[i]; k < rp[i + 1]; k++)
            if (a[ci[k]] >= 0) cnt[a[ci[k]]] = 0;
        second[i] = best;
    }
    for (int i = 0; i < n; i++)
        if (a[i] < 0) a[i] = second[i] >= 0 ? second[i] : na++;
    return na;
}

// Drops from the vertex level's pattern the pairs that have no P1 stiffness on
// any of their cells: a statement about the mesh that holds for every
// coefficient, so one hierarchy serves them all.  (Not the pairs whose cells
// cancel for the unit coefficient, as the diagonals of isosceles trapezoids:
// they couple as soon as the coefficient varies, and a coupling that the
// pattern lacks goes to the diagonal, which then need not stay positive.)
void filter_vertex_level(MgStep *s, int dim, int ncells, int ld, const int32_t *celldofs, const std::vector<int32_t> &vert,
                         const double *coords, const int32_t *cells) {
    const int nv = dim + 1, nc = s->nc;
    std::vector<int32_t> ptr((size_t)nc + 1, 0);
    for (long long c = 0; c < ncells; c++)
        for (int v = 0; v < nv; v++) ptr[vert[celldofs[c * ld + v]] + 1]++;
    for (int i = 0; i < nc; i++) ptr[i + 1] += ptr[i];
    std::vector<int32_t> inc(ptr[nc]), at(ptr.begin(), ptr.end() - 1);
    for (long long c = 0; c < ncells; c++)
        for (int v = 0; v < nv; v++) inc[at[vert[celldofs[c * ld + v]]]++] = (int32_t)(c * 4 + v);
    std::vector<double> K(s->Ac.ci.size(), 0.0), diag(nc, 0.0);
    const int nt = host_threads(nc);
    auto rows = [&](int t, auto fn) {
        for (int i = (int)((long long)nc * t / nt); i < (int)((long long)nc * (t + 1) / nt); i++) fn(i);
    };
    auto parallel = [&](auto fn) {
        std::vector<std::thread> pool;
        for (int t = 1; t < nt; t++) pool.emplace_back([&, t] { rows(t, fn); });
        rows(0, fn);
        for (auto &t : pool) t.join();
    };
    parallel([&](int i) {
        for (int q = ptr[i]; q < ptr[i + 1]; q++) {
            const long long c = inc[q] >> 2;
            const int a = inc[q] & 3;
            double E[3][3], G[4][3] = {}, det;
            const double *x0 = coords + (size_t)cells[c * nv] * dim;
            for (int j = 0; j < dim; j++)
                for (int k = 0; k < dim; k++) E[j][k] = coords[(size_t)cells[c * nv + j + 1] * dim + k] - x0[k];
            if (dim == 2) {
                det = E[0][0] * E[1][1] - E[0][1] * E[1][0];
                G[1][0] = E[1][1], G[1][1] = -E[1][0];
                G[2][0] = -E[0][1], G[2][1] = E[0][0];
            } else {
                for (int j = 0; j < 3; j++) {
                    const double *u = E[(j + 1) % 3], *w = E[(j + 2) % 3];
                    for (int k = 0; k < 3; k++)
                        G[j + 1][k] = u[(k + 1) % 3] * w[(k + 2) % 3] - u[(k + 2) % 3] * w[(k + 1) % 3];
                }
                det = E[0][0] * G[1][0] + E[0][1] * G[1][1] + E[0][2] * G[1][2];
            }
            for (int k = 0; k < dim; k++)
                for (int j = 1; j <= dim; j++) G[0][k] -= G[j][k];
            for (int b = 0; b < nv; b++) {
                double d = 0;
                for (int k = 0; k < dim; k++) d += G[a][k] * G[b][k];
                const int J = vert[celldofs[c * ld + b]];
                const int32_t *r = s->Ac.ci.data() + s->Ac.rp[i], *re = s->Ac.ci.data() + s->Ac.rp[i + 1];
                const int32_t *f = std::lower_bound(r, re, J);
                if (f != re && *f == J) K[f - s->Ac.ci.data()] += std::fabs(d) / (det != 0 ? std::fabs(det) : 1.0);
            }
        }
        for (int k = s->Ac.rp[i]; k < s->Ac.rp[i + 1]; k++)
            if (s->Ac.ci[k] == i) diag[i] = K[k];
    });
    MgCsr F;
    build_rows(nc, nc, &F, [&](int i, auto add) {
        for (int k = s->Ac.rp[i]; k < s->Ac.rp[i + 1]; k++) {
            const int j = s->Ac.ci[k];
            if (j == i || K[k] > 1e-6 * std::sqrt(diag[i] * diag[j])) add(j);
        }
    });
    s->filtered = F.ci.size() < s->Ac.ci.size();
    if (s->filtered) s->Ac = std::move(F);
}

void products(MgStep *s, const int32_t *rp, const int32_t *ci) {
    const MgCsr &P = s->P;
    build_rows(s->n, s->nc, &s->AP, [&](int i, auto add) {
        for (int k = rp[i]; k < rp[i + 1]; k++)
            for (int q = P.rp[ci[k]]; q < P.rp[ci[k] + 1]; q++) add(P.ci[q]);
    });
    transpose(s->n, s->nc, P, &s->R, &s->Rperm);
    build_rows(s->nc, s->nc, &s->Ac, [&](int I, auto add) {
        add(I);
        for (int k = s->R.rp[I]; k < s->R.rp[I + 1]; k++) {
            const int i = s->R.ci[k];
            for (int q = s->AP.rp[i]; q < s->AP.rp[i + 1]; q++) add(s->AP.ci[q]);
        }
    });
}

}  // namespace

int mg_symbolic_build(int n, const int32_t *rp, const int32_t *ci, int dim, int ncells, int ld, const int32_t *celldofs,
                      const double *coords, const int32_t *cells, bool cell_terms, bool fine_q, MgSymbolic *S) {
    S->step.clear();
    const int32_t *crp = rp, *cci = ci;
    int cn = n;
    while ((cn > kMgBottom || S->step.empty()) && (int)S->step.size() + 1 < kMgMaxLevels) {
        MgStep s;
        s.n = cn;
        std::vector<int32_t> vert;
        if (S->step.empty() && celldofs) {
            // coarse number of each vertex DoF, ascending; edge DoFs get their two vertices
            const int nv = dim + 1;
            std::vector<int32_t> e0(n, -1), e1(n, -1);
            vert.assign(n, -1);
            for (long long c = 0; c < ncells; c++)
                for (int v = 0; v < nv; v++) vert[celldofs[c * ld + v]] = 0;
            const int ed2[3][2] = {{0, 1}, {1, 2}, {2, 0}};
            const int ed3[6][2] = {{0, 1}, {0, 2}, {0, 3}, {1, 2}, {1, 3}, {2, 3}};
            const int ne = dim == 2 ? 3 : 6;
            for (int i = 0, k = 0; i < n; i++)
                if (vert[i] == 0) vert[i] = k++, s.nc = k;
            for (long long c = 0; c < ncells; c++)
                for (int e = 0; e < ne; e++) {
                    const int32_t *d = celldofs + c * ld;
                    const int i = d[nv + e];
                    e0[i] = vert[d[dim == 2 ? ed2[e][0] : ed3[e][0]]];
                    e1[i] = vert[d[dim == 2 ? ed2[e][1] : ed3[e][1]]];
                }
            s.geometric = true;
            for (int i = 0; i < n && s.geometric; i++)   // each DoF is a vertex or an edge
                s.geometric = (vert[i] >= 0) != (e0[i] >= 0) && (vert[i] >= 0 || e0[i] != e1[i]);
            if (s.geometric)
                build_rows(n, s.nc, &s.P, [&](int i, auto add) {
                    if (vert[i] >= 0) {
                        add(vert[i]);
                    } else {
                        add(e0[i]);
                        add(e1[i]);
                    }
                });
        }
        if (!s.geometric) {
            s.nc = aggregate(cn, crp, cci, &s.agg);
            if (s.nc > 0.7 * cn) break;   // does not coarsen further
            build_rows(cn, s.nc, &s.P, [&](int i, auto add) {
                add(s.agg[i]);
                for (int k = crp[i]; k < crp[i + 1]; k++) add(s.agg[cci[k]]);
            });
        }
        products(&s, crp, cci);
        if (s.geometric && cell_terms) filter_vertex_level(&s, dim, ncells, ld, celldofs, vert, coords, cells);
        if (fine_q || !S->step.empty()) transpose(s.n, s.nc, s.AP, &s.QT, &s.QTperm);
        cn = s.nc;
        S->step.push_back(std::move(s));
        crp = S->step.back().Ac.rp.data();   // stays valid: vectors keep their storage when the step is moved
        cci = S->step.back().Ac.ci.data();
    }
    return S->step.empty() ? 1 : 0;
}
