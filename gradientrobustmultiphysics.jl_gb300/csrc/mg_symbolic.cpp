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
// 128: 56 iterations with them, about half without).
//
// On stretched meshes the neighbours are not alike: the error that the
// smoother leaves is smooth along the short cell sides only, and aggregates
// that span long sides cannot represent it, nor can the vertices of P2 cells
// (160 x 160 P1 on strips 1 : 10, 1 : 30 and 1 : 100: 81, 226 and 510 iterations, 19
// on the square; 80 x 80 P2 98, 272 and 531).  There a row aggregates with strong
// neighbours only, on every level and P2's first one too: those whose stiffness
// for the unit coefficient exceeds kStrong of the diagonal (half of that on
// each coarser level, as in the paper), and the prolongation adds weak
// couplings to the row's own aggregate: 18 to 27 iterations on the P1 strips and
// graded meshes, 23 to 25 on the P2 strips; plates and rods of 40^3 P1 cubes 14 to 20
// (118 at 1 : 20 before), a P2 plate 1 : 20 of 20^3 cubes 51 (157 before).  Patterns include the DoFs that a call
// fixes later (they are masked by values), so one hierarchy serves every set
// of boundary DoFs.
#include <algorithm>
#include <cmath>
#include <exception>
#include <mutex>
#include <thread>

#include "mg_symbolic.h"

namespace {

// P1 and coarse levels: 0.05 takes 28 iterations on a strip 1 : 3, 0.08 16; 0.2 leaves nothing strong on Kuhn
// cubes.  P2: 0.08 takes 38 iterations on a strip 1 : 30 and 105 on a plate 1 : 20, 0.2 24 and 36.
constexpr double kStrong = 0.08, kStrongP2 = 0.2;

int host_threads(int n) {
    const int hw = std::max(1, (int)std::thread::hardware_concurrency());
    return std::max(1, std::min({hw, 16, n / 4096}));
}

// work(0), ..., work(nt - 1), a thread each; what one throws is thrown here
// after all have ended.  Where threads cannot be had this one does their work.
template <typename F>
void run_threads(int nt, F work) {
    std::exception_ptr thrown;
    std::mutex mu;
    auto guarded = [&](int t) {
        try {
            work(t);
        } catch (...) {
            std::lock_guard<std::mutex> lk(mu);
            if (!thrown) thrown = std::current_exception();
        }
    };
    std::vector<std::thread> pool;
    pool.reserve(nt);
    int t = 1;
    try {
        for (; t < nt; t++) pool.emplace_back(guarded, t);
    } catch (const std::exception &) {
    }
    guarded(0);
    for (; t < nt; t++) guarded(t);
    for (auto &p : pool) p.join();
    if (thrown) std::rethrow_exception(thrown);
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
    run_threads(nt, work);
    for (int i = 0; i < n; i++) out->rp[i + 1] += out->rp[i];
    out->ci.resize(out->rp[n]);
    for (int t = 0; t < nt; t++)
        std::copy(part[t].begin(), part[t].end(), out->ci.begin() + out->rp[(size_t)((long long)n * t / nt)]);
}

template <typename F>
void parallel_rows(int n, F fn) {
    const int nt = host_threads(n);
    run_threads(nt, [&](int t) {
        for (int i = (int)((long long)n * t / nt); i < (int)((long long)n * (t + 1) / nt); i++) fn(i);
    });
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

// vertices of the P2 edge functions
constexpr int kEdge2[3][2] = {{0, 1}, {1, 2}, {2, 0}};
constexpr int kEdge3[6][2] = {{0, 1}, {0, 2}, {0, 3}, {1, 2}, {1, 3}, {2, 3}};

// Entry (a, b) of a cell's P1 (p2 = false) or P2 stiffness from h_ij =
// |T| grad lambda_i . grad lambda_j (assemble.cu derives the P2 form).
double local_stiffness(int dim, bool p2, const double h[4][4], int a, int b) {
    const int nv = dim + 1;
    if (!p2) return h[a][b];
    const double e = 16.0 / (nv * (nv + 1)), c = 1.0 - 8.0 / nv, g = e - 4.0 / nv;
    if (a < nv && b < nv) return (a == b ? 2 * e + c : e + c) * h[a][b];
    if (a < nv) std::swap(a, b);   // a: an edge
    const int i = dim == 2 ? kEdge2[a - nv][0] : kEdge3[a - nv][0], j = dim == 2 ? kEdge2[a - nv][1] : kEdge3[a - nv][1];
    if (b < nv) return g * (h[i][b] + h[j][b]) + (b == i || b == j ? e * h[i][j] : 0.0);
    const int k = dim == 2 ? kEdge2[b - nv][0] : kEdge3[b - nv][0], l = dim == 2 ? kEdge2[b - nv][1] : kEdge3[b - nv][1];
    double s = h[i][k] + h[j][k] + h[i][l] + h[j][l];
    if (k == i) s += h[j][l];
    if (l == i) s += h[j][k];
    if (k == j) s += h[i][l];
    if (l == j) s += h[i][k];
    return e * s;
}

// Contributions of the cells to the stiffness of the unit coefficient, P2 (all
// local DoFs) or P1 (the vertex DoFs), in the pattern A of n rows; row[d]: row
// of the DoF d.  Mode Sum: their sums; Size: the sums of their absolute values.
enum class Mode { Sum, Size };
std::vector<double> unit_stiffness(Mode mode, int n, const MgCsr &A, const MgCells &m, bool p2,
                                   const std::vector<int32_t> &row) {
    const int dim = m.dim, nv = dim + 1, nb = p2 ? (dim == 2 ? 6 : 10) : nv;
    std::vector<int64_t> ptr((size_t)n + 1, 0);
    for (long long c = 0; c < m.ncells; c++)
        for (int v = 0; v < nb; v++) ptr[row[m.celldofs[c * m.ld + v]] + 1]++;
    for (int i = 0; i < n; i++) ptr[i + 1] += ptr[i];
    std::vector<int32_t> inc(ptr[n]);   // cells of each row, ascending
    std::vector<int64_t> at(ptr.begin(), ptr.end() - 1);
    for (long long c = 0; c < m.ncells; c++)
        for (int v = 0; v < nb; v++) inc[at[row[m.celldofs[c * m.ld + v]]]++] = (int32_t)c;
    std::vector<double> K(A.ci.size(), 0.0);
    parallel_rows(n, [&](int i) {
        int a = 0;
        for (int64_t q = ptr[i]; q < ptr[i + 1]; q++) {
            const long long c = inc[q];
            a = q > ptr[i] && inc[q - 1] == c ? a + 1 : 0;   // the row's function in the cell (the next one if it has two)
            while (row[m.celldofs[c * m.ld + a]] != i) a++;
            double E[3][3], G[4][3] = {}, h[4][4], det;
            const double *x0 = m.coords + (size_t)m.cells[c * nv] * dim;
            for (int j = 0; j < dim; j++)
                for (int k = 0; k < dim; k++) E[j][k] = m.coords[(size_t)m.cells[c * nv + j + 1] * dim + k] - x0[k];
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
            for (int j = p2 ? 0 : a; j < (p2 ? nv : a + 1); j++)   // (P1: the row's own)
                for (int l = 0; l < nv; l++) {
                    double d = 0;
                    for (int k = 0; k < dim; k++) d += G[j][k] * G[l][k];
                    h[j][l] = d / (det != 0 ? std::fabs(det) : 1.0);   // the common factor 1 / dim! does not matter
                }
            for (int b = 0; b < nb; b++) {
                const int J = row[m.celldofs[c * m.ld + b]];
                const int32_t *r = A.ci.data() + A.rp[i], *re = A.ci.data() + A.rp[i + 1];
                const int32_t *f = std::lower_bound(r, re, J);
                if (f == re || *f != J) continue;
                const double v = local_stiffness(dim, p2, h, a, b);
                K[f - A.ci.data()] += mode == Mode::Size ? std::fabs(v) : v;
            }
        }
    });
    return K;
}

// the pattern's pairs whose entry exceeds theta times the two diagonal entries' mean
MgCsr strong_pairs(int n, const MgCsr &A, const std::vector<double> &K, double theta) {
    std::vector<double> d(n, 0.0);
    parallel_rows(n, [&](int i) {
        for (int k = A.rp[i]; k < A.rp[i + 1]; k++)
            if (A.ci[k] == i) d[i] = std::fabs(K[k]);
    });
    MgCsr F;
    build_rows(n, n, &F, [&](int i, auto add) {
        for (int k = A.rp[i]; k < A.rp[i + 1]; k++) {
            const int j = A.ci[k];
            if (j == i || std::fabs(K[k]) > theta * std::sqrt(d[i] * d[j])) add(j);
        }
    });
    return F;
}

// Drops from the vertex level's pattern the pairs that have no P1 stiffness on
// any of their cells: a statement about the mesh that holds for every
// coefficient, so one hierarchy serves them all.  (Not the pairs whose cells
// cancel for the unit coefficient, as the diagonals of isosceles trapezoids:
// they couple as soon as the coefficient varies, and a coupling that the
// pattern lacks goes to the diagonal, which then need not stay positive.)
void filter_vertex_level(MgStep *s, const MgCells &m, const std::vector<int32_t> &vert) {
    const std::vector<double> K = unit_stiffness(Mode::Size, s->nc, s->Ac, m, false, vert);
    s->Ac = strong_pairs(s->nc, s->Ac, K, 1e-6);
}

// The next level's unit stiffness, P^T K P with P = (I - w D K) P_agg as on the
// device: couplings to aggregates that a row of P lacks go to its own.
std::vector<double> coarse_stiffness(const MgStep &s, const MgCsr &A, const std::vector<double> &K) {
    const MgCsr &P = s.P, &AP = s.AP;
    std::vector<double> pv(P.ci.size()), av(AP.ci.size()), cv(s.Ac.ci.size());
    auto find = [](const MgCsr &M, int i, int c) {
        const int32_t *b = M.ci.data() + M.rp[i], *e = M.ci.data() + M.rp[i + 1], *f = std::lower_bound(b, e, c);
        return f != e && *f == c ? (int)(f - M.ci.data()) : -1;
    };
    parallel_rows(s.n, [&](int i) {
        double sum = 0.0;
        for (int k = A.rp[i]; k < A.rp[i + 1]; k++) sum += std::fabs(K[k]);
        const double w = sum > 0 ? kMgProlong / sum : 0.0;
        const int own = find(P, i, s.agg[i]);
        pv[own] += 1.0;
        for (int k = A.rp[i]; k < A.rp[i + 1]; k++) {
            const int q = find(P, i, s.agg[A.ci[k]]);
            pv[q < 0 ? own : q] -= w * K[k];
        }
    });
    parallel_rows(s.n, [&](int i) {
        for (int k = A.rp[i]; k < A.rp[i + 1]; k++)
            for (int q = P.rp[A.ci[k]]; q < P.rp[A.ci[k] + 1]; q++) av[find(AP, i, P.ci[q])] += K[k] * pv[q];
    });
    parallel_rows(s.nc, [&](int I) {
        for (int k = s.R.rp[I]; k < s.R.rp[I + 1]; k++) {
            const int i = s.R.ci[k];
            for (int q = AP.rp[i]; q < AP.rp[i + 1]; q++) cv[find(s.Ac, I, AP.ci[q])] += pv[s.Rperm[k]] * av[q];
        }
    });
    return cv;
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

int mg_symbolic_build(int n, const MgCsr &A, const MgCells &m, bool p2, bool cell_terms, bool stretched, bool fine_q,
                      MgSymbolic *S) {
    S->step.clear();
    S->step.reserve(kMgMaxLevels);   // C points into it
    const MgCsr *C = &A;
    int cn = n;
    const int dim = m.dim, ncells = m.ncells, ld = m.ld;
    const int32_t *celldofs = m.celldofs;
    std::vector<double> K;   // unit stiffness of the level (stretched meshes)
    double theta = p2 ? kStrongP2 : kStrong;
    if (stretched) {
        std::vector<int32_t> same(n);
        for (int i = 0; i < n; i++) same[i] = i;
        K = unit_stiffness(Mode::Sum, n, A, m, p2, same);
    }
    while ((cn > kMgBottom || S->step.empty()) && (int)S->step.size() + 1 < kMgMaxLevels) {
        MgStep s;
        s.n = cn;
        std::vector<int32_t> vert;
        if (S->step.empty() && p2 && !stretched) {
            // coarse number of each vertex DoF, ascending; edge DoFs get their two vertices
            const int nv = dim + 1;
            std::vector<int32_t> e0(n, -1), e1(n, -1);
            vert.assign(n, -1);
            for (long long c = 0; c < ncells; c++)
                for (int v = 0; v < nv; v++) vert[celldofs[c * ld + v]] = 0;
            const int ne = dim == 2 ? 3 : 6;
            for (int i = 0, k = 0; i < n; i++)
                if (vert[i] == 0) vert[i] = k++, s.nc = k;
            for (long long c = 0; c < ncells; c++)
                for (int e = 0; e < ne; e++) {
                    const int32_t *d = celldofs + c * ld;
                    const int i = d[nv + e];
                    e0[i] = vert[d[dim == 2 ? kEdge2[e][0] : kEdge3[e][0]]];
                    e1[i] = vert[d[dim == 2 ? kEdge2[e][1] : kEdge3[e][1]]];
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
            MgCsr F;
            if (stretched) F = strong_pairs(cn, *C, K, theta);
            const MgCsr &N = stretched ? F : *C;
            s.nc = aggregate(cn, N.rp.data(), N.ci.data(), &s.agg);
            if (s.nc > 0.7 * cn) break;   // does not coarsen further
            build_rows(cn, s.nc, &s.P, [&](int i, auto add) {
                add(s.agg[i]);
                for (int k = N.rp[i]; k < N.rp[i + 1]; k++) add(s.agg[N.ci[k]]);
            });
            s.lump = stretched;
        }
        products(&s, C->rp.data(), C->ci.data());
        if (s.geometric) {
            if (cell_terms) filter_vertex_level(&s, m, vert);
        } else if (stretched) {
            K = coarse_stiffness(s, *C, K);
            theta = theta > kStrong ? kStrong : 0.5 * theta;
        }
        if (fine_q || !S->step.empty()) transpose(s.n, s.nc, s.AP, &s.QT, &s.QTperm);
        cn = s.nc;
        S->step.push_back(std::move(s));
        C = &S->step.back().Ac;
    }
    return S->step.empty() ? 1 : 0;
}
