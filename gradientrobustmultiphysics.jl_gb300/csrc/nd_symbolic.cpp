// Nested-dissection ordering and multifrontal symbolic analysis of one
// problem's sparsity pattern (host side of the batched direct solver).
//
// The reference solves every iterated-penalty sweep with a sparse direct
// solver (UMFPACK through LinearSolve.jl, src/solvers.jl:89-101); on the GPU
// each problem of a batch gets a multifrontal Cholesky factorisation, done
// once and reused by every sweep.  This file computes, for a symmetric
// pattern:
//   * a nested-dissection elimination order: separators from the level sets of
//     a breadth-first search started at a pseudo-peripheral DoF (the DoFs of
//     one level that touch the next one), recursively, down to leaves of at
//     most kLeaf DoFs.  On these meshes a whole level holds two lines of DoFs
//     where one separates: factor flops on 256 x 256 P2 elasticity (526k DoFs)
//     1.12e11 with whole levels, 2.49e10 with the touching DoFs (largest front
//     3,500 and 1,956 rows, factor 159M and 74M entries); 96 x 96
//     Bernardi-Raugel 1.51e9 and 5.8e8; 6^3 Bernardi-Raugel cubes 6.0e8 and
//     8.3e7 (largest front 969 and 345).  Choosing the level of the smallest
//     separator near the median takes the same time as the median level did,
//     with three searches per separator instead of up to six;
//     The search runs in the mesh's graph where one is given: a pattern that
//     dropped exact zeros is full of holes on structured meshes, its levels are
//     ragged (45 x 45 elasticity: 4.7e8 flops and 15 levels with them, 1.5e8
//     and 11 with the mesh's) and the two components need only one search;
//   * the assembly tree in post-order (children before parents, which is
//     the elimination order), each node with its front = its own DoFs
//     followed by its structure (later-eliminated DoFs coupled to them);
//   * for every node the map of original matrix entries into its front and
//     the map of each child's update matrix into the parent's front;
//   * storage offsets of the factor columns and update matrices.
// Everything depends on the pattern only, so problems with equal local
// patterns share one analysis.
#include <algorithm>
#include <cstdint>
#include <vector>

#include "nd_symbolic.h"

namespace {

constexpr int kLeaf = 48;

struct Builder {
    const int32_t *rp, *ci;      // graph (the pattern, or one that covers it)
    const int32_t *mptr = nullptr, *mem = nullptr;   // DoFs of each node (nullptr: node = DoF)
    std::vector<int> stamp;      // membership stamps
    int cur = 0;
    std::vector<int> level;
    std::vector<std::vector<int>> own;   // own DoFs per node (creation = post-order)
    std::vector<std::vector<int>> kids;

    int bfs(int start, int setstamp, std::vector<int> &order_out) {
        // returns the eccentricity of `start` in the subgraph; order_out = BFS order
        order_out.clear();
        ++cur;
        const int visit = cur;
        order_out.push_back(start);
        level[start] = 0;
        stamp[start] = visit;
        int far = 0;
        for (size_t h = 0; h < order_out.size(); h++) {
            const int v = order_out[h];
            for (int k = rp[v]; k < rp[v + 1]; k++) {
                const int w = ci[k];
                if (w == v || stamp[w] != setstamp) continue;
                stamp[w] = visit;
                level[w] = level[v] + 1;
                far = std::max(far, level[w]);
                order_out.push_back(w);
            }
        }
        // restore the set stamp for the members reached
        for (int v : order_out) stamp[v] = setstamp;
        return far;
    }

    int dissect(std::vector<int> set) {
        if (dofs(set) <= kLeaf) return leaf(std::move(set));
        ++cur;
        const int setstamp = cur;
        for (int v : set) stamp[v] = setstamp;
        std::vector<int> ord, o2;
        int ecc = bfs(set[0], setstamp, ord);
        if (ord.size() < set.size()) {
            // disconnected: split off the component of set[0]
            std::vector<int> a = ord, b;
            ++cur;
            for (int v : a) stamp[v] = cur;
            for (int v : set)
                if (stamp[v] != cur) b.push_back(v);
            int ca = dissect(std::move(a));
            int cb = dissect(std::move(b));
            return join({}, {ca, cb});
        }
        // pseudo-peripheral start: the levels of the last of three searches,
        // each from the DoF that the one before it reached last
        for (int rep = 0; rep < 2; rep++) {
            const int e2 = bfs(ord.back(), setstamp, o2);
            ord.swap(o2);
            if (e2 <= ecc) { ecc = e2; break; }
            ecc = e2;
        }
        if (ecc < 2) return leaf(std::move(set));
        // Separator of level l: its DoFs with a neighbour in level l + 1 (the
        // rest of the level has none there and stays with the lower part).
        // Taken is the level whose separator is smallest, weighted by how far
        // the larger part exceeds half, among those that leave at most 0.65 of
        // the DoFs on one side (the median level where none does).
        std::vector<int> first(ecc + 2, (int)ord.size()), touching(ecc + 1, 0);
        std::vector<char> touch(ord.size(), 0);
        for (int h = (int)ord.size() - 1; h >= 0; h--) first[level[ord[h]]] = h;
        for (size_t h = 0; h < ord.size(); h++) {
            const int v = ord[h], up = level[v] + 1;
            for (int k = rp[v]; k < rp[v + 1]; k++) {
                const int w = ci[k];
                if (level[w] == up && stamp[w] == setstamp) {
                    touch[h] = 1;
                    break;
                }
            }
            touching[level[v]] += touch[h];
        }
        const double tot = (double)set.size();
        int L = 1;
        while (L < ecc - 1 && first[L + 1] < 0.5 * tot) L++;
        double best = -1.0;
        const int median = L;
        for (int l = 1; l < ecc; l++) {
            const double lower = first[l + 1] - touching[l], upper = tot - first[l + 1];
            const double share = std::max(lower, upper) / tot;
            if (share > 0.65 && l != median) continue;
            const double cost = touching[l] * (1.0 + 2.0 * (share - 0.5));
            if (best < 0 || cost < best) {
                best = cost;
                L = l;
            }
        }
        std::vector<int> a, b, sep;
        for (size_t h = 0; h < ord.size(); h++) {
            const int v = ord[h];
            if (level[v] > L) b.push_back(v);
            else if (level[v] == L && touch[h]) sep.push_back(v);
            else a.push_back(v);
        }
        std::vector<int> ch;
        if (!a.empty()) ch.push_back(dissect(std::move(a)));
        if (!b.empty()) ch.push_back(dissect(std::move(b)));
        return join(std::move(sep), std::move(ch));
    }

    int dofs(const std::vector<int> &set) const {
        if (!mptr || set.size() > kLeaf) return (int)set.size();   // a node has a DoF at least
        int k = 0;
        for (int v : set) k += mptr[v + 1] - mptr[v];
        return k;
    }

    int leaf(std::vector<int> set) { return join(std::move(set), {}); }

    int join(std::vector<int> mine, std::vector<int> children) {
        if (mptr) {
            std::vector<int> d;
            for (int v : mine) d.insert(d.end(), mem + mptr[v], mem + mptr[v + 1]);
            mine.swap(d);
        }
        own.push_back(std::move(mine));
        kids.push_back(std::move(children));
        return (int)own.size() - 1;
    }
};

}  // namespace

int nd_cell_graph(int n, int ncells, int ld, int ncomp, const int32_t *celldofs, NdGraph *G) {
    const int nb = ld / ncomp;
    if (nb * ncomp != ld) return 1;
    // node of each DoF: the node of its first component's DoF
    std::vector<int32_t> node(n, -1);
    int nn = 0;
    for (long long c = 0; c < ncells; c++)
        for (int a = 0; a < nb; a++) {
            int32_t &q = node[celldofs[c * ld + a]];
            if (q < 0) q = nn++;
        }
    for (long long c = 0; c < ncells; c++)
        for (int k = nb; k < ld; k++) {
            const int32_t v = node[celldofs[c * ld + k % nb]];
            int32_t &q = node[celldofs[c * ld + k]];
            if (q >= 0 && q != v) return 1;
            q = v;
        }
    for (int i = 0; i < n; i++)
        if (node[i] < 0) node[i] = nn++;   // in no cell
    G->n = nn;
    G->mptr.assign((size_t)nn + 1, 0);
    for (int i = 0; i < n; i++) G->mptr[node[i] + 1]++;
    for (int v = 0; v < nn; v++) G->mptr[v + 1] += G->mptr[v];
    G->mem.resize(n);
    std::vector<int32_t> at(G->mptr.begin(), G->mptr.end() - 1);
    for (int i = 0; i < n; i++) G->mem[at[node[i]]++] = i;
    // cells of each node, then the nodes of those cells
    std::vector<int32_t> ptr((size_t)nn + 1, 0);
    for (long long c = 0; c < ncells; c++)
        for (int a = 0; a < nb; a++) ptr[node[celldofs[c * ld + a]] + 1]++;
    for (int v = 0; v < nn; v++) ptr[v + 1] += ptr[v];
    std::vector<int32_t> inc(ptr[nn]);
    at.assign(ptr.begin(), ptr.end() - 1);
    for (long long c = 0; c < ncells; c++)
        for (int a = 0; a < nb; a++) inc[at[node[celldofs[c * ld + a]]]++] = (int32_t)c;
    G->rp.assign((size_t)nn + 1, 0);
    G->ci.reserve((size_t)inc.size() * 2);
    std::vector<int32_t> mark(nn, -1);
    for (int v = 0; v < nn; v++) {
        for (int q = ptr[v]; q < ptr[v + 1]; q++)
            for (int a = 0; a < nb; a++) {
                const int32_t w = node[celldofs[(long long)inc[q] * ld + a]];
                if (mark[w] != v) {
                    mark[w] = v;
                    G->ci.push_back(w);
                }
            }
        G->rp[v + 1] = (int32_t)G->ci.size();
    }
    return 0;
}

int nd_symbolic_build(int n, const int32_t *rowptr, const int32_t *cols, NdSymbolic *S, const NdGraph *graph) {
    *S = NdSymbolic();
    if (n <= 0) return 1;
    Builder B;
    const int gn = graph ? graph->n : n;
    B.rp = graph ? graph->rp.data() : rowptr;
    B.ci = graph ? graph->ci.data() : cols;
    if (graph) {
        B.mptr = graph->mptr.data();
        B.mem = graph->mem.data();
    }
    B.stamp.assign(gn, 0);
    B.level.assign(gn, 0);
    std::vector<int> all(gn);
    for (int i = 0; i < gn; i++) all[i] = i;
    B.dissect(std::move(all));
    const int nn = (int)B.own.size();
    // elimination order = own lists in node (post-)order
    std::vector<int> order(n, -1), node_of(n, -1);
    std::vector<int> last(nn, -1);   // last elimination index in the node's subtree
    int k = 0;
    for (int t = 0; t < nn; t++) {
        for (int v : B.own[t]) {
            order[v] = k++;
            node_of[v] = t;
        }
        int l = B.own[t].empty() ? -1 : order[B.own[t].back()];
        for (int c : B.kids[t]) l = std::max(l, last[c]);
        last[t] = l;
    }
    if (k != n) return 2;
    // structures, bottom-up
    std::vector<std::vector<int>> strct(nn);
    std::vector<int> mark(n, -1);
    for (int t = 0; t < nn; t++) {
        std::vector<int> &st = strct[t];
        auto add = [&](int j) {
            if (order[j] > last[t] && mark[j] != t) {
                mark[j] = t;
                st.push_back(j);
            }
        };
        for (int v : B.own[t])
            for (int q = rowptr[v]; q < rowptr[v + 1]; q++) add(cols[q]);
        for (int c : B.kids[t])
            for (int j : strct[c]) add(j);
        std::sort(st.begin(), st.end(), [&](int a, int b) { return order[a] < order[b]; });
    }
    // parents
    std::vector<int> parent(nn, -1);
    for (int t = 0; t < nn; t++)
        for (int c : B.kids[t]) parent[c] = t;
    // fronts, maps, offsets
    S->n = n;
    S->nnodes = nn;
    S->perm.resize(n);
    for (int v = 0; v < n; v++) S->perm[order[v]] = v;
    std::vector<int> pos(n, -1);
    int64_t Loff = 0, Uoff = 0;
    S->node.resize(nn);
    for (int t = 0; t < nn; t++) {
        NdNode &nd = S->node[t];
        nd.s = (int)B.own[t].size();
        nd.f = nd.s + (int)strct[t].size();
        nd.parent = parent[t];
        nd.front_off = (int)S->front.size();
        for (int v : B.own[t]) S->front.push_back(v);
        for (int v : strct[t]) S->front.push_back(v);
        nd.child_off = (int)S->child.size();
        nd.nchild = (int)B.kids[t].size();
        for (int c : B.kids[t]) S->child.push_back(c);
        nd.L_off = Loff;
        Loff += (int64_t)nd.f * nd.s;
        nd.U_off = Uoff;
        const int64_t sc = nd.f - nd.s;
        Uoff += sc * sc;
        S->max_f = std::max(S->max_f, nd.f);
        S->max_s = std::max(S->max_s, nd.s);
        // original entries (r, c) with c in own(t), order[r] >= order[c]
        for (int i = 0; i < nd.f; i++) pos[S->front[nd.front_off + i]] = i;
        nd.entry_off = (int)S->ent_rel.size();
        for (int v : B.own[t])
            for (int q = rowptr[v]; q < rowptr[v + 1]; q++) {
                const int r = cols[q];
                if (order[r] < order[v]) continue;
                if (pos[r] < 0) return 3;
                S->ent_rel.push_back(q - rowptr[0]);
                S->ent_pos.push_back(pos[r] * nd.f + pos[v]);
            }
        nd.nentry = (int)S->ent_rel.size() - nd.entry_off;
        // children's structures into this front
        for (int c : B.kids[t]) {
            NdNode &cn = S->node[c];
            cn.ext_off = (int)S->ext.size();
            for (int j : strct[c]) {
                if (pos[j] < 0) return 4;
                S->ext.push_back(pos[j]);
            }
        }
        for (int i = 0; i < nd.f; i++) pos[S->front[nd.front_off + i]] = -1;
    }
    S->L_size = Loff;
    S->U_size = Uoff;
    // level schedule (height above the leaves) and update-vector offsets
    std::vector<int> height(nn, 0);
    int maxh = 0;
    for (int t = 0; t < nn; t++) {
        for (int c : B.kids[t]) height[t] = std::max(height[t], height[c] + 1);
        maxh = std::max(maxh, height[t]);
    }
    S->level_ptr.assign(maxh + 2, 0);
    for (int t = 0; t < nn; t++) S->level_ptr[height[t] + 1]++;
    for (int l = 0; l <= maxh; l++) S->level_ptr[l + 1] += S->level_ptr[l];
    S->level_nodes.resize(nn);
    S->level_maxf.assign(maxh + 1, 0);
    std::vector<int> fill(S->level_ptr.begin(), S->level_ptr.end() - 1);
    for (int t = 0; t < nn; t++) {
        S->level_nodes[fill[height[t]]++] = t;
        S->level_maxf[height[t]] = std::max(S->level_maxf[height[t]], S->node[t].f);
    }
    S->uv_off.resize(nn);
    int64_t uo = 0;
    for (int t = 0; t < nn; t++) {
        S->uv_off[t] = uo;
        uo += S->node[t].f - S->node[t].s;
    }
    S->uv_size = uo;
    return 0;
}
