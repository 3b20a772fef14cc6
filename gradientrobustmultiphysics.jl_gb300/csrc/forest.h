// Multifrontal Cholesky of one or many independent problems, level by level
// over all of their assembly trees (forest.cu).
#pragma once
#include <vector>

#include "grmp_internal.h"
#include "nd_symbolic.h"

// one front; offsets of values are relative to its problem's bases
struct FoNode {
    int s, f, front_off, child_off, nchild, entry_off, nentry, ext_off;
    long long L_off, U_off, uv_off;
};

struct FoProb {
    int row0, pad;
    long long nnz0, Lb, Ub, uvb;   // first value of the matrix, bases of factor columns, update matrices, update vectors
};

struct FoDev {
    const FoNode *node;
    const int32_t *front, *child, *ent_rel, *ent_pos, *ext;
    const int2 *src;               // per front row: up to two update-vector entries of the children that add to it (-1: none)
    const FoProb *prob;
};

// items {problem, node} of one level and size class
struct FoItems {
    const int2 *d = nullptr;
    int count = 0, maxf = 0;
};

struct FoLevel {
    FoItems small_[4];             // fronts factored in shared memory, by size
    FoItems big;                   // fronts factored by groups of blocks
    FoItems solve[3];              // by size, for the solves
    // blocks of the large fronts' launch: {item, rank in its group, blocks of the group, groups}
    const int4 *blocks = nullptr;
    int nblocks = 0;
};

// fronts up to these sizes are solved by 64 and 128 threads, larger ones by 512
// (96 squares, f = 550, s = 290: 130 us with 128 threads, bound by the loads in flight)
constexpr int kFoSolve[2] = {96, 224};

struct MfForest {
    FoDev dev{};
    std::vector<std::pair<void *, size_t>> bufs;
    std::vector<FoLevel> level;
    int nprob = 0, max_f = 0, max_s = 0;
    long long L_size = 0, U_size = 0, uv_size = 0;
    // numeric storage (sizeof of the values)
    int esize = 0;
    void *L = nullptr, *U = nullptr, *uv = nullptr, *pool = nullptr;
    size_t Lb = 0, Ub = 0, uvb = 0, poolb = 0;
    void *cs = nullptr;            // barriers of the grouped factorisation
};

struct FoProblem {
    int group, row0;
    long long nnz0;
};

// device bytes of the numeric storage of a growing set of problems: factors and
// updates, and the buffers of the fronts that groups of blocks work on (as many
// as a level of theirs needs, within a quarter of the pool's bound, one at the least)
class FoNeed {
  public:
    FoNeed(const std::vector<const NdSymbolic *> &groups, int esize);
    void add(int group);
    size_t with(int group) const;    // bytes with one more problem of this group
    size_t bytes() const { return total(fac, pool, slot); }
    size_t trees() const { return tree; }   // of all groups' trees, which every part keeps for its problems

  private:
    struct Group {
        size_t fac, pool, slot;
    };
    std::vector<Group> of;
    size_t fac = 0, pool = 0, slot = 0, tree = 0;
    static size_t total(size_t fac, size_t pool, size_t slot);
};
// esize: precision the size classes are made for
int grmp_forest_create(grmp_context ctx, const std::vector<const NdSymbolic *> &groups, const std::vector<FoProblem> &probs,
                       int esize, MfForest **out);
void grmp_forest_free(grmp_context ctx, MfForest *F);
// gives the numeric storage back (the next factorisation takes it again)
void grmp_forest_release(grmp_context ctx, MfForest *F);
// factors every problem of vals (the matrix values, CSR order); err[p] (device,
// zeroed here) = 1 + node of a non-positive pivot.  FP64 keeps the inverses of
// the factor's 32 x 32 diagonal blocks in their place (grmp_forest_solve64).
int grmp_forest_factor64(grmp_context ctx, MfForest *F, const double *vals, int *err);
int grmp_forest_factor32(grmp_context ctx, MfForest *F, const double *vals, int *err);
// w <- A^-1 w for the problems with active[p] != 0 (nullptr: all)
void grmp_forest_solve64(grmp_context ctx, MfForest *F, double *w, const int *active);
