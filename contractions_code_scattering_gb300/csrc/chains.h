// Stages of block products over (t_sink, t_src) pairs, shared by the chain diagrams
// (engine_chains.cu) and the profile adjoint (adjoint.cu).
#pragma once

#include <map>
#include <utility>
#include <vector>

#include "kernels.h"

namespace ctr {

constexpr int G5[4] = {1, 1, -1, -1};  // gamma_5 = diag(1,1,-1,-1) of the table basis

struct Ctx {
  int N, Nt;
  size_t N2;
  cudaStream_t s;
  int engine = CTR_ENGINE_FP64;
  bool full = false;  // split engine: grids of more than 128 k at full scale
};

// Elemental of a call: Phi(t) = p + t * stride (an [Nt][N][N] array, or one momentum
// of an [Nt][nphi][N][N] array).
struct Elem {
  const double2* p;
  size_t stride;
};

const float kOne[4] = {1.f, 1.f, 1.f, 1.f};
const float kG5[4] = {(float)G5[0], (float)G5[1], (float)G5[2], (float)G5[3]};

// The pairs of one call in batches.  All pairs: tiles of t_sink x t_src, both
// extents as even as the batch allows, so that the pairs that share a t_src (the
// right operands R and Phi(t_src)) and those that share a t_sink (L and
// Phi(t_sink)) both stack along M: from 7 pairs of 4 slabs up, the padding rows of
// a 128-row tile are below 2 %.  At most hmax sink times a batch.  A list of pairs
// keeps the list's order.
struct PairBatch {
  std::vector<int> ent, tf, ti;       // position in the output, time slices
  std::vector<const double2*> T;      // tau(tf, ti)
  std::vector<std::vector<int>> by_ti, by_tf;  // groups of batch indices
  std::vector<int> gti, pti, gtf, ptf;         // group and position of each pair
};

// plist: the listed pairs (t_sink row * Nt + t_src), else all rows x Nt pairs.
std::vector<PairBatch> pair_batches(const double2* tau, size_t blk16, int Nt, int tf_begin, int rows, int batch,
                                    const std::vector<int>* plist, int hmax = 1 << 30);

// Distinct pairs of elementals, and the time slices each is needed at.
struct Combos {
  std::vector<std::pair<int, int>> list;
  std::vector<std::vector<char>> need;
  std::map<std::pair<int, int>, int> at;
  int Nt;
  explicit Combos(int nt) : Nt(nt) {}
  int use(int a, int b) {
    auto it = at.emplace(std::make_pair(a, b), (int)list.size()).first;
    if (it->second == (int)list.size()) {
      list.push_back({a, b});
      need.emplace_back(Nt, 0);
    }
    return it->second;
  }
};

// A grid of nterm terms with weights w (its operands and outputs are filled in by the caller).
GridTask make_grid(int nslab, int nb, int nterm, const float* w, int adag, int bdag);
// One stage on the call's engine: plain tasks, or grids (stacked along M on the split engine).
int run_stage(const Ctx& c, const std::vector<ZTask>& tasks, int slot);
int run_grids(const Ctx& c, const std::vector<GridTask>& g, int slot);
int per_t_products(const Ctx& c, const double2* diag, size_t dstride, const std::vector<Elem>& el, int slot,
                   const std::vector<std::pair<int, int>>& combos, const std::vector<std::vector<char>>& need,
                   size_t cap, std::vector<const double2*>& M);
// One call's own elementals, [nt][nev][nev] each; set[k]: the first of them with the k-th one's address.
std::vector<Elem> elems(int nev, const std::vector<const double*>& p, int32_t* set);
// Scratch budget of a batch of pairs: of a momentum-set call, and of every other call, which
// has to run beside a caller's own tensors.
size_t sets_budget();
constexpr size_t CHAIN_BUDGET = (size_t)3 << 30;

}  // namespace ctr
