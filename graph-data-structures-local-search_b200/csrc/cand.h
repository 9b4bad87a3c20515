// cand.h -- host interface of the candidate pass.
#pragma once
#include "ts_host.h"

namespace tsb {

constexpr size_t kCandSmem = 220 * 1024;     // dynamic shared memory a CTA may ask for
constexpr size_t kCandPersistSmem = 200 * 1024;  // the same beside the persistent kernels' static part

struct CandPlan {
  int cs = 0;               // CTAs of the cluster; 0: the state does not fit
  int threads = 0;          // per CTA
  int32_t rpc = 0, cpc = 0; // rows and columns per CTA (multiples of 4)
  int32_t vpc = 0;          // vertices per CTA of the position slice; 0: positions stay in HBM
  uint32_t inv[3] = {0, 0, 0};  // ceil(2^32 / slice): rows, columns, vertices
  int32_t list = 0;         // entries of a CTA's candidate lists
  int32_t fav = 0;          // every c*w >= 0
  int64_t plus = 0;         // upper bound of c*w
  int64_t pairs = 0;        // candidate pairs per CTA before a sweep is cheaper
  size_t smem = 0;
};
// Slices for a given cluster size within `limit` bytes of shared memory.
CandPlan cand_slices(const ts_graph* g, int32_t problem, int32_t m, bool wide, int cs, size_t limit);
// The same for a persistent (batched, served) solve; cs 0 when the pass does
// not apply: a pinned sweep, a graph on which every pair ties, or a state too
// large for the cluster.
CandPlan cand_persist(const ts_graph* g, int32_t problem, int32_t m, bool wide, int32_t pass, int cs);
// Whether the graph's weights may all be equal and positive: its heaviest row
// says so (a row of weights that happen to be the largest does too).
bool equal_weights(const ts_graph* g);
// Cluster size of a persistent solve whose caller leaves it open; 0 when no
// cluster has the pass.
int cand_cluster(const ts_graph* g, int32_t problem, int32_t m, bool wide, int32_t pass);
// The plain form's choice of cluster size.
CandPlan cand_plan(const ts_graph* g, int32_t problem, int32_t m, bool wide);
// `solver` points to a DevSolver<KeyT> (KeyT by `wide`).
cudaError_t launch_cand(int32_t problem, int kind, bool wide, const DevGraph& g, const void* solver, const CandPlan& plan,
                        cudaStream_t st, long long budget);

}  // namespace tsb
