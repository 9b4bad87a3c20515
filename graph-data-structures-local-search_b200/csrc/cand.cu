// cand.cu -- host side of the candidate pass (cand.cuh) for the plain form:
// slices, cluster size and the launch.
#include <algorithm>

#include "cand.cuh"
#include "cand.h"

namespace cg = cooperative_groups;

namespace tsb {
namespace {

// Up to `budget` iterations by one cluster (cand_run); a launch past the
// admitted target or after the search's end does nothing.
template <int PROB, int ST, class KeyT>
__global__ void __launch_bounds__(kCandTPB, 1)
cand_kernel(const DevGraph g, const DevSolver<KeyT> s, long long budget) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ CandShared<KeyT> sh;
  cg::cluster_group cl = cg::this_cluster();
  const long long target = __ldcg(&s.st->target);
  if (__ldcg(&s.st->done) || __ldcg(&s.st->iter) >= target) {
    if (blockIdx.x == 0 && threadIdx.x == 0) s.st->owed = 0;
    return;
  }
  cand_run<PROB, ST, KeyT>(g, s, target, budget, cl, sh, smem_raw);
}

template <int PROB, int ST, class KeyT>
cudaError_t configure(const CandPlan& p, cudaStream_t st, cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr) {
  const void* fn = reinterpret_cast<const void*>(cand_kernel<PROB, ST, KeyT>);
  cudaError_t e = allow_dyn_smem(fn, p.smem);
  if (e != cudaSuccess) return e;
  if (p.cs > 8) {
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
  }
  cfg = {};
  cfg.gridDim = dim3((unsigned)p.cs);
  cfg.blockDim = dim3((unsigned)p.threads);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)p.cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaSuccess;
}

template <int PROB, int ST, class KeyT>
struct Launch {
  static cudaError_t run(const DevGraph& g, const void* s, const CandPlan& p, cudaStream_t st, long long budget) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    const cudaError_t e = configure<PROB, ST, KeyT>(p, st, cfg, attr);
    if (e != cudaSuccess) return e;
    return cudaLaunchKernelEx(&cfg, cand_kernel<PROB, ST, KeyT>, g, *static_cast<const DevSolver<KeyT>*>(s), budget);
  }
  // Clusters of the plan's size the device can hold (0: none).
  static int resident(const CandPlan& p) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    int n = 0;
    if (configure<PROB, ST, KeyT>(p, nullptr, cfg, attr) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, cand_kernel<PROB, ST, KeyT>, &cfg) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    return n;
  }
};

// Calls F<PROB, ST, KeyT>::f for the run-time choice.
template <int PROB, class KeyT, class Fn>
auto by_struct(int kind, Fn&& fn) {
  switch (kind) {
    case S_CSR: return fn(Launch<PROB, S_CSR, KeyT>{});
    case S_HASH: return fn(Launch<PROB, S_HASH, KeyT>{});
    case S_WSWAP: return fn(Launch<PROB, S_WSWAP, KeyT>{});
    case S_BITSET: return fn(Launch<PROB, S_BITSET, KeyT>{});
    case S_BB: return fn(Launch<PROB, S_BB, KeyT>{});
    default: return fn(Launch<PROB, S_BITSET_BB, KeyT>{});
  }
}
template <class Fn>
auto by_kind(int problem, int kind, bool wide, Fn&& fn) {
  if (problem == P_MDP)
    return wide ? by_struct<P_MDP, long long>(kind, fn) : by_struct<P_MDP, int32_t>(kind, fn);
  return wide ? by_struct<P_MAXBS, long long>(kind, fn) : by_struct<P_MAXBS, int32_t>(kind, fn);
}

}  // namespace

CandPlan cand_slices(const ts_graph* g, int32_t problem, int32_t m, bool wide, int cs, size_t limit) {
  CandPlan p;
  p.plus = problem == P_MDP ? (g->neg_w ? g->max_abs_w : 0) : 2 * g->max_abs_w;
  p.fav = problem == P_MAXBS && !g->neg_w;
  const int32_t delta = g->n - m;
  p.rpc = ((m + cs - 1) / cs + 3) & ~3;
  p.cpc = ((delta + cs - 1) / cs + 3) & ~3;
  const int kb = wide ? 8 : 4;
  // Lists for three quarters of the slice (sparse graphs of few distinct
  // contributions have that many candidates) or what fits, then the positions
  // by vertex where they fit too.
  const bool edges = p.plus > 0;
  const int32_t whole = p.rpc + p.cpc;
  const size_t bare = cand_layout(g->n, p.rpc, p.cpc, kb, 0, edges, 0).total;
  int64_t list = std::min<int64_t>(std::max<int64_t>(kCandList, (int64_t)whole * 3 / 4), whole);
  if (bare < limit) list = std::min<int64_t>(list, (int64_t)(limit - bare) / 8);
  p.list = (int32_t)(std::max<int64_t>(list, std::min<int32_t>(whole, kCandList)) + 3) & ~3;
  if (p.list > whole) p.list = whole;
  const int32_t vpc = ((g->n + cs - 1) / cs + 3) & ~3;
  p.vpc = cand_layout(g->n, p.rpc, p.cpc, kb, vpc, edges, p.list).total <= limit ? vpc : 0;
  p.smem = cand_layout(g->n, p.rpc, p.cpc, kb, p.vpc, edges, p.list).total;
  if (p.smem > limit && p.list > kCandList) {  // rounding of the fit
    p.list -= 4;
    p.smem = cand_layout(g->n, p.rpc, p.cpc, kb, p.vpc, edges, p.list).total;
  }
  p.threads = kCandTPB;
  // Divisions by a slice are a multiplication by ceil(2^32 / slice), exact
  // for up to 16 slices of fewer than 2^14.
  const int32_t per[3] = {p.rpc, p.cpc, p.vpc};
  bool exact = true;
  for (int k = 0; k < 3; k++) {
    if (!per[k]) continue;
    p.inv[k] = (uint32_t)(((1ULL << 32) + per[k] - 1) / per[k]);
    exact = exact && (uint64_t)cs * per[k] * per[k] < (1ULL << 32);
  }
  if (p.smem <= limit && exact) p.cs = cs;
  // Looking up 64 pairs a thread takes about as long as a small sweep launch.
  p.pairs = 64 * kCandTPB;
  return p;
}

bool equal_weights(const ts_graph* g) {
  if (g->max_degree < 0) {
    int64_t d = 0;
    for (int32_t v = 0; v < g->n; v++) d = std::max(d, g->h_rowptr[v + 1] - g->h_rowptr[v]);
    g->max_degree = d;
  }
  return !g->neg_w && g->max_wdeg == g->max_degree * g->max_abs_w;
}

// In a complete graph of equal weights all vertices of a side are alike: every
// pair ties and the pass never settles an iteration.  Its shared memory would
// only keep other CTAs of the sweeps off the SM (200 MDP solves of n = 600: 92
// ms without it, 175 with it).  With both signs (weights of 1 and -1) the
// contributions differ.
static bool every_pair_ties(const ts_graph* g) {
  return g->entries == (int64_t)g->n * (g->n - 1) && equal_weights(g);
}

CandPlan cand_persist(const ts_graph* g, int32_t problem, int32_t m, bool wide, int32_t pass, int cs) {
  if (pass != TS_PASS_AUTO || every_pair_ties(g)) return CandPlan{};
  CandPlan p = cand_slices(g, problem, m, wide, cs, kCandPersistSmem);
  if (!p.cs) return CandPlan{};
  // The cluster's own sweep is the alternative: it passes eight pairs or more
  // in the time of one candidate lookup.
  p.pairs = std::max<int64_t>(64 * 256, (int64_t)m * (g->n - m) / 8 / cs);
  return p;
}

// One 256-thread CTA while the batch has solves for every SM: per iteration one
// CTA against four took 2.7 against 3.4 us (MDP, n = 5,000), 12.9 against 10.0
// us (Max Bisection, n = 5,000) and 22 against 11.7 us (n = 12,000) -- less
// than twice as fast on four times the SMs.  Larger solves need the other
// CTAs' shared memory: as many as hold the state, up to eight.
int cand_cluster(const ts_graph* g, int32_t problem, int32_t m, bool wide, int32_t pass) {
  for (int cs = g->n <= 6144 ? 1 : (g->n <= 16384 ? 2 : 4); cs <= 8; cs *= 2)
    if (cand_persist(g, problem, m, wide, pass, cs).cs) return cs;
  return 0;
}

CandPlan cand_plan(const ts_graph* g, int32_t problem, int32_t m, bool wide) {
  // Max Bisection spends most of an iteration on candidate rows, which more
  // CTAs share; an MDP iteration mostly scans and applies, and one CTA needs
  // no cluster barriers.  1 / 8 / 16 CTAs, us per iteration: MDP ER n = 2,000
  // 2.5 / 3.5 / 3.7; dense n = 2,000 7.8 / 8.6 / 10.4; bisection n = 5,000
  // 14.5 / 10.1 / 10.4, n = 30,011 16.8 / 10.6 / 10.3, n = 100,000 - / 16.5 /
  // 13.9; n = 18,000 of degree 5 (half of the vertices are candidates) - / 23 /
  // 17, n = 1,000 of degree 5 16 / 9.5 / -, of degree 25 8.3 / 9.6 / -.
  const int n = g->n;
  const bool edges = problem == P_MAXBS || g->neg_w;
  int cs = edges ? (n <= 768 ? 1 : (n <= 12288 ? 8 : 16)) : (n <= 8192 ? 1 : (n <= 32768 ? 4 : 16));
  for (; cs <= kCandMaxCluster; cs *= 2) {
    CandPlan p = cand_slices(g, problem, m, wide, cs, kCandSmem);
    p.threads = n <= 1024 ? 256 : kCandTPB;
    if (p.cs && by_kind(problem, g->kind, wide, [&](auto l) { return decltype(l)::resident(p); }) > 0) return p;
  }
  return CandPlan{};
}

cudaError_t launch_cand(int32_t problem, int kind, bool wide, const DevGraph& g, const void* solver, const CandPlan& plan,
                        cudaStream_t st, long long budget) {
  return by_kind(problem, kind, wide, [&](auto l) { return decltype(l)::run(g, solver, plan, st, budget); });
}

}  // namespace tsb
