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
cudaError_t configure(int cs, size_t smem, cudaStream_t st, cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr) {
  const void* fn = reinterpret_cast<const void*>(cand_kernel<PROB, ST, KeyT>);
  cudaError_t e = allow_dyn_smem(fn, smem);
  if (e != cudaSuccess) return e;
  if (cs > 8) {
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
  }
  cfg = {};
  cfg.gridDim = dim3((unsigned)cs);
  cfg.blockDim = dim3(kCandTPB);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaSuccess;
}

template <int PROB, int ST, class KeyT>
struct Launch {
  static cudaError_t run(const DevGraph& g, const void* s, int cs, size_t smem, cudaStream_t st, long long budget) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    const cudaError_t e = configure<PROB, ST, KeyT>(cs, smem, st, cfg, attr);
    if (e != cudaSuccess) return e;
    return cudaLaunchKernelEx(&cfg, cand_kernel<PROB, ST, KeyT>, g, *static_cast<const DevSolver<KeyT>*>(s), budget);
  }
  // Clusters of cs CTAs the device can hold (0: none).
  static int resident(int cs, size_t smem) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    int n = 0;
    if (configure<PROB, ST, KeyT>(cs, smem, nullptr, cfg, attr) != cudaSuccess ||
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
  p.smem = cand_layout(g->n, p.rpc, p.cpc, wide ? 8 : 4, p.plus > 0).total;
  if (p.smem <= limit) p.cs = cs;
  // Looking up 64 pairs a thread takes about as long as a small sweep launch.
  p.pairs = 64 * kCandTPB;
  return p;
}

CandPlan cand_persist(const ts_graph* g, int32_t problem, int32_t m, bool wide, int32_t pass, int cs) {
  if (pass != TS_PASS_AUTO) return CandPlan{};
  CandPlan p = cand_slices(g, problem, m, wide, cs, kCandPersistSmem);
  if (!p.cs) return CandPlan{};
  // The cluster's own sweep is the alternative: it passes eight pairs or more
  // in the time of one candidate lookup.
  p.pairs = std::max<int64_t>(64 * 256, (int64_t)m * (g->n - m) / 8 / cs);
  return p;
}

// One CTA while the batch has solves for every SM: per iteration one 256-thread
// CTA against two took 4.5 against 4.2 us (MDP, n = 5,000) and 33 against 21 us
// (Max Bisection, n = 3,000) -- less than twice as fast on twice the SMs.
// Larger solves need the second CTA's shared memory.
int cand_cluster(int32_t n) { return n <= 6144 ? 1 : (n <= 16384 ? 2 : 4); }

CandPlan cand_plan(const ts_graph* g, int32_t problem, int32_t m, bool wide) {
  // A CTA scans about 4,000 positions in the time of one cluster barrier;
  // more CTAs also share the candidates' rows.
  int cs = 1;
  while (cs < kCandMaxCluster && (int64_t)cs * kCandSlice < g->n) cs *= 2;
  for (; cs <= kCandMaxCluster; cs *= 2) {
    CandPlan p = cand_slices(g, problem, m, wide, cs, kCandSmem);
    if (p.cs && by_kind(problem, g->kind, wide, [&](auto l) { return decltype(l)::resident(cs, p.smem); }) > 0) return p;
  }
  return CandPlan{};
}

cudaError_t launch_cand(int32_t problem, int kind, bool wide, const DevGraph& g, const void* solver, int cs, size_t smem,
                        cudaStream_t st, long long budget) {
  return by_kind(problem, kind, wide, [&](auto l) { return decltype(l)::run(g, solver, cs, smem, st, budget); });
}

}  // namespace tsb
