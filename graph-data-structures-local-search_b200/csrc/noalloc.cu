// noalloc.cu -- best admissible swap of a caller-held state, with no device
// allocation.
//
// Who needs it: callers that may not allocate device memory -- plugins whose
// host application owns all of HBM through its own pool allocator, and
// services that run under a fixed device-memory budget.  They keep the graph
// and the tabu state in their own buffers and get one iteration's decision:
// every swap evaluated with the reference's key rule (tabu/aspiration filter,
// MDP -99999 sentinel, MaxBS float-quantised penalty) and the ArgMax with its
// lowest-index tie rule.  This entry point has no counterpart in the reference.
//
// Scratch: one file-scope device array (kScratchBytes, about 3 MiB) holding the
// position-ordered contributions and tabu flags, the positions by vertex, the
// per-CTA records, the bounds and two last-CTA tickets.  Every GPU that loads
// the library keeps it until the process exits.  All calls share it and it
// keeps the last call's contents.  Calls that overlap on the GPU (from other
// streams or host threads) race on it and decide wrongly; they read and write
// nothing out of bounds, and leave nothing behind: the staging ticket wraps
// after every kNaStageCtas numbers, so it is 0 again however calls were mixed,
// and the staging launch clears the other.
//
// Cost: the pairs are bounded as in the solver's candidate pass (cand.cuh).
// One launch orders the state, takes the maxima of both sides and of the
// weights, and looks up the seed pairs: LB.  The second visits the rows whose
// bound reaches LB -- their own entries (adjacent pairs, exactly), and for
// non-adjacent pairs the columns with A + B >= LB, one binary search each.
// Where no pair is allowed, or a penalised key could win, it visits every
// pair with the reference's key rule, a binary search each (roughly P / 1e10
// s for P pairs); so it does for fewer than 2^20 pairs.  n = 20,001, m = 1,000:
// 173 us (every pair) -> 29 us.
#include <climits>
#include <cstdint>
#include <mutex>

#include "sweep.cuh"
#include "ts_host.h"

namespace tsb {
namespace {

constexpr int32_t kNaMaxN = TS_NOALLOC_MAX_N;
constexpr int kNaTPB = 256;
constexpr int kNaMaxCtas = 148 * 8;  // one wave: more CTAs only queue at the ticket
constexpr long long kNaBoundPairs = 1 << 20;
constexpr int kNaStageCtas = 148;    // every launch: the weights are read by all of them
constexpr size_t kNaPvgOff = 0;                                        // long long[kNaMaxN]
constexpr size_t kNaPosOff = kNaPvgOff + sizeof(long long) * kNaMaxN;  // int32[kNaMaxN], by vertex
constexpr size_t kNaTabOff = kNaPosOff + sizeof(int32_t) * kNaMaxN;    // uint8[kNaMaxN]
constexpr size_t kNaRecOff = kNaTabOff + kNaMaxN;                      // CtaRec[kNaMaxCtas]
constexpr size_t kNaCntOff = kNaRecOff + sizeof(CtaRec) * kNaMaxCtas;  // tickets, bounds
constexpr size_t kScratchBytes = kNaCntOff + 256;

static __device__ __align__(256) unsigned char g_na_scratch[kScratchBytes];

// Written by the staging launch for the second one.
struct NaGoal {
  long long Am, AA, Bm, BA, LB, LT, plus;
  long long seed_key[2], seed_idx[2];  // LLONG_MIN: none
  int32_t all_pairs, nt_ok, need_n;
};
struct NaView {
  long long* pvg;
  int32_t* pos;
  uint8_t* ptab;
  CtaRec* recs;
  unsigned int* counter;
  unsigned int* staged;
  NaGoal* goal;
};
static_assert(sizeof(NaGoal) <= 224, "the bounds fit behind the tickets");

NaView view_of(void* base) {
  unsigned char* b = static_cast<unsigned char*>(base);
  NaView v;
  v.pvg = reinterpret_cast<long long*>(b + kNaPvgOff);
  v.pos = reinterpret_cast<int32_t*>(b + kNaPosOff);
  v.ptab = b + kNaTabOff;
  v.recs = reinterpret_cast<CtaRec*>(b + kNaRecOff);
  v.counter = reinterpret_cast<unsigned int*>(b + kNaCntOff);
  v.staged = v.counter + 1;
  v.goal = reinterpret_cast<NaGoal*>(b + kNaCntOff + 16);
  return v;
}

// First entry of v in u's sorted row by a whole warp, 32 probes a step.
__device__ __forceinline__ int32_t na_warp_lookup(const int64_t* rowptr, const int32_t* col, const int32_t* w,
                                                  int32_t u, int32_t v) {
  const int lane = threadIdx.x & 31;
  long long lo = rowptr[u], len = rowptr[u + 1] - lo;
  while (len > 32) {
    const long long step = (len + 31) >> 5, at = (lane + 1) * step - 1;
    const bool below = at < len && col[lo + at] < v;
    const long long skip = __popc(__ballot_sync(0xffffffffu, below)) * step;
    lo += skip;
    len = step < len - skip ? step : len - skip;
  }
  const bool hit = lane < len && col[lo + lane] == v;
  const unsigned b = __ballot_sync(0xffffffffu, hit);
  return b ? w[lo + __ffs(b) - 1] : 0;
}

// Position order: pvg[p] = vg[sol[p]], ptab[p] = tab[sol[p]] > iter; maxima of
// the rows' A and the columns' B (0 row non-tabu, 1 row all, 2 column non-tabu,
// 3 column all) and of the weights; the last CTA forms the bounds.  Without
// BOUNDS the second launch visits every pair.
template <bool BOUNDS>
__global__ void __launch_bounds__(kNaTPB)
k_na_stage(int32_t problem, int32_t n, int32_t m, long long iter, long long D, const int64_t* __restrict__ rowptr,
           const int32_t* __restrict__ col, const int32_t* __restrict__ w, const int32_t* __restrict__ sol,
           const long long* __restrict__ vg, const int32_t* __restrict__ tab, NaView sc) {
  __shared__ CtaRec red[kNaTPB / 32];
  __shared__ CtaRec s_top[5];
  __shared__ int32_t s_last;
  const int tid = threadIdx.x;
  const long long stride = (long long)gridDim.x * blockDim.x;
  long long k4[4], i4[4];
#pragma unroll
  for (int q = 0; q < 4; q++) { k4[q] = LLONG_MIN; i4[q] = LLONG_MAX; }
  for (long long p = blockIdx.x * (long long)blockDim.x + tid; p < n; p += stride) {
    const int32_t v = sol[p];
    const long long x = vg[v];
    const bool t = tab[v] > iter, row = p < m;
    sc.pvg[p] = x;
    if constexpr (!BOUNDS) {  // the flags as whole words, in the positions' place
      sc.pos[p] = t;
      continue;
    }
    sc.ptab[p] = t;
    sc.pos[v] = (int32_t)p;
    const long long y = problem == P_MDP && row ? -x : x;
#pragma unroll
    for (int q = 0; q < 4; q++)
      if ((q < 2) == row && ((q & 1) || !t)) better_rec(k4[q], i4[q], y, p);
  }
  if constexpr (!BOUNDS) {
    if (blockIdx.x == 0 && tid == 0) *sc.counter = 0u;
    return;
  }
  // the weights' range, as records of (max, .) and (-min, .)
  long long hi = 0, lo = 0;
  const long long E = rowptr[n];
  for (long long k = rowptr[0] + blockIdx.x * (long long)blockDim.x + tid; k < E; k += 8 * stride) {
    int32_t x[8];
#pragma unroll
    for (int q = 0; q < 8; q++) x[q] = k + q * stride < E ? w[k + q * stride] : 0;
#pragma unroll
    for (int q = 0; q < 8; q++) {
      hi = x[q] > hi ? x[q] : hi;
      lo = -(long long)x[q] > lo ? -(long long)x[q] : lo;
    }
  }
  long long d0 = 0;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    block_best(k4[q], i4[q], red);
    if (tid == 0) { sc.recs[5 * blockIdx.x + q].key = k4[q]; sc.recs[5 * blockIdx.x + q].idx = i4[q]; }
  }
  block_best(hi, d0, red);
  d0 = 0;
  block_best(lo, d0, red);
  if (tid == 0) {
    sc.recs[5 * blockIdx.x + 4].key = hi;
    sc.recs[5 * blockIdx.x + 4].idx = lo;
    __threadfence();
    s_last = atomicInc(sc.staged, gridDim.x - 1) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
#pragma unroll
  for (int q = 0; q < 4; q++) { k4[q] = LLONG_MIN; i4[q] = LLONG_MAX; }
  hi = lo = 0;
  for (int b = tid; b < (int)gridDim.x; b += blockDim.x) {
#pragma unroll
    for (int q = 0; q < 4; q++) better_rec(k4[q], i4[q], __ldcg(&sc.recs[5 * b + q].key), __ldcg(&sc.recs[5 * b + q].idx));
    const long long h = __ldcg(&sc.recs[5 * b + 4].key), l = __ldcg(&sc.recs[5 * b + 4].idx);
    hi = h > hi ? h : hi;
    lo = l > lo ? l : lo;
  }
#pragma unroll
  for (int q = 0; q < 4; q++) {
    block_best(k4[q], i4[q], red);
    if (tid == 0) { s_top[q].key = k4[q]; s_top[q].idx = i4[q]; }
  }
  d0 = 0;
  block_best(hi, d0, red);
  d0 = 0;
  block_best(lo, d0, red);
  if (tid == 0) { s_top[4].key = hi; s_top[4].idx = lo; }
  __syncthreads();
  const long long Am = s_top[0].key, AA = s_top[1].key, Bm = s_top[2].key, BA = s_top[3].key;
  const bool nt_ok = Am != LLONG_MIN && Bm != LLONG_MIN;
  const long long plus = problem == P_MDP ? s_top[4].idx : 2 * s_top[4].key;
  // c*w of the pairs of the maxima 0, 2 and 1, 3: a warp each
  if (tid < 64 && (tid >= 32 || nt_ok)) {
    const int q = tid >> 5;
    // (records of an overlapping call may hold positions of its larger state)
    const long long i = s_top[q].idx, j = s_top[q + 2].idx;
    const bool in = i >= 0 && i < n && j >= 0 && j < n;
    const long long x = in ? na_warp_lookup(rowptr, col, w, sol[i], sol[j]) : 0;
    if ((tid & 31) == 0) red[q].key = problem == P_MDP ? -x : 2 * x;
  }
  __syncthreads();
  const long long c1 = nt_ok ? red[0].key : 0, c2 = red[1].key;
  if (tid != 0) return;
  NaGoal g;
  const int32_t delta = n - m;
  g.Am = Am; g.AA = AA; g.Bm = Bm; g.BA = BA; g.plus = plus; g.nt_ok = nt_ok;
  g.seed_key[0] = g.seed_key[1] = LLONG_MIN;
  g.seed_idx[0] = g.seed_idx[1] = LLONG_MAX;
  g.LB = LLONG_MIN;
  if (nt_ok) {
    g.LB = g.seed_key[0] = Am + Bm + c1;
    g.seed_idx[0] = s_top[0].idx * delta + (s_top[2].idx - m);
  }
  if (AA + BA + c2 > D) {
    g.seed_key[1] = AA + BA + c2;
    g.seed_idx[1] = s_top[1].idx * delta + (s_top[3].idx - m);
    if (g.seed_key[1] > g.LB) g.LB = g.seed_key[1];
  }
  g.LT = g.LB > D ? g.LB : (D == LLONG_MAX ? D : D + 1);
  // every pair: none is allowed, or the key of one that is not could win
  g.all_pairs = g.LB == LLONG_MIN ||
                (problem == P_MDP ? g.LB <= kMdpSentinel : g.LB <= maxbs_penalty(AA + BA + plus));
  // non-adjacent pairs, and adjacent ones with c*w <= 0, are bounded by A + B:
  // a seed with c*w >= 0 is the best of them
  g.need_n = (nt_ok && c1 < 0 && Am + Bm >= g.LB) || (c2 < 0 && AA + BA >= g.LT);
  *sc.goal = g;
  *sc.counter = 0u;
}

// First entry of u's sorted row with neighbour v (lower_bound), else 0.
__device__ __forceinline__ int32_t na_lookup(const int64_t* rowptr, const int32_t* col,
                                             const int32_t* w, int32_t u, int32_t v) {
  long long lo = rowptr[u], len = rowptr[u + 1] - lo;
  const long long end = lo + len;
  while (len > 0) {
    const long long half = len >> 1;
    if (col[lo + half] < v) { lo += half + 1; len -= half + 1; }
    else len = half;
  }
  return (lo < end && col[lo] == v) ? w[lo] : 0;
}

template <bool BOUNDS>
__global__ void __launch_bounds__(kNaTPB)
k_na_sweep(int32_t problem, int32_t n, int32_t m, long long cur, long long best,
           const int64_t* __restrict__ rowptr, const int32_t* __restrict__ col,
           const int32_t* __restrict__ w, const int32_t* __restrict__ sol, NaView sc,
           int64_t* __restrict__ out) {
  __shared__ CtaRec red[kNaTPB / 32];
  __shared__ int32_t s_last;
  const int32_t delta = n - m;
  const long long P = (long long)m * delta;
  const long long D = best - cur;
  long long bk = LLONG_MIN, bi = LLONG_MAX;
  if (BOUNDS && !sc.goal->all_pairs) {
    const NaGoal g = *sc.goal;
    if (blockIdx.x == 0 && threadIdx.x < 2 && g.seed_key[threadIdx.x] != LLONG_MIN)
      better_rec(bk, bi, g.seed_key[threadIdx.x], g.seed_idx[threadIdx.x]);
    for (int32_t i = blockIdx.x; i < m; i += gridDim.x) {
      const long long a = sc.pvg[i], A = problem == P_MDP ? -a : a;
      const bool rt = sc.ptab[i] != 0, rn = !rt && g.nt_ok;
      // adjacent pairs: the row's own entries
      if (g.plus > 0 && ((rn && A + g.Bm + g.plus >= g.LB) || A + g.BA + g.plus >= g.LT)) {
        const int32_t u = sol[i];
        const long long r0 = rowptr[u], r1 = rowptr[u + 1];
        for (long long k = r0 + threadIdx.x; k < r1; k += blockDim.x) {
          const int32_t z = col[k];
          const long long c = problem == P_MDP ? -(long long)w[k] : 2LL * w[k];
          if (A + g.BA + c < g.LB) continue;
          if ((uint32_t)z >= (uint32_t)n) continue;
          const int32_t p = sc.pos[z];
          if (p < m || p >= n || (k > r0 && col[k - 1] == z)) continue;  // inside, or not the pair's first entry
          const long long x = A + sc.pvg[p] + c;
          if (x >= g.LB && allowed(rt, sc.ptab[p] != 0, x, D)) better_rec(bk, bi, x, (long long)i * delta + (p - m));
        }
      }
      // the other pairs: columns with A + B in reach
      if (g.need_n && ((rn && A + g.Bm >= g.LB) || A + g.BA >= g.LT)) {
        const int32_t u = sol[i];
        for (int32_t j = m + threadIdx.x; j < n; j += blockDim.x) {
          const long long y = A + sc.pvg[j];
          if (y < g.LB) continue;
          const bool t = rt || sc.ptab[j] != 0;
          if (t && y < g.LT) continue;
          const long long wt = na_lookup(rowptr, col, w, u, sol[j]);
          const long long x = y + (problem == P_MDP ? -wt : 2 * wt);
          if (!t || x > D) better_rec(bk, bi, x, (long long)i * delta + (j - m));
        }
      }
    }
  } else {
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < P;
         idx += (long long)gridDim.x * blockDim.x) {
      const int32_t i = (int32_t)(idx / delta), j = (int32_t)(idx % delta) + m;
      const int32_t wt = na_lookup(rowptr, col, w, sol[i], sol[j]);
      const long long x = problem == P_MDP ? sc.pvg[j] - sc.pvg[i] - wt
                                           : sc.pvg[i] + sc.pvg[j] + 2LL * wt;
      long long key = x;
      const bool rt = BOUNDS ? sc.ptab[i] != 0 : sc.pos[i] != 0, ct = BOUNDS ? sc.ptab[j] != 0 : sc.pos[j] != 0;
      if (!allowed(rt, ct, x, D))
        key = problem == P_MDP ? kMdpSentinel : maxbs_penalty(x);
      better_rec(bk, bi, key, idx);
    }
  }
  block_best(bk, bi, red);
  if (threadIdx.x == 0) {
    sc.recs[blockIdx.x].key = bk;
    sc.recs[blockIdx.x].idx = bi;
    __threadfence();
    s_last = atomicAdd(sc.counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  bk = LLONG_MIN;
  bi = LLONG_MAX;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x)
    better_rec(bk, bi, __ldcg(&sc.recs[b].key), __ldcg(&sc.recs[b].idx));
  block_best(bk, bi, red);
  if (threadIdx.x == 0) {
    out[0] = bk;
    out[1] = bi;
    *sc.counter = 0u;
  }
}

constexpr int kMaxDevices = 64;
std::mutex g_na_mu;
// The scratch array has one address per CUDA context: cached per device
// together with the id of the context it was looked up in, and looked up again
// when the caller's current context on that device is another one (a context
// the caller created itself, or a new primary context after a device reset,
// which may have the old one's address but not its id).
struct NaAddr {
  uint64_t ctx;
  void* addr;
};
NaAddr g_na_addr[kMaxDevices];

}  // namespace
}  // namespace tsb

using namespace tsb;

extern "C" ts_status ts_best_swap_noalloc(int32_t problem, int32_t n, int32_t m, int64_t iter,
                                          int64_t cur, int64_t best, const int64_t* d_rowptr,
                                          const int32_t* d_col, const int32_t* d_w,
                                          const int32_t* d_sol, const int64_t* d_vg,
                                          const int32_t* d_tab, int64_t* d_out, void* stream) {
  if (problem != TS_PROBLEM_MDP && problem != TS_PROBLEM_MAXBS) {
    set_error("ts_best_swap_noalloc: unknown problem");
    return TS_ERR_INVALID_ARG;
  }
  if (n < 2 || n > kNaMaxN) {
    set_error("ts_best_swap_noalloc: n must be in [2, " + std::to_string(kNaMaxN) +
              "]; the fixed scratch area holds that many positions");
    return TS_ERR_INVALID_ARG;
  }
  if (m < 1 || m >= n) { set_error("ts_best_swap_noalloc: need 1 <= m < n"); return TS_ERR_INVALID_ARG; }
  if (!d_rowptr || !d_col || !d_w || !d_sol || !d_vg || !d_tab || !d_out) {
    set_error("ts_best_swap_noalloc: NULL device pointer");
    return TS_ERR_INVALID_ARG;
  }
  int dev = 0;
  TS_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) { set_error("ts_best_swap_noalloc: device index out of range"); return TS_ERR_UNSUPPORTED; }
  void* base = nullptr;
  {
    // With the caller's device current: the scratch array's device address in
    // the current context (its name in host code is only a host-side
    // stand-in).  The first call in a context looks it up; later calls in the
    // same context reuse it.
    const uint64_t ctx = context_id();
    if (!ctx) {
      set_error("ts_best_swap_noalloc: no current CUDA context on the calling thread");
      return TS_ERR_CUDA;
    }
    std::lock_guard<std::mutex> lock(g_na_mu);
    if (g_na_addr[dev].ctx != ctx || !g_na_addr[dev].addr) {
      void* p = nullptr;
      cudaError_t e = cudaGetSymbolAddress(&p, g_na_scratch);
      if (e != cudaSuccess) return cuda_fail(e, "ts_best_swap_noalloc: cudaGetSymbolAddress");
      g_na_addr[dev].ctx = ctx;
      g_na_addr[dev].addr = p;
    }
    base = g_na_addr[dev].addr;
  }
  const NaView sc = view_of(base);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const long long P = (long long)m * (n - m);
  long long grid = (P + kNaTPB - 1) / kNaTPB;
  if (grid > kNaMaxCtas) grid = kNaMaxCtas;
  // Below about a million pairs visiting all of them costs less than the bounds
  // (Max Bisection: n = 700 11 us every pair, 24 bounded; n = 2,000 28 and 27;
  // n = 20,000 809 and 33).
  const bool bounds = P >= kNaBoundPairs;
  const auto stage = bounds ? k_na_stage<true> : k_na_stage<false>;
  const auto sweep = bounds ? k_na_sweep<true> : k_na_sweep<false>;
  stage<<<bounds ? kNaStageCtas : (n + kNaTPB - 1) / kNaTPB, kNaTPB, 0, st>>>(
      problem, n, m, (long long)iter, (long long)(best - cur), d_rowptr, d_col, d_w, d_sol,
      reinterpret_cast<const long long*>(d_vg), d_tab, sc);
  TS_CUDA(cudaGetLastError());
  sweep<<<(int)grid, kNaTPB, 0, st>>>(problem, n, m, (long long)cur, (long long)best, d_rowptr, d_col, d_w, d_sol, sc,
                                      d_out);
  TS_CUDA(cudaGetLastError());
  return TS_OK;
}
