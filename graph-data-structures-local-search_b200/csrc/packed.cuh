// packed.cuh -- one solve per CTA cluster: the start state, the iteration
// loop and the result of a solve whose state lives in a slot of HBM.  Shared
// by the batched form (batch.cu) and the server (serve.cu).
#pragma once
#include <cooperative_groups.h>

#include "cand.cuh"
#include "sweep.cuh"

namespace tsb {

struct BatchResultDev {
  long long iterations, evaluations, cur, best, best_true, perturbations;
  int32_t stopped, err;
  int32_t complete, given_up;  // complete: written when the solve has ended (served: until then iterations alone)
};

__device__ __forceinline__ long long block_sum(long long v, long long* sc) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sc[threadIdx.x >> 5] = v;
  __syncthreads();
  long long t = 0;
  for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sc[w];
  __syncthreads();
  return t;
}

// Lanes that share a row in the start and the result of a packed MDP solve.
constexpr int kRowLanes = 8;

// Start state of a solve in its slot, by one CTA: ascending ids per side
// (initialSolution, GPU-MDP-CSR.cu:479-500), contributions and objective
// (calculateVertexGain :502-519; computeGainsFromScratch /
// computeFitnessFromScratch, GPU-MAXBS-CSR.cu:197-219), WSwap matrix
// (calculateEdgeGain, GPU-MDP-WSwap.cu:607-626) and CSR neighbour positions.
// The same values as the plain solver's init kernels.  MDP takes
// eight lanes per selected row: the whole CTA on one row after another left
// most threads idle on rows of 5-50 entries (n = 5,000, m = 625, degree 25,
// start and result of a solve 0.56 -> 0.13 ms, with a WSwap matrix 1.1 -> 0.34).
// Bisection's rows stay a thread each: there are n of them (0.18 ms; eight
// lanes 0.41, a warp 0.76).
template <int PROB, int ST, class KeyT>
__device__ void slot_init(const DevGraph& g, const DevSolver<KeyT>& s, const int32_t* init,
                          long long max_iter, long long* sc, int32_t* s_cnt) {
  const int tid = threadIdx.x, T = blockDim.x;
  const int32_t n = s.n, m = s.m;
  int32_t* flag = s.pos;  // inside flags first, positions afterwards
  for (int32_t v = tid; v < n; v += T) flag[v] = PROB == P_MDP ? 0 : (init[v] == 0);
  __syncthreads();
  if (PROB == P_MDP)
    for (int32_t i = tid; i < m; i += T) flag[init[i]] = 1;
  __syncthreads();
  const int32_t per = (n + T - 1) / T, a0 = min(n, tid * per), a1 = min(n, a0 + per);
  int32_t cnt = 0;
  for (int32_t v = a0; v < a1; v++) cnt += flag[v];
  s_cnt[tid] = cnt;
  __syncthreads();
  int32_t x = 0;
#pragma unroll 8
  for (int t2 = 0; t2 < tid; t2++) x += s_cnt[t2];
  int32_t y = a0 - x;
  for (int32_t v = a0; v < a1; v++) {
    if (flag[v]) { s.sol_in[x] = v; flag[v] = x; x++; }
    else { s.sol_out[y] = v; flag[v] = m + y; y++; }
  }
  for (int32_t j = s.delta + tid; j < s.ldc; j += T) s.sol_out[j] = 0;
  for (int32_t i = tid; i < m; i += T) { s.vg_in[i] = 0; s.tab_in[i] = 0; }
  for (int32_t j = tid; j < s.ldc; j += T) { s.vg_out[j] = 0; s.tab_out[j] = 0; }
  if (ST == S_WSWAP) {  // whole rows of ldc (a multiple of 4) elements
    const long long words = (long long)s.n_row_blocks * Rows<ST>::R * s.ldc / (s.w16 ? 8 : 4);
    for (long long q = tid; q < words; q += T) reinterpret_cast<int4*>(s.W)[q] = make_int4(0, 0, 0, 0);
  }
  __syncthreads();
  long long acc = 0;
  if (PROB == P_MDP) {
    for (int32_t i = tid / kRowLanes; i < m; i += T / kRowLanes) {
      const int32_t u = s.sol_in[i];
#pragma unroll 4
      for (long long k = g.rowptr[u] + tid % kRowLanes; k < g.rowptr[u + 1]; k += kRowLanes) {
        const int2 e = g.adj[k];
        const int32_t p = s.pos[e.x];
        atomic_add_key(vg_at(s, p), (KeyT)e.y);
        if (p < m) acc += e.y;
      }
    }
  } else {
    for (int32_t z = tid; z < n; z += T) {
      const int32_t pz = s.pos[z];
      const bool side = pz < m;
      long long same = 0, opp = 0;
      for (long long k = g.rowptr[z]; k < g.rowptr[z + 1]; k++) {
        const int2 e = g.adj[k];
        if ((s.pos[e.x] < m) == side) {
          same += e.y;
        } else {
          opp += e.y;
          if (e.x > z) acc += e.y;
        }
      }
      *vg_at(s, pz) = (KeyT)(same - opp);
    }
  }
  if (ST == S_CSR)
    for (long long k = tid; k < g.entries; k += T) s.cpos[k] = s.pos[g.adj[k].x];
  if (ST == S_WSWAP) {
    for (int32_t i = tid / kRowLanes; i < m; i += T / kRowLanes) {
      const int32_t u = s.sol_in[i];
      const long long k0 = g.rowptr[u];
      for (long long k = k0 + tid % kRowLanes; k < g.rowptr[u + 1]; k += kRowLanes) {
        const int2 e = g.adj[k];
        if (k > k0 && g.adj[k - 1].x == e.x) continue;  // first entry of a duplicated pair
        const int32_t p = s.pos[e.x];
        if (p >= m) w_set(s, (long long)i * s.ldc + (p - m), e.y);
      }
    }
  }
  long long obj = block_sum(acc, sc);
  if (PROB == P_MDP) obj /= 2;
  if (tid == 0) {
    DevState z;
    memset(&z, 0, sizeof(z));
    z.cur = obj;
    z.best = obj;
    z.target = max_iter;
    z.pert_limit = s.draw_events;  // every event of the solve is staged
    *s.st = z;
  }
  __syncthreads();
}

// Best solution (the current one with the moves after the last improvement
// undone; a swap is its own inverse), its objective from the graph, result.
template <int PROB, class KeyT>
__device__ void slot_finish(const DevGraph& g, const DevSolver<KeyT>& s, BatchResultDev* out,
                            int32_t* best_out, long long* sc) {
  const int tid = threadIdx.x, T = blockDim.x;
  const DevState* st = s.st;
  if (tid == 0) {
    const long long to = min(__ldcg(&st->log_n), s.log_cap);
    const long long from = __ldcg(&st->best_log_n);
    for (long long q = to - 1; q >= from; q--) {
      const int2 mv = s.movelog[q];
      const int32_t a = s.sol_in[mv.x];
      s.sol_in[mv.x] = s.sol_out[mv.y];
      s.sol_out[mv.y] = a;
    }
  }
  __syncthreads();
  for (int32_t v = tid; v < s.n; v += T) s.pos[v] = 0;
  __syncthreads();
  for (int32_t i = tid; i < s.m; i += T) s.pos[s.sol_in[i]] = 1;
  __syncthreads();
  long long acc = 0;
  constexpr int kLanes = PROB == P_MDP ? kRowLanes : 1;
  for (int32_t x = tid / kLanes; x < (PROB == P_MDP ? s.m : s.n); x += T / kLanes) {
    const int32_t a = PROB == P_MDP ? s.sol_in[x] : x;
    const int32_t fa = s.pos[a];
    for (long long k = g.rowptr[a] + tid % kLanes; k < g.rowptr[a + 1]; k += kLanes) {
      const int2 e = g.adj[k];
      const int32_t fz = s.pos[e.x];
      if (PROB == P_MDP) {
        if (fz) acc += e.y;
      } else if (e.x > a && fa != fz) {
        acc += e.y;
      }
    }
  }
  long long bt = block_sum(acc, sc);
  if (PROB == P_MDP) bt /= 2;
  if (PROB == P_MDP)
    for (int32_t i = tid; i < s.m; i += T) best_out[i] = s.sol_in[i];
  else
    for (int32_t v = tid; v < s.n; v += T) best_out[v] = s.pos[v] ? 0 : 1;
  if (tid == 0) {
    BatchResultDev r;
    r.iterations = __ldcg(&st->iter);
    r.evaluations = __ldcg(&st->evaluations);
    r.cur = __ldcg(&st->cur);
    r.best = __ldcg(&st->best);
    r.best_true = bt;
    r.perturbations = __ldcg(&st->pert_moves);
    r.stopped = __ldcg(&st->stopped);
    r.err = __ldcg(&st->err);
    r.complete = 1;
    *out = r;
  }
  __syncthreads();
}

constexpr int32_t kTryFails = 4;   // tries of the candidate pass in a row that settle nothing
constexpr int32_t kTrySweeps = 8;  // and the sweeps between two more of them, at most

// Shared memory of the candidate pass in kernels that have it.
template <bool CAND, class KeyT>
struct CandSharedIf {
  CandShared<KeyT> v;
};
template <class KeyT>
struct CandSharedIf<false, KeyT> {};

// Runs a solve's iterations up to `stop_at` with the CTAs of the calling
// cluster: the candidate pass where the solve has it, else (and for the
// iterations it leaves) round-robin tiles, the leader merging the records over
// distributed shared memory and applying the move.  A try of the candidate pass
// that stops at once moves the whole state to shared memory and back: once four
// in a row settled nothing, up to eight sweeps come between two of them
// (bisection of n = 150 with ties everywhere, 2,000 iterations: 149 ms with a try
// at each, 121 with fewer, 119 with the sweep pinned).  Not sooner: a sweep on few
// CTAs takes many times the pass's iteration, and ties that pass are common in
// graphs of equal weights.
// Every CTA of the cluster calls it.
//
// CAND: the solve has the candidate pass.  Kernels for solves without it
// (pinned sweeps above all) are compiled without it: its registers and its code
// beside the sweep's cost them up to two thirds (64 MDP solves of n = 2,000 on
// the tile pass 23.5 -> 38.6 ms, 300 bisections 112 -> 140, on the per-row pass
// 302 -> 387).
//
// give_up > 0: a kernel without the pass can sweep the solve, on that many times
// the CTAs.  It returns false once eight iterations were swept and their share
// says that this is the better way.  Iterations without an allowed pair do not
// count: the pass saves a sweep there.  A served solve goes on from its state;
// a batched one starts again, so that the rest must be worth all of it.
//
// TIMED (served): sweeps end after `budget_ns` too, wherever the search is then.
// How many iterations of a solve the candidate pass will leave to them is not
// known beforehand, and other requests wait for the launch.
template <int PROB, int ST, class KeyT, bool CAND, bool TIMED>
__device__ bool cluster_iterate(const DevGraph& g, const DevSolver<KeyT>& s, long long stop_at,
                                [[maybe_unused]] long long budget_ns, [[maybe_unused]] int32_t give_up,
                                cooperative_groups::cluster_group& cl, TailShared& sh, CtaRec& s_rec,
                                CandSharedIf<CAND, KeyT>& s_cand) {
  [[maybe_unused]] extern __shared__ __align__(16) unsigned char smem_raw[];
  const unsigned rank = cl.block_rank(), cs = cl.num_blocks();
  const int tid = threadIdx.x;
  const int ntiles = s.n_row_blocks * s.n_chunks;
  const DevState* st = s.st;
  const long long first = CAND ? __ldcg(&st->iter) : 0;
  long long at = first;                     // the iteration before the last sweep
  bool moving = false;                      // it was one that moves, if it finds a pair
  int32_t fails = 0, wait = 0, swept = 0;   // tries in a row that settled nothing; sweeps until the next; swept iterations
  bool finished = true;
  [[maybe_unused]] __shared__ int32_t late;       // the leader's word on the time
  [[maybe_unused]] const long long began = TIMED ? (long long)global_ns() : 0;
  for (;;) {
    const bool tried = CAND && wait == 0;
    if constexpr (CAND)
      if (tried && cand_run<PROB, ST, KeyT>(g, s, stop_at, LLONG_MAX, cl, s_cand.v, smem_raw) == kCandEnd) break;
    // every CTA reads the same state: the leader wrote it before the last barrier
    const long long it = __ldcg(&st->iter);
    if (__ldcg(&st->done) || it >= stop_at) break;
    const int mode = __ldcg(&st->mode);
    if constexpr (CAND) {
      if (moving && it > at) swept++;
      if (tried) {
        // (a try that found no allowed pair saved the sweep that would find it)
        fails = mode != 0 || it > at + moving ? 0 : fails + 1;
        wait = fails <= kTryFails ? 1 : min(1 << (fails - kTryFails), kTrySweeps);
      }
      if (give_up && swept >= 8) {
        const float made = (float)(it - first), rest = (float)(stop_at - it), all = (float)(stop_at - first);
        const float better = TIMED ? 2.f * swept - made
                             : give_up > 1 ? 0.8f * rest * swept * give_up - all * made
                                           : (2.f * swept >= made ? all - 32.f * made : 0.f);
        if (better > 0.f) {
          finished = false;
          break;
        }
      }
      wait--;
      moving = mode == 0;
      at = it;
    }
    const long long D64 = __ldcg(&st->best) - __ldcg(&st->cur);
    long long k = LLONG_MIN, i = LLONG_MAX;
    for (int t = (int)rank; t < ntiles; t += (int)cs) {
      long long tk, ti;
      // k (valid in thread 0, the thread that uses it): the CTA's best so far
      tile_eval<PROB, ST, KeyT, true>(g, s, mode, it, D64, t / s.n_chunks, t % s.n_chunks, tk, ti, sh,
                                      mode == 0 ? k : LLONG_MIN);
      if (tid == 0) better_rec(k, i, tk, ti);
    }
    if (tid == 0) { s_rec.key = k; s_rec.idx = i; }
    cl.sync();
    if (rank == 0) {
      if (tid == 0)
        for (unsigned r = 1; r < cs; r++) {
          const CtaRec* o = cl.map_shared_rank(&s_rec, r);
          better_rec(k, i, o->key, o->idx);
        }
      decide_apply<PROB, ST, KeyT>(g, s, mode, k, i, sh);
      __threadfence();
      if (TIMED && tid == 0) late = (long long)global_ns() - began > budget_ns;
    }
    cl.sync();
    if (TIMED && *cl.map_shared_rank(&late, 0)) break;
  }
  if (TIMED) cl.sync();  // the leader stays until its word is read
  return finished;
}

}  // namespace tsb
