// cand.cuh -- the candidate pass: exact best swap of an iteration from the
// few rows and columns that can hold it, iterations run by one CTA cluster.
//
// Every gain has the form  A[i] + B[j] + c*w(i,j)  (MDP: -vg[u] + vg[v] - w,
// Max Bisection: vg[u] + vg[v] + 2w; the reference evaluates it for all m*(n-m)
// pairs, src/mdp/GPU-MDP-CSR.cu:567-584, src/maxbisection/GPU-MAXBS-CSR.cu:337-353).
// With Am, Bm the largest A and B and LB the gain of one known allowed pair, a
// pair can reach LB only if A[i] >= LB - Bm - p and B[j] >= LB - Am - p, where
// p >= 0 bounds c*w from above.  So an iteration is
//   1. the maxima of A and B over all and over the non-tabu positions (and
//      the lowest position of each): O(n), from shared memory;
//   2. the seed pairs (the two argmax pairs) with their weight from the lookup
//      structure: LB.  An MDP seed of non-adjacent vertices already is the
//      answer: nothing can exceed Am + Bm, and no tie has a lower position;
//   3. otherwise the rows and columns within the bound.  N: where c*w <= 0 the
//      pairs with A + B >= LB, each looked up in the structure.  E: where
//      c*w > 0 the candidate rows' own entries whose neighbour is a candidate
//      column (a bitmap by vertex in shared memory), evaluated exactly;
//   4. the same argmax rule as the sweeps (largest allowed gain, then lowest
//      flat index) and the move.
// Tabu pairs count only above best - cur, so their threshold is
// max(LB, best - cur + 1).  Nothing is estimated: a pair that is not evaluated
// is below LB.  When the candidates are too many (ties everywhere), or no pair
// is allowed, the pass hands the iteration to the sweeps (sweep.cuh).
//
// Each CTA of the cluster holds a slice of the rows' and columns' contributions,
// tabu stamps and vertex ids in shared memory for the whole launch; a move's
// contribution updates are shared-memory atomics on the owner CTA.  What bounds
// it is latency: two to four cluster barriers and about five dependent L2 round
// trips per iteration, at any size.  Measured per iteration, sweeps before and
// this pass after: MDP ER n = 2,000 (CSR) 17.0 -> 3.9 us; dense n = 2,000
// (CSR+BB) 42.7 -> 13.7; Chung-Lu n = 200,000 (Hash) 811 -> 5.9; bisection
// conflict graph n = 100,000 (CSR) 153 -> 14.4, n = 60,001 (WSwap) 390 -> 11.9,
// n = 30,011 (CSR+Bitset) 179 -> 11.1; n = 10,007 with 64-bit contributions
// (CSR+BB) 115 -> 14.9.
#pragma once
#include <cooperative_groups.h>

#include "sweep.cuh"

namespace tsb {

constexpr int kCandTPB = 512;        // threads per CTA of the plain form
constexpr int kCandMaxCluster = 16;
constexpr int kCandList = 2048;      // candidates a CTA can hold per side
constexpr int kCandStage = 1024;     // candidate columns staged per round of N
constexpr int kCandHeavy = 1024;     // E: rows of more entries are walked by the whole CTA
constexpr int kCandHeavyList = 64;

enum { kCandEnd = 0, kCandBail = 1 };

struct CandLayout {
  uint32_t va, vb, ta, tb, ua, ub, rl, cl, map, total;
  uint32_t map_bytes;
  int32_t rcap, ccap;  // list lengths
};
// Shared memory of one CTA: rpc rows and cpc columns (multiples of 4), lists,
// and one area that is the candidate-column bitmap (E) or the staged columns (N).
__host__ __device__ inline CandLayout cand_layout(int32_t n, int32_t rpc, int32_t cpc, int kb, bool edges) {
  CandLayout L;
  uint32_t off = 0;
  L.va = off; off += (uint32_t)kb * rpc;
  L.vb = off; off += (uint32_t)kb * cpc;
  L.ta = off; off += 4u * rpc;
  L.tb = off; off += 4u * cpc;
  L.ua = off; off += 4u * rpc;
  L.ub = off; off += 4u * cpc;
  L.rcap = rpc < kCandList ? rpc : kCandList;
  L.ccap = cpc < kCandList ? cpc : kCandList;
  L.rl = off; off += 4u * (uint32_t)L.rcap;
  L.cl = off; off += 4u * (uint32_t)L.ccap;
  L.map = off;
  L.map_bytes = edges ? 16u * (uint32_t)((n + 127) / 128) : 0u;
  const uint32_t stage = (uint32_t)(8 + kb) * kCandStage;
  off += L.map_bytes > stage ? L.map_bytes : stage;
  L.total = off;
  return L;
}

template <class KeyT>
struct alignas(16) CandTop {  // a CTA's maxima: rows, columns; non-tabu, all
  KeyT k[4];                  // row nt, row all, col nt, col all
  int32_t i[4];
  int32_t v[4];
};
template <class KeyT>
struct alignas(16) CandBest {  // a CTA's best evaluated pair
  KeyT key, a, b;              // gain; raw contributions of the pair
  int32_t i, j, u, v;          // j < 0: none
};
struct CandScalars {
  long long iter, cur, best, evaluations, isi, log_n, best_log_n, trace_n, pert_events, pert_moves;
  int32_t done, stopped, err, mode, perturb, pad;
};
template <class KeyT>
struct CandShared {
  CandTop<KeyT> top[kCandMaxCluster];
  CandBest<KeyT> rec[kCandMaxCluster];
  CandBest<KeyT> wbest[kCandTPB / 32];
  KeyT wk[4][kCandTPB / 32];
  int32_t wi[4][kCandTPB / 32];
  int32_t nrow, ncol, nheavy, wuv;
  int32_t pre[kCandMaxCluster + 1];
  int32_t heavy[kCandHeavyList];
  CandScalars sc;
};

__device__ __forceinline__ int32_t lane_min(int32_t v) { return __reduce_min_sync(0xffffffffu, v); }

// Largest key, then lowest index, over a warp; all lanes get the result.
template <class KeyT>
__device__ __forceinline__ void warp_top(KeyT& k, int32_t& i) {
  const KeyT m = warp_max(k);
  i = lane_min(k == m ? i : INT_MAX);
  k = m;
}

// Candidate (i, j) precedes the held best: larger key, then lower flat index.
template <class KeyT>
__device__ __forceinline__ void cand_better(CandBest<KeyT>& x, const CandBest<KeyT>& y) {
  if (y.j < 0) return;
  if (x.j < 0 || y.key > x.key || (y.key == x.key && (y.i < x.i || (y.i == x.i && y.j < x.j)))) x = y;
}

template <class KeyT>
__device__ __forceinline__ void warp_best(CandBest<KeyT>& b) {
  const KeyT none = KeyLim<KeyT>::none;
  const KeyT k = b.j < 0 ? none : b.key;
  const KeyT m = warp_max(k);
  const bool has = b.j >= 0 && k == m;
  const int32_t i = lane_min(has ? b.i : INT_MAX);
  const int32_t j = lane_min(has && b.i == i ? b.j : INT_MAX);
  const unsigned who = __ballot_sync(0xffffffffu, has && b.i == i && b.j == j);
  if (!who) { b.j = -1; return; }
  const int src = __ffs(who) - 1;
  b.key = m;
  b.i = i;
  b.j = j;
  b.a = __shfl_sync(0xffffffffu, b.a, src);
  b.b = __shfl_sync(0xffffffffu, b.b, src);
  b.u = __shfl_sync(0xffffffffu, b.u, src);
  b.v = __shfl_sync(0xffffffffu, b.v, src);
}

// First entry of v in a sorted CSR row by the whole warp: 32 probes a step.
__device__ __forceinline__ int32_t warp_row_lookup(const int2* row, int32_t len, int32_t v) {
  const int lane = threadIdx.x & 31;
  int32_t lo = 0;
  while (len > 32) {
    const int32_t step = (len + 31) >> 5;
    const int32_t at = (lane + 1) * step - 1;
    const bool below = at < len && __ldg(&row[lo + at].x) < v;
    const int32_t skip = __popc(__ballot_sync(0xffffffffu, below)) * step;
    lo += skip;
    len = min(step, len - skip);
  }
  int2 e = make_int2(-1, 0);
  if (lane < len) e = __ldg(row + lo + lane);
  const unsigned hit = __ballot_sync(0xffffffffu, e.x == v);
  return hit ? __shfl_sync(0xffffffffu, e.y, __ffs(hit) - 1) : 0;
}
__device__ __forceinline__ int32_t row_lookup(const int2* row, int32_t len, int32_t v) {
  const int32_t* k = reinterpret_cast<const int32_t*>(row);
  return bb_lower<2>(k, k + 1, len, v);
}

// w(i, j) of the seed pair, by a whole warp, in the solver's structure.  A CSR
// row is searched from the end of smaller degree (both rows hold the entry,
// duplicates in the same order); the bitmaps answer first where there are any.
template <int ST, class KeyT>
__device__ __forceinline__ int32_t cand_seed_w(const DevGraph& g, const DevSolver<KeyT>& s, int32_t i, int32_t j,
                                               int32_t u, int32_t v) {
  if (ST == S_WSWAP) return w_get<true>(s, (long long)i * s.ldc + j);
  if (ST == S_HASH) {
    const long long b = __ldg(g.hoff + u);
    const long long cap = __ldg(g.hoff + u + 1) - b;
    return hash_probe(g.hkey + b, g.hval + b, (uint32_t)(cap / 4 - 1), hash_gshift(cap), v);
  }
  if (ST == S_BITSET || ST == S_BITSET_BB) {
    if (!bit_test(g.bits + (long long)u * g.wpr, v)) return 0;
  }
  const long long ru = __ldg(g.rowptr + u), rv = __ldg(g.rowptr + v);
  const int32_t du = (int32_t)(__ldg(g.rowptr + u + 1) - ru), dv = (int32_t)(__ldg(g.rowptr + v + 1) - rv);
  return du <= dv ? warp_row_lookup(g.adj + ru, du, v) : warp_row_lookup(g.adj + rv, dv, u);
}
// The same for one thread's pair.
template <int ST, class KeyT>
__device__ __forceinline__ int32_t cand_pair_w(const DevGraph& g, const DevSolver<KeyT>& s, int32_t i, int32_t j,
                                               int32_t u, int32_t v) {
  if (ST == S_WSWAP) return w_get<true>(s, (long long)i * s.ldc + j);
  if (ST == S_HASH) {
    const long long b = __ldg(g.hoff + u);
    const long long cap = __ldg(g.hoff + u + 1) - b;
    return hash_probe(g.hkey + b, g.hval + b, (uint32_t)(cap / 4 - 1), hash_gshift(cap), v);
  }
  if (ST == S_BITSET || ST == S_BITSET_BB) {
    if (!bit_test(g.bits + (long long)u * g.wpr, v)) return 0;
  }
  const long long ru = __ldg(g.rowptr + u), rv = __ldg(g.rowptr + v);
  const int32_t du = (int32_t)(__ldg(g.rowptr + u + 1) - ru), dv = (int32_t)(__ldg(g.rowptr + v + 1) - rv);
  return du <= dv ? row_lookup(g.adj + ru, du, v) : row_lookup(g.adj + rv, dv, u);
}

// One thread's maxima over a slice: non-tabu and all, lowest index of each
// (its indices ascend, so a strict comparison keeps the lowest).
template <bool NEG, class KeyT>
__device__ __forceinline__ void cand_scan(const KeyT* val, const int32_t* tab, int32_t cnt, int32_t now, KeyT& nt,
                                          int32_t& int_, KeyT& all, int32_t& iall) {
  for (int32_t q = (int32_t)threadIdx.x * 4; q < cnt; q += (int32_t)blockDim.x * 4) {
    KeyT x[4];
    int32_t t[4];
    const int4 t4 = *reinterpret_cast<const int4*>(tab + q);
    t[0] = t4.x; t[1] = t4.y; t[2] = t4.z; t[3] = t4.w;
    if constexpr (sizeof(KeyT) == 4) {
      const int4 v4 = *reinterpret_cast<const int4*>(val + q);
      x[0] = v4.x; x[1] = v4.y; x[2] = v4.z; x[3] = v4.w;
    } else {
      const longlong2 a = *reinterpret_cast<const longlong2*>(val + q), b = *reinterpret_cast<const longlong2*>(val + q + 2);
      x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (q + k >= cnt) break;
      const KeyT y = NEG ? -x[k] : x[k];
      if (y > all) { all = y; iall = q + k; }
      if (t[k] <= now && y > nt) { nt = y; int_ = q + k; }
    }
  }
}

// Runs iterations up to `stop_at`, at most `budget` of them, by the calling
// cluster (every CTA, all threads).  State is read from the solver's arrays at
// entry and written back at exit.  Returns kCandEnd, or kCandBail when the
// next iteration needs a sweep (too many candidates, or the exact pass).
template <int PROB, int ST, class KeyT>
__device__ int cand_run(const DevGraph& g, const DevSolver<KeyT>& s, long long stop_at, long long budget,
                        cooperative_groups::cluster_group& cl, CandShared<KeyT>& sh, unsigned char* smem) {
  using Lim = KeyLim<KeyT>;
  const int T = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = T >> 5;
  const int nb = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int32_t m = s.m, delta = s.delta, rpc = s.cand_rpc, cpc = s.cand_cpc;
  const bool edges = s.cand_plus > 0;
  const CandLayout L = cand_layout(s.n, rpc, cpc, sizeof(KeyT), edges);
  KeyT* va = reinterpret_cast<KeyT*>(smem + L.va);
  KeyT* vb = reinterpret_cast<KeyT*>(smem + L.vb);
  int32_t* ta = reinterpret_cast<int32_t*>(smem + L.ta);
  int32_t* tb = reinterpret_cast<int32_t*>(smem + L.tb);
  int32_t* ua = reinterpret_cast<int32_t*>(smem + L.ua);
  int32_t* ub = reinterpret_cast<int32_t*>(smem + L.ub);
  int32_t* rl = reinterpret_cast<int32_t*>(smem + L.rl);
  int32_t* cll = reinterpret_cast<int32_t*>(smem + L.cl);
  uint32_t* map = reinterpret_cast<uint32_t*>(smem + L.map);
  const int32_t row0 = rank * rpc, col0 = rank * cpc;
  const int32_t nr = max(0, min(rpc, m - row0)), nc = max(0, min(cpc, delta - col0));
  const KeyT plus = (KeyT)s.cand_plus;
  const bool fav = s.cand_fav != 0;

  auto slot_of = [&](int32_t p) -> KeyT* {  // contribution of position p, in its owner's shared memory
    if (p < m) {
      const int32_t o = p / rpc;
      return cl.map_shared_rank(va, o) + (p - o * rpc);
    }
    const int32_t q = p - m, o = q / cpc;
    return cl.map_shared_rank(vb, o) + (q - o * cpc);
  };

  for (int32_t i = tid; i < nr; i += T) {
    va[i] = __ldcg(s.vg_in + row0 + i);
    ta[i] = __ldcg(s.tab_in + row0 + i);
    ua[i] = __ldcg(s.sol_in + row0 + i);
  }
  for (int32_t j = tid; j < nc; j += T) {
    vb[j] = __ldcg(s.vg_out + col0 + j);
    tb[j] = __ldcg(s.tab_out + col0 + j);
    ub[j] = __ldcg(s.sol_out + col0 + j);
  }
  for (uint32_t q = tid; q < L.map_bytes / 16; q += T) reinterpret_cast<uint4*>(map)[q] = make_uint4(0, 0, 0, 0);
  if (tid == 0) {
    const DevState* st = s.st;
    CandScalars& c = sh.sc;
    c.iter = __ldcg(&st->iter); c.cur = __ldcg(&st->cur); c.best = __ldcg(&st->best);
    c.evaluations = __ldcg(&st->evaluations); c.isi = __ldcg(&st->isi);
    c.log_n = __ldcg(&st->log_n); c.best_log_n = __ldcg(&st->best_log_n); c.trace_n = __ldcg(&st->trace_n);
    c.pert_events = __ldcg(&st->pert_events); c.pert_moves = __ldcg(&st->pert_moves);
    c.done = __ldcg(&st->done); c.stopped = __ldcg(&st->stopped); c.err = __ldcg(&st->err);
    c.mode = __ldcg(&st->mode);
    c.perturb = 0;
  }
  const long long pert_base = __ldcg(&s.st->pert_base), pert_limit = __ldcg(&s.st->pert_limit);
  cl.sync();

  // One swap's updates by the whole cluster: contributions along the rows of u
  // and v (shared-memory atomics on the owners), the swapped slots, positions,
  // CSR cpos and the clearing half of the WSwap patch.  a, b: contributions of
  // u and v before the swap.  Ends with a cluster barrier.
  auto apply = [&](int32_t iu, int32_t jv, int32_t u, int32_t v, KeyT a, KeyT b, int32_t stamp_row, int32_t stamp_col) {
    const long long su = __ldg(g.rowptr + u), sv = __ldg(g.rowptr + v);
    const int32_t nu = (int32_t)(__ldg(g.rowptr + u + 1) - su), nv = (int32_t)(__ldg(g.rowptr + v + 1) - sv);
    const int32_t total = nu + nv;
    for (int32_t k = rank * T + tid; k < total; k += nb * T) {
      const bool from_u = k < nu;
      const long long at = from_u ? su + k : sv + (k - nu);
      const int2 e = __ldg(g.adj + at);
      const int32_t z = e.x, w = e.y;
      if (ST == S_CSR) s.cpos[__ldg(g.rev + at)] = from_u ? m + jv : iu;  // new position of u / v
      if (PROB == P_MAXBS && from_u && z == v && (k == 0 || __ldg(&g.adj[at - 1].x) != z))
        *cl.map_shared_rank(&sh.wuv, 0) = w;
      KeyT d;
      if (z == u || z == v) {  // the moved vertices themselves: their slots after the swap
        const bool z_in = z == u;
        if (PROB == P_MDP) d = from_u ? -(KeyT)w : (KeyT)w;
        else d = (from_u == z_in) ? (KeyT)2 * (KeyT)w : -(KeyT)2 * (KeyT)w;  // negated with the slot
        atomic_add_key(slot_of(z_in ? m + jv : iu), d);
        continue;
      }
      const int32_t p = __ldcg(s.pos + z);
      if (PROB == P_MDP) {
        d = from_u ? -(KeyT)w : (KeyT)w;
      } else {
        const bool z_in = p < m;
        d = (from_u == z_in) ? -(KeyT)2 * (KeyT)w : (KeyT)2 * (KeyT)w;
      }
      atomic_add_key(slot_of(p), d);
      if (ST == S_WSWAP) {
        // row iu stops being u's, column jv stops being v's
        if (from_u && p >= m) w_set(s, (long long)iu * s.ldc + (p - m), 0);
        if (!from_u && p < m) w_set(s, (long long)p * s.ldc + jv, 0);
      }
    }
    if (rank == 0 && tid == T - 1) {
      // v takes slot iu, u takes slot jv; added as a difference, so that it
      // commutes with the entries' updates of the two slots
      const KeyT fa = PROB == P_MDP ? a : -a, fb = PROB == P_MDP ? b : -b;
      atomic_add_key(slot_of(iu), fb - a);
      atomic_add_key(slot_of(m + jv), fa - b);
      const int32_t oi = iu / rpc, oj = jv / cpc;
      cl.map_shared_rank(ua, oi)[iu - oi * rpc] = v;
      cl.map_shared_rank(ub, oj)[jv - oj * cpc] = u;
      int32_t* pa = cl.map_shared_rank(ta, oi) + (iu - oi * rpc);
      int32_t* pb = cl.map_shared_rank(tb, oj) + (jv - oj * cpc);
      if (stamp_row >= 0) {
        *pa = stamp_row;
        *pb = stamp_col;
      } else {  // perturbation: the stamps travel with the vertices
        const int32_t t = *pa;
        *pa = *pb;
        *pb = t;
      }
      s.pos[u] = m + jv;
      s.pos[v] = iu;
    }
    cl.sync();
    if (ST == S_WSWAP) {
      // the setting half: row iu at v's outside neighbours, column jv at u's
      // inside ones, first entry of a duplicated pair, (iu, jv) left alone
      for (int32_t k = rank * T + tid; k < total; k += nb * T) {
        const bool from_u = k < nu;
        const long long at = from_u ? su + k : sv + (k - nu);
        const int2 e = __ldg(g.adj + at);
        if (e.x == u || e.x == v) continue;
        if (at != (from_u ? su : sv) && __ldg(&g.adj[at - 1].x) == e.x) continue;
        const int32_t p = __ldcg(s.pos + e.x);
        if (!from_u && p >= m) w_set(s, (long long)iu * s.ldc + (p - m), e.y);
        if (from_u && p < m) w_set(s, (long long)p * s.ldc + jv, e.y);
      }
    }
  };
  auto trace_put = [&](long long iter, long long idx, long long key, int32_t kind, int32_t t1, int32_t t2) {
    CandScalars& c = sh.sc;
    if (rank == 0 && s.trace && c.trace_n < s.trace_cap) {
      TraceRec r;
      r.iter = iter; r.idx = idx; r.key = key; r.cur = c.cur; r.best = c.best;
      r.kind = kind; r.tenure = t1; r.tenure2 = t2; r.pad = 0;
      s.trace[c.trace_n] = r;
    }
    c.trace_n++;
  };
  auto log_move = [&](int32_t iu, int32_t jv) {
    CandScalars& c = sh.sc;
    if (c.log_n < s.log_cap) {
      if (rank == 0) s.movelog[c.log_n] = make_int2(iu, jv);
    } else {
      c.err |= E_LOG_FULL;
    }
    c.log_n++;
  };

  int status = kCandEnd;
  for (;;) {
    const long long iter = sh.sc.iter;
    if (sh.sc.done || iter >= stop_at || budget <= 0) break;
    if (sh.sc.mode != 0) { status = kCandBail; break; }
    const long long D64 = sh.sc.best - sh.sc.cur;
    const int32_t now = (int32_t)min(iter, (long long)INT32_MAX);  // stamps are 32-bit
    KeyT D = Lim::clampD(D64);
    if (sizeof(KeyT) == 4 && D == (KeyT)INT32_MAX) D = (KeyT)(INT32_MAX - 1);  // D + 1 is formed below

    // ---- 1. maxima of the slices
    KeyT k4[4];
    int32_t i4[4];
#pragma unroll
    for (int q = 0; q < 4; q++) { k4[q] = Lim::none; i4[q] = INT_MAX; }
    cand_scan<PROB == P_MDP, KeyT>(va, ta, nr, now, k4[0], i4[0], k4[1], i4[1]);
    cand_scan<false, KeyT>(vb, tb, nc, now, k4[2], i4[2], k4[3], i4[3]);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      warp_top<KeyT>(k4[q], i4[q]);
      if (lane == 0) { sh.wk[q][warp] = k4[q]; sh.wi[q][warp] = i4[q]; }
    }
    if (tid == 0) { sh.nrow = 0; sh.ncol = 0; sh.nheavy = 0; }
    __syncthreads();
    if (warp == 0) {
      CandTop<KeyT> t;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        KeyT k = lane < nw ? sh.wk[q][lane] : Lim::none;
        int32_t i = lane < nw ? sh.wi[q][lane] : INT_MAX;
        warp_top<KeyT>(k, i);
        t.k[q] = k;
        t.i[q] = k == Lim::none ? -1 : i + (q < 2 ? row0 : col0);
        t.v[q] = k == Lim::none ? -1 : (q < 2 ? ua[i] : ub[i]);
      }
      if (lane < nb) *cl.map_shared_rank(&sh.top[rank], lane) = t;
    }
    cl.sync();
    // every warp: the cluster's maxima
    KeyT gk[4];
    int32_t gi[4], gv[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      KeyT k = lane < nb ? sh.top[lane].k[q] : Lim::none;
      int32_t i = k == Lim::none ? INT_MAX : sh.top[lane].i[q];
      warp_top<KeyT>(k, i);
      gk[q] = k;
      gi[q] = i;
      gv[q] = k == Lim::none ? -1 : sh.top[q < 2 ? i / rpc : i / cpc].v[q];
    }
    const KeyT Am = gk[0], AA = gk[1], Bm = gk[2], BA = gk[3];
    const bool nt_ok = Am != Lim::none && Bm != Lim::none;

    // ---- 2. seeds and thresholds
    CandBest<KeyT> best;
    best.j = -1;
    KeyT c1 = 0, c2 = 0;  // c*w of the non-tabu and of the overall seed pair
    const bool one_seed = nt_ok && gi[0] == gi[1] && gi[2] == gi[3];
    const bool asp = AA + BA + plus > D;  // some tabu pair might be aspirated
    if (!fav) {
      if (nt_ok) {
        const int32_t w = cand_seed_w<ST, KeyT>(g, s, gi[0], gi[2], gv[0], gv[2]);
        c1 = PROB == P_MDP ? -(KeyT)w : (KeyT)2 * (KeyT)w;
      }
      if (one_seed) {
        c2 = c1;
      } else if (asp) {
        const int32_t w = cand_seed_w<ST, KeyT>(g, s, gi[1], gi[3], gv[1], gv[3]);
        c2 = PROB == P_MDP ? -(KeyT)w : (KeyT)2 * (KeyT)w;
      }
    }
    KeyT LB = Lim::none;
    if (nt_ok) {
      best.key = LB = Am + Bm + c1;
      best.i = gi[0]; best.j = gi[2]; best.u = gv[0]; best.v = gv[2];
      best.a = PROB == P_MDP ? -Am : Am;
      best.b = Bm;
    }
    if (!one_seed && AA + BA + c2 > D) {
      CandBest<KeyT> y;
      y.key = AA + BA + c2;
      y.i = gi[1]; y.j = gi[3]; y.u = gv[1]; y.v = gv[3];
      y.a = PROB == P_MDP ? -AA : AA;
      y.b = BA;
      if (y.key > LB) LB = y.key;
      cand_better(best, y);
    }
    const KeyT LT = LB > D ? LB : D + 1;  // threshold of pairs with a tabu side
    // N: non-adjacent pairs, and adjacent ones with c*w <= 0, bounded by A + B
    const bool need_n = !fav && ((nt_ok && c1 < 0 && Am + Bm >= LB) || (c2 < 0 && asp && AA + BA >= LT));
    // E: adjacent pairs with c*w > 0, bounded by A + B + plus
    const bool need_e = edges && ((nt_ok && Am + Bm + plus >= LB) || AA + BA + plus >= LT);

    bool bail = false;
    if (need_n || need_e) {
      CandBest<KeyT> mine;
      mine.j = -1;
      auto collect = [&](KeyT pl, bool ids) {
        for (int32_t i = tid; i < nr; i += T) {
          const KeyT x = PROB == P_MDP ? -va[i] : va[i];
          const bool nt = ta[i] <= now;
          if ((nt && nt_ok && x + Bm + pl >= LB) || x + BA + pl >= LT) {
            const int32_t at = atomicAdd(&sh.nrow, 1);
            if (at < L.rcap) rl[at] = i;
          }
        }
        for (int32_t j = tid; j < nc; j += T) {
          const KeyT x = vb[j];
          const bool nt = tb[j] <= now;
          if ((nt && nt_ok && x + Am + pl >= LB) || x + AA + pl >= LT) {
            const int32_t at = atomicAdd(&sh.ncol, 1);
            if (at < L.ccap) cll[at] = ids ? ub[j] : j;
          }
        }
        cl.sync();
        // counts of the cluster: column prefix, largest lists
        const int32_t cr = lane < nb ? *cl.map_shared_rank(&sh.nrow, lane) : 0;
        const int32_t cc = lane < nb ? *cl.map_shared_rank(&sh.ncol, lane) : 0;
        int32_t incl = cc;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int32_t t = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += t;
        }
        if (warp == 0 && lane < nb) sh.pre[lane + 1] = incl;
        if (tid == 0) sh.pre[0] = 0;
        const int32_t mr = __reduce_max_sync(0xffffffffu, cr), mc = __reduce_max_sync(0xffffffffu, cc);
        const int32_t tc = __shfl_sync(0xffffffffu, incl, 31);
        if (mr > L.rcap || mc > L.ccap) bail = true;
        if (!ids && (long long)mr * tc > s.cand_pairs) bail = true;
        __syncthreads();
      };
      auto col_rank = [&](int32_t e) {  // CTA whose list holds candidate column e
        int32_t r = 0;
        while (e >= sh.pre[r + 1]) r++;
        return r;
      };
      if (need_n) {
        collect((KeyT)0, false);
        if (!bail) {
          KeyT* sb = reinterpret_cast<KeyT*>(smem + L.map);
          int32_t* sj = reinterpret_cast<int32_t*>(sb + kCandStage);
          int32_t* sv = sj + kCandStage;  // vertex, bit 31: tabu
          const int32_t tc = sh.pre[nb], lr = sh.nrow;
          for (int32_t e0 = 0; e0 < tc; e0 += kCandStage) {
            const int32_t ec = min(kCandStage, tc - e0);
            for (int32_t e = tid; e < ec; e += T) {
              const int32_t r = col_rank(e0 + e);
              const int32_t j = cl.map_shared_rank(cll, r)[e0 + e - sh.pre[r]];
              sb[e] = cl.map_shared_rank(vb, r)[j];
              sj[e] = r * cpc + j;
              const bool tabu = cl.map_shared_rank(tb, r)[j] > now;
              sv[e] = cl.map_shared_rank(ub, r)[j] | (tabu ? INT_MIN : 0);
            }
            __syncthreads();
            for (int32_t p = tid; p < lr * ec; p += T) {
              const int32_t i = rl[p / ec], e = p % ec;
              const KeyT a = va[i], A = PROB == P_MDP ? -a : a, b = sb[e];
              const bool tabu = sv[e] < 0 || ta[i] > now;
              if (A + b < (tabu ? LT : LB)) continue;
              const int32_t u = ua[i], v = sv[e] & INT_MAX, j = sj[e];
              const int32_t w = cand_pair_w<ST, KeyT>(g, s, row0 + i, j, u, v);
              CandBest<KeyT> y;
              y.key = pair_gain<PROB, KeyT>(a, b, w);
              if (tabu && !(y.key > D)) continue;
              y.a = a; y.b = b; y.i = row0 + i; y.j = j; y.u = u; y.v = v;
              cand_better(mine, y);
            }
            __syncthreads();
          }
          if (edges)  // the staging area is the bitmap of E
            for (uint32_t q = tid; q < L.map_bytes / 16; q += T) reinterpret_cast<uint4*>(map)[q] = make_uint4(0, 0, 0, 0);
          if (need_e) {
            cl.sync();  // the lists are rewritten
            if (tid == 0) { sh.nrow = 0; sh.ncol = 0; }
            __syncthreads();
          }
        }
      }
      if (need_e && !bail) {
        collect(plus, true);
        if (!bail) {
          const int32_t tc = sh.pre[nb], lr = sh.nrow;
          for (int32_t e = tid; e < tc; e += T) {
            const int32_t r = col_rank(e);
            const int32_t v = cl.map_shared_rank(cll, r)[e - sh.pre[r]];
            atomicOr(&map[v >> 5], 1u << (v & 31));
          }
          __syncthreads();
          auto entry = [&](int32_t i, int32_t u, KeyT a, bool row_tabu, long long rs, long long k, const int2 e) {
            if (!((map[e.x >> 5] >> (e.x & 31)) & 1u)) return;
            if (k > rs && __ldg(&g.adj[k - 1].x) == e.x) return;  // duplicated pair: first entry
            const int32_t j = __ldcg(s.pos + e.x) - m;
            if (j < 0) return;
            const int32_t o = j / cpc, jl = j - o * cpc;
            CandBest<KeyT> y;
            y.b = cl.map_shared_rank(vb, o)[jl];
            const bool tabu = row_tabu || cl.map_shared_rank(tb, o)[jl] > now;
            y.key = pair_gain<PROB, KeyT>(a, y.b, e.y);
            if (y.key < LB || (tabu && !(y.key > D))) return;
            y.a = a; y.i = row0 + i; y.j = j; y.u = u; y.v = e.x;
            cand_better(mine, y);
          };
          for (int32_t r = warp; r < lr; r += nw) {
            const int32_t i = rl[r], u = ua[i];
            const long long rs = __ldg(g.rowptr + u);
            const int32_t len = (int32_t)(__ldg(g.rowptr + u + 1) - rs);
            if (len > kCandHeavy) {
              int32_t at = 0;
              if (lane == 0) at = atomicAdd(&sh.nheavy, 1);
              at = __shfl_sync(0xffffffffu, at, 0);
              if (at < kCandHeavyList) {
                if (lane == 0) sh.heavy[at] = i;
                continue;
              }
            }
            const KeyT a = va[i];
            const bool rt = ta[i] > now;
            for (int32_t base = 0; base < len; base += 128) {
              int2 e[4];
#pragma unroll
              for (int q = 0; q < 4; q++) {
                const int32_t k = base + q * 32 + lane;
                e[q] = k < len ? __ldg(g.adj + rs + k) : make_int2(-1, 0);
              }
#pragma unroll
              for (int q = 0; q < 4; q++)
                if (e[q].x >= 0) entry(i, u, a, rt, rs, rs + base + q * 32 + lane, e[q]);
            }
          }
          __syncthreads();
          const int32_t nh = min(sh.nheavy, kCandHeavyList);
          for (int32_t h = 0; h < nh; h++) {
            const int32_t i = sh.heavy[h], u = ua[i];
            const long long rs = __ldg(g.rowptr + u);
            const int32_t len = (int32_t)(__ldg(g.rowptr + u + 1) - rs);
            const KeyT a = va[i];
            const bool rt = ta[i] > now;
            for (int32_t k = tid; k < len; k += T) entry(i, u, a, rt, rs, rs + k, __ldg(g.adj + rs + k));
          }
        }
      }
      if (bail) { status = kCandBail; break; }
      // ---- block, then cluster best
      warp_best<KeyT>(mine);
      if (lane == 0) sh.wbest[warp] = mine;
      __syncthreads();
      if (warp == 0) {
        CandBest<KeyT> b;
        b.j = -1;
        if (lane < nw) b = sh.wbest[lane];
        warp_best<KeyT>(b);
        if (lane < nb) *cl.map_shared_rank(&sh.rec[rank], lane) = b;
      }
      if (need_e)
        for (uint32_t q = tid; q < L.map_bytes / 16; q += T) reinterpret_cast<uint4*>(map)[q] = make_uint4(0, 0, 0, 0);
      cl.sync();
      CandBest<KeyT> b;
      b.j = -1;
      if (lane < nb) b = sh.rec[lane];
      warp_best<KeyT>(b);
      cand_better(best, b);
    }

    // ---- 4. decision and move (decide_apply's rules)
    if (best.j < 0 || (PROB == P_MDP && (long long)best.key <= kMdpSentinel)) {
      __syncthreads();
      if (tid == 0) sh.sc.mode = 1;  // no allowed pair above the sentinel: the exact pass decides
      __syncthreads();
      status = kCandBail;
      break;
    }
    int32_t t_u, t_v, t2 = 0;
    if (PROB == P_MDP) {
      const int32_t c = s.tenure_policy == 0 ? mdp_ref_tenure(iter) : s.tenure;
      t_u = c;
      t_v = t2 = s.tenure_policy == 0 ? s.c2_tab[c == 15 ? 0 : c == 30 ? 1 : c == 60 ? 2 : 3] : s.c2_fixed;
    } else {
      t_u = t_v = s.tenure_policy == 0 ? maxbs_ref_tenure(iter, s.maxt) : s.tenure;
    }
    const int32_t iu = best.i, jv = best.j;
    budget--;
    __syncthreads();  // every thread has read this iteration's scalars
    if (tid == 0) {
      CandScalars& c = sh.sc;
      const long long key = (long long)best.key;
      log_move(iu, jv);
      c.cur += (PROB == P_MAXBS && key < kMaxbsRecoverBelow) ? key + kMaxbsInf : key;
      c.evaluations += s.P;
      if (c.cur > c.best) {
        c.best = c.cur;
        c.best_log_n = c.log_n;
        c.isi = 0;
      } else {
        c.isi += 1;
      }
      trace_put(iter, (long long)iu * delta + jv, key, 0, t_u, t2);
      c.iter = iter + 1;
      c.perturb = PROB == P_MAXBS && c.isi >= s.piter;
    }
    apply(iu, jv, best.u, best.v, best.a, best.b, (int32_t)(iter + t_v), (int32_t)(iter + t_u));
    if (PROB == P_MAXBS && sh.sc.perturb) {
      const long long ev = sh.sc.pert_events - pert_base;
      const bool in_window = ev >= 0 && ev < s.draw_events && ev < pert_limit;
      bool bad = false;
      if (in_window) {
        for (int32_t q = 0; q < s.num_pert; q++) {
          const long long mv = __ldg(s.draws + ev * s.num_pert + q);
          if (mv < 0 || mv >= s.P) { bad = true; break; }
          const int32_t pu = (int32_t)(mv / delta), pv = (int32_t)(mv % delta);
          const int32_t oi = pu / rpc, oj = pv / cpc;
          const int32_t u = cl.map_shared_rank(ua, oi)[pu - oi * rpc], v = cl.map_shared_rank(ub, oj)[pv - oj * cpc];
          const KeyT a = cl.map_shared_rank(va, oi)[pu - oi * rpc], b = cl.map_shared_rank(vb, oj)[pv - oj * cpc];
          if (rank == 0 && tid == 0) sh.wuv = 0;
          cl.sync();  // slots read before anyone updates them
          apply(pu, pv, u, v, a, b, -1, -1);
          if (tid == 0) {
            CandScalars& c = sh.sc;
            // the slots now hold the negated contributions after the update
            const KeyT na = *slot_of(m + pv), nb2 = *slot_of(pu);
            const long long aux = -(long long)na - (long long)nb2 - 2LL * *cl.map_shared_rank(&sh.wuv, 0);
            log_move(pu, pv);
            c.cur += aux;
            c.pert_moves += 1;
            trace_put(iter + 1, mv, aux, 2, 0, 0);
          }
          cl.sync();
        }
      }
      __syncthreads();
      if (tid == 0) {
        CandScalars& c = sh.sc;
        c.perturb = 0;
        if (!in_window) {
          c.err |= E_PERTURB_WINDOW;
          c.done = 1;
        } else {
          if (bad) { c.err |= E_BAD_INDEX; c.done = 1; }
          c.pert_events += 1;
          c.isi = 0;
        }
      }
      __syncthreads();
    }
  }

  for (int32_t i = tid; i < nr; i += T) {
    s.vg_in[row0 + i] = va[i];
    s.tab_in[row0 + i] = ta[i];
    s.sol_in[row0 + i] = ua[i];
  }
  for (int32_t j = tid; j < nc; j += T) {
    s.vg_out[col0 + j] = vb[j];
    s.tab_out[col0 + j] = tb[j];
    s.sol_out[col0 + j] = ub[j];
  }
  if (rank == 0 && tid == 0) {
    DevState* st = s.st;
    const CandScalars& c = sh.sc;
    st->iter = c.iter; st->cur = c.cur; st->best = c.best; st->evaluations = c.evaluations; st->isi = c.isi;
    st->log_n = c.log_n; st->best_log_n = c.best_log_n; st->trace_n = c.trace_n;
    st->pert_events = c.pert_events; st->pert_moves = c.pert_moves;
    st->done = c.done; st->stopped = c.stopped; st->err |= c.err; st->mode = c.mode;
    st->owed = status == kCandBail ? (int32_t)min(budget, (long long)INT32_MAX) : 0;
  }
  cl.sync();  // no CTA leaves (or reuses its shared memory) while another may still read it
  return status;
}

}  // namespace tsb
