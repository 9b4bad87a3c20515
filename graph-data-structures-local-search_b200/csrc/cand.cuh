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
// it is latency, not bytes: an iteration is one walk by a few warps through
// two to five barriers and about four dependent L2 round trips, at any size.
// Per iteration, sweeps before and this pass now: MDP ER n = 2,000 (CSR) 17.0
// -> 2.5 us; dense n = 2,000 (CSR+BB) 42.7 -> 7.8; Chung-Lu n = 200,000 (Hash)
// 811 -> 5.2; bisection conflict graph n = 100,000 (CSR) 153 -> 14.0, n =
// 60,001 (WSwap) 390 -> 11.8, n = 30,011 (CSR+Bitset) 179 -> 11.0; n = 10,007
// with 64-bit contributions (CSR+BB) 115 -> 11.5.  (The pass's first form took
// 3.9, 13.7, 5.9, 14.4, 11.9, 11.1 and 14.9 us: warp reduction instructions in
// every warp, all rows within the whole slack enumerated.)
#pragma once
#include <cooperative_groups.h>

#include "sweep.cuh"

namespace tsb {

constexpr int kCandTPB = 512;        // most threads per CTA
constexpr int kCandMaxCluster = 16;
constexpr int kCandList = 2048;      // entries of a CTA's candidate lists, at least (or its whole slice)
constexpr int kCandStage = 1024;     // candidate columns staged per round of N
constexpr int kCandHeavy = 512;      // E: rows of more entries are walked by the whole CTA
constexpr int kCandHeavyList = 64;
constexpr int kCandHits = 2048;      // E: entries kept for evaluation per round (more: a sweep)
constexpr int kCandRowBits = 22;     // E: a kept entry's place in its row, beside 9 bits for the row
constexpr int kCandGroupPairs = 12;  // N: up to this many pairs a warp, eight lanes look each one up

enum { kCandEnd = 0, kCandBail = 1 };
enum { kPairNone = -1, kPairOverflow = -2 };  // CandBest::j without a pair

struct CandLayout {
  uint32_t va, vb, ta, tb, ua, ub, pv, rl, cl, map, hits, stage, total;
  uint32_t map_bytes;
  int32_t rcap, ccap;  // list lengths
  int32_t vpc;         // vertices per CTA of the position slice (0: positions stay in HBM)
};
// Shared memory of one CTA: rpc rows and cpc columns (multiples of 4), a slice
// of the positions by vertex (vpc > 0), lists, for E the candidates' bitmap
// and a queue, and one area for the staged columns (N) or rows (E).
__host__ __device__ inline CandLayout cand_layout(int32_t n, int32_t rpc, int32_t cpc, int kb, int32_t vpc, bool edges,
                                                      int32_t list) {
  CandLayout L;
  uint32_t off = 0;
  L.va = off; off += (uint32_t)kb * rpc;
  L.vb = off; off += (uint32_t)kb * cpc;
  L.ta = off; off += 4u * rpc;
  L.tb = off; off += 4u * cpc;
  L.ua = off; off += 4u * rpc;
  L.ub = off; off += 4u * cpc;
  L.vpc = vpc;
  L.pv = off; off += 4u * (uint32_t)vpc;
  L.rcap = L.ccap = list;
  L.rl = off; off += 4u * (uint32_t)L.rcap;
  L.cl = off; off += 4u * (uint32_t)L.ccap;
  L.map_bytes = edges ? 16u * (uint32_t)((n + 127) / 128) : 0u;
  L.map = off; off += L.map_bytes;
  L.hits = off; off += edges ? 4u * kCandHits : 0u;
  L.stage = off; off += (uint32_t)(8 + kb) * kCandStage;
  L.total = off;
  return L;
}

// A value and the lowest position that has it (none: below every other).
// 32-bit values compare as one word with the complemented position.
template <class KeyT>
struct CandMax {
  long long k;
  int32_t p;
  __device__ static CandMax none() { return CandMax{LLONG_MIN, INT_MAX}; }
  __device__ static CandMax of(KeyT k, int32_t i) { return CandMax{k, i}; }
  __device__ KeyT key() const { return k; }
  __device__ int32_t pos() const { return p == INT_MAX ? -1 : p; }
  __device__ bool below(const CandMax& b) const { return b.k > k || (b.k == k && b.p < p); }
  __device__ CandMax from(int mask) const {
    return CandMax{__shfl_xor_sync(0xffffffffu, k, mask), __shfl_xor_sync(0xffffffffu, p, mask)};
  }
  __device__ CandMax lane(int l) const { return CandMax{__shfl_sync(0xffffffffu, k, l), __shfl_sync(0xffffffffu, p, l)}; }
};
template <>
struct CandMax<int32_t> {
  unsigned long long w;
  __device__ static CandMax none() { return CandMax{0ull}; }
  __device__ static CandMax of(int32_t k, int32_t i) {
    return CandMax{((unsigned long long)((uint32_t)k ^ 0x80000000u) << 32) | (uint32_t)~i};
  }
  __device__ int32_t key() const { return (int32_t)((uint32_t)(w >> 32) ^ 0x80000000u); }
  __device__ int32_t pos() const { return w ? (int32_t)~(uint32_t)w : -1; }
  __device__ bool below(const CandMax& b) const { return b.w > w; }
  __device__ CandMax from(int mask) const { return CandMax{__shfl_xor_sync(0xffffffffu, w, mask)}; }
  __device__ CandMax lane(int l) const { return CandMax{__shfl_sync(0xffffffffu, w, l)}; }
};
template <class KeyT>
struct alignas(16) CandTop {  // a CTA's maxima: row non-tabu, row all, column non-tabu, column all
  CandMax<KeyT> m[4];
  int32_t v[4];
};
template <class KeyT>
struct alignas(16) CandBest {  // a pair
  KeyT key, a, b;              // gain; raw contributions of the pair
  int32_t i, j, u, v;          // j < 0: no pair
};
struct CandScalars {
  long long iter, cur, best, evaluations, isi, log_n, best_log_n, trace_n, pert_events, pert_moves;
  int32_t done, stopped, err, mode, perturb, pad;
};
// What warp 0 works out after the maxima are known.
template <class KeyT>
struct CandGoal {
  CandBest<KeyT> best;           // better seed (j < 0: none)
  KeyT Am, AA, Bm, BA, LB, LT;   // maxima; thresholds of non-tabu pairs and of pairs with a tabu side
  KeyT s_nt, s_all;              // E: LB - Am - Bm, LT - AA - BA
  int32_t nt_ok, need_n, need_e;
  int32_t len_u, len_v;          // CSR rows of the best seed's vertices
  long long row_u, row_v;
};
template <class KeyT>
struct CandShared {
  CandTop<KeyT> top[kCandMaxCluster];
  CandBest<KeyT> rec[kCandMaxCluster];
  CandBest<KeyT> wbest[kCandTPB / 32];
  CandGoal<KeyT> goal;
  CandMax<KeyT> wmax[4][kCandTPB / 32];
  int32_t nrow, ncol, nheavy, nhits, wuv;
  int32_t pre[kCandMaxCluster + 1];
  int32_t heavy[kCandHeavyList];
  CandScalars sc;
};

__device__ __forceinline__ int32_t lane_min(int32_t v) { return __reduce_min_sync(0xffffffffu, v); }

template <class KeyT>
__device__ __forceinline__ CandMax<KeyT> max_of(const CandMax<KeyT>& a, const CandMax<KeyT>& b) {
  return a.below(b) ? b : a;
}
// The four maxima of a warp at once: after two exchanges each lane works for
// one of them (lane / 8), so six exchanges do instead of twenty.  (Warp
// reduction instructions are slow here: eight of them in each of 16 warps took
// 2,000 of the iteration's cycles.)
template <class KeyT>
__device__ __forceinline__ CandMax<KeyT> warp_max4(const CandMax<KeyT> (&q)[4]) {
  const int lane = threadIdx.x & 31;
  const bool h = lane & 16, l = lane & 8;
  const CandMax<KeyT> a = max_of(h ? q[2] : q[0], (h ? q[0] : q[2]).from(16));
  const CandMax<KeyT> b = max_of(h ? q[3] : q[1], (h ? q[1] : q[3]).from(16));
  CandMax<KeyT> r = max_of(l ? b : a, (l ? a : b).from(8));
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) r = max_of(r, r.from(o));
  return r;
}
template <class KeyT>
__device__ __forceinline__ CandMax<KeyT> octet_max(CandMax<KeyT> r) {  // over the eight lanes of a maximum
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) r = max_of(r, r.from(o));
  return r;
}

// Candidate (i, j) precedes the held best: larger key, then lower flat index.
template <class KeyT>
__device__ __forceinline__ void cand_better(CandBest<KeyT>& x, const CandBest<KeyT>& y) {
  if (y.j < 0) return;
  if (x.j < 0 || y.key > x.key || (y.key == x.key && (y.i < x.i || (y.i == x.i && y.j < x.j)))) x = y;
}

// Best pair of a warp in every lane.  Few lanes hold one, mostly none.
template <class KeyT>
__device__ __forceinline__ void warp_best(CandBest<KeyT>& b) {
  unsigned who = __ballot_sync(0xffffffffu, b.j >= 0);
  if (!who) { b.j = kPairNone; return; }
  if (who & (who - 1)) {
    const KeyT m = warp_max(b.j >= 0 ? b.key : KeyLim<KeyT>::none);
    const bool has = b.j >= 0 && b.key == m;
    const int32_t i = lane_min(has ? b.i : INT_MAX);
    const int32_t j = lane_min(has && b.i == i ? b.j : INT_MAX);
    who = __ballot_sync(0xffffffffu, has && b.i == i && b.j == j);
  }
  const int src = __ffs(who) - 1;
  b.key = __shfl_sync(0xffffffffu, b.key, src);
  b.a = __shfl_sync(0xffffffffu, b.a, src);
  b.b = __shfl_sync(0xffffffffu, b.b, src);
  b.i = __shfl_sync(0xffffffffu, b.i, src);
  b.j = __shfl_sync(0xffffffffu, b.j, src);
  b.u = __shfl_sync(0xffffffffu, b.u, src);
  b.v = __shfl_sync(0xffffffffu, b.v, src);
}

// First entry of v in a sorted CSR row by the whole warp: 32 probes a step.
__device__ __forceinline__ int32_t warp_row_lookup(const int2* row, int32_t len, int32_t v) {
  const int lane = threadIdx.x & 31;
  int32_t lo = 0;
#pragma unroll 1
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

// w(i, j) of a pair, by a whole warp, in the solver's structure.  A CSR row is
// searched from the end of smaller degree (both rows hold the entry,
// duplicates in the same order); the bitmaps answer first where there are any.
// ru, du, rv, dv: the vertices' CSR rows (start, length).
template <int ST, class KeyT>
__device__ __forceinline__ int32_t cand_warp_w(const DevGraph& g, const DevSolver<KeyT>& s, int32_t i, int32_t j,
                                               int32_t u, int32_t v, long long ru, int32_t du, long long rv, int32_t dv) {
  if (ST == S_WSWAP) return w_get<true>(s, (long long)i * s.ldc + j);
  if (ST == S_HASH) {
    const long long b = __ldg(g.hoff + u);
    const long long cap = __ldg(g.hoff + u + 1) - b;
    return hash_probe(g.hkey + b, g.hval + b, (uint32_t)(cap / 4 - 1), hash_gshift(cap), v);
  }
  if (ST == S_BITSET || ST == S_BITSET_BB) {
    if (!bit_test(g.bits + (long long)u * g.wpr, v)) return 0;
  }
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

// A pair per eight lanes of the warp (all lanes call it; `on`: the octet has a
// pair).  CSR rows only: Hash and WSwap are answered by a thread.
template <int ST, class KeyT>
__device__ __forceinline__ int32_t cand_octet_w(const DevGraph& g, const DevSolver<KeyT>& s, int32_t i, int32_t j,
                                                int32_t u, int32_t v, bool on) {
  const int lane = threadIdx.x & 31, t = lane & 7, o = lane & 24;
  long long row = 0;
  int32_t len = 0, key = v;
  if (on && (ST == S_BITSET || ST == S_BITSET_BB)) on = bit_test(g.bits + (long long)u * g.wpr, v);
  if (on) {
    const long long ru = __ldg(g.rowptr + u), rv = __ldg(g.rowptr + v);
    const int32_t du = (int32_t)(__ldg(g.rowptr + u + 1) - ru), dv = (int32_t)(__ldg(g.rowptr + v + 1) - rv);
    row = du <= dv ? ru : rv;
    len = du <= dv ? du : dv;
    key = du <= dv ? v : u;
  }
#pragma unroll 1
  while (__any_sync(0xffffffffu, len > 8)) {  // (shorter octets repeat a harmless step)
    const int32_t step = (len + 7) >> 3;
    const int32_t at = (t + 1) * step - 1;
    const bool below = len > 8 && at < len && __ldg(&g.adj[row + at].x) < key;
    const unsigned b = __ballot_sync(0xffffffffu, below);
    if (len > 8) {
      const int32_t skip = __popc(b >> o & 0xffu) * step;
      row += skip;
      len = min(step, len - skip);
    }
  }
  int2 e = make_int2(-1, 0);
  if (t < len) e = __ldg(g.adj + row + t);
  const unsigned hit = __ballot_sync(0xffffffffu, e.x == key) >> o & 0xffu;
  const int32_t w = __shfl_sync(0xffffffffu, e.y, hit ? o + __ffs(hit) - 1 : lane);
  return hit ? w : 0;
}

// One thread's maxima over a slice, non-tabu and all: the value and the first
// entry of the quad that has it (its quads ascend, so a strict comparison
// keeps the first; the entry is picked later, by the winner alone).
template <bool NEG, class KeyT>
__device__ __forceinline__ void cand_scan(const KeyT* val, const int32_t* tab, int32_t cnt, int32_t i0, int32_t now,
                                          CandMax<KeyT>& nt, CandMax<KeyT>& all) {
  constexpr KeyT none = KeyLim<KeyT>::none;
  KeyT kn = none, ka = none;
  int32_t in = 0, ia = 0;
#pragma unroll 1
  for (int32_t q = (int32_t)threadIdx.x * 4; q < cnt; q += (int32_t)blockDim.x * 4) {
    KeyT x[4], y[4];
    const int4 t = *reinterpret_cast<const int4*>(tab + q);
    if constexpr (sizeof(KeyT) == 4) {
      const int4 v4 = *reinterpret_cast<const int4*>(val + q);
      x[0] = v4.x; x[1] = v4.y; x[2] = v4.z; x[3] = v4.w;
    } else {
      const longlong2 a = *reinterpret_cast<const longlong2*>(val + q), b = *reinterpret_cast<const longlong2*>(val + q + 2);
      x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (NEG) x[k] = -x[k];
      if (k > 0 && q + k >= cnt) x[k] = none;
    }
    y[0] = t.x <= now ? x[0] : none;
    y[1] = t.y <= now ? x[1] : none;
    y[2] = t.z <= now ? x[2] : none;
    y[3] = t.w <= now ? x[3] : none;
    const KeyT ma = max(max(x[0], x[1]), max(x[2], x[3])), mn = max(max(y[0], y[1]), max(y[2], y[3]));
    if (ma > ka) { ka = ma; ia = q; }
    if (mn > kn) { kn = mn; in = q; }
  }
  all = ka == none ? CandMax<KeyT>::none() : CandMax<KeyT>::of(ka, i0 + ia);
  nt = kn == none ? CandMax<KeyT>::none() : CandMax<KeyT>::of(kn, i0 + in);
}

// Shared memory of the cluster, by 32-bit shared::cluster addresses.
__device__ __forceinline__ uint32_t cta_smem(uint32_t own, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(own), "r"(rank));
  return r;
}
__device__ __forceinline__ int32_t ld_cta32(uint32_t a) {
  int32_t v;
  asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void ld_cta(uint32_t a, int32_t& v) { v = ld_cta32(a); }
__device__ __forceinline__ void ld_cta(uint32_t a, long long& v) {
  asm volatile("ld.shared::cluster.s64 %0, [%1];" : "=l"(v) : "r"(a));
}
__device__ __forceinline__ void st_cta32(uint32_t a, int32_t v) {
  asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void add_cta(uint32_t a, int32_t v) {
  asm volatile("red.relaxed.cluster.shared::cluster.add.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void add_cta(uint32_t a, long long v) {
  asm volatile("red.relaxed.cluster.shared::cluster.add.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}
// x / d for x < 2^19 and the d of cand_slices, from ceil(2^32 / d)
__device__ __forceinline__ int32_t div_by(int32_t x, uint32_t inv) { return (int32_t)__umulhi((uint32_t)x, inv); }

// Runs iterations up to `stop_at`, at most `budget` of them, by the calling
// cluster (every CTA, all threads).  State is read from the solver's arrays at
// entry and written back at exit.  Returns kCandEnd, or kCandBail when the
// next iteration needs a sweep (too many candidates, or the exact pass).
//
// An iteration is one walk through this code by a few warps, so its length
// counts: every step has one call site, and loops that run once or twice stay
// rolled.  (At 220-320 KB a kernel, with inlined copies, the walk missed the
// instruction cache and every step took 1.3 to 2 times as long.)
template <int PROB, int ST, class KeyT>
__device__ int cand_run(const DevGraph& g, const DevSolver<KeyT>& s, long long stop_at, long long budget,
                        cooperative_groups::cluster_group& cl, CandShared<KeyT>& sh, unsigned char* smem) {
  constexpr KeyT kNoKey = KeyLim<KeyT>::none;
  constexpr int kKb = (int)sizeof(KeyT);
  const int T = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = T >> 5;
  const int nb = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int32_t m = s.m, delta = s.delta, rpc = s.cand_rpc, cpc = s.cand_cpc;
  const CandLayout L = cand_layout(s.n, rpc, cpc, kKb, s.cand_vpc, s.cand_plus > 0, s.cand_list);
  // one array each: the slice's rows, then (from rpc) its columns
  KeyT* val = reinterpret_cast<KeyT*>(smem + L.va);
  int32_t* stamp = reinterpret_cast<int32_t*>(smem + L.ta);
  int32_t* ids = reinterpret_cast<int32_t*>(smem + L.ua);
  int32_t* pv = reinterpret_cast<int32_t*>(smem + L.pv);
  int32_t* rl = reinterpret_cast<int32_t*>(smem + L.rl);
  int32_t* cll = reinterpret_cast<int32_t*>(smem + L.cl);
  uint32_t* map = reinterpret_cast<uint32_t*>(smem + L.map);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t inv_r = s.cand_inv[0], inv_c = s.cand_inv[1], inv_v = s.cand_inv[2];
  const int32_t row0 = rank * rpc, col0 = rank * cpc;
  const int32_t nr = max(0, min(rpc, m - row0)), nc = max(0, min(cpc, delta - col0));
  const KeyT plus = (KeyT)s.cand_plus;
  const bool fav = s.cand_fav != 0;

  auto barrier = [&]() {  // of the cluster; one CTA needs no cluster barrier
    if (nb == 1) __syncthreads();
    else cl.sync();
  };
  // Position p: its index in its owner's arrays, and the owner's shared memory.
  auto place = [&](int32_t p, uint32_t& base) -> int32_t {
    const bool in = p < m;
    const int32_t q = in ? p : p - m, o = div_by(q, in ? inv_r : inv_c);
    base = cta_smem(sbase, o);
    return q - o * (in ? rpc : cpc) + (in ? 0 : rpc);
  };
  auto pos_of = [&](int32_t z) -> int32_t {
    if (!L.vpc) return __ldcg(s.pos + z);
    const int32_t o = div_by(z, inv_v);
    return ld_cta32(cta_smem(sbase, o) + L.pv + 4u * (uint32_t)(z - o * L.vpc));
  };
  auto row_of = [&](int32_t u, long long& at) -> int32_t {  // CSR row: start and length
    at = __ldg(g.rowptr + u);
    return (int32_t)(__ldg(g.rowptr + u + 1) - at);
  };

#pragma unroll 1
  for (int32_t x = tid; x < rpc + cpc; x += T) {
    const bool row = x < rpc;
    const int32_t i = row ? x : x - rpc;
    if (i >= (row ? nr : nc)) continue;
    val[x] = __ldcg((row ? s.vg_in + row0 : s.vg_out + col0) + i);
    stamp[x] = __ldcg((row ? s.tab_in + row0 : s.tab_out + col0) + i);
    ids[x] = __ldcg((row ? s.sol_in + row0 : s.sol_out + col0) + i);
  }
#pragma unroll 1
  for (uint32_t q = tid; q < L.map_bytes / 16; q += T) reinterpret_cast<uint4*>(map)[q] = make_uint4(0, 0, 0, 0);
  const int32_t v0 = rank * L.vpc, nv = max(0, min(L.vpc, s.n - v0));
#pragma unroll 1
  for (int32_t v = tid; v < nv; v += T) pv[v] = __ldcg(s.pos + v0 + v);
  if (tid == 0) {
    const DevState* st = s.st;
    CandScalars& c = sh.sc;
    c.iter = __ldcg(&st->iter); c.cur = __ldcg(&st->cur); c.best = __ldcg(&st->best);
    c.evaluations = __ldcg(&st->evaluations); c.isi = __ldcg(&st->isi);
    c.log_n = __ldcg(&st->log_n); c.best_log_n = __ldcg(&st->best_log_n); c.trace_n = __ldcg(&st->trace_n);
    c.pert_events = __ldcg(&st->pert_events); c.pert_moves = __ldcg(&st->pert_moves);
    c.done = __ldcg(&st->done); c.stopped = __ldcg(&st->stopped); c.err = __ldcg(&st->err);
    c.mode = __ldcg(&st->mode);
  }
  const long long pert_base = __ldcg(&s.st->pert_base), pert_limit = __ldcg(&s.st->pert_limit);
  cl.sync();

  int status = kCandEnd;
  for (;;) {
    const long long iter = sh.sc.iter;
    if (sh.sc.done || iter >= stop_at || budget <= 0) break;
    if (sh.sc.mode != 0) { status = kCandBail; break; }
    const int32_t now = (int32_t)min(iter, (long long)INT32_MAX);  // stamps are 32-bit
    long long D64 = sh.sc.best - sh.sc.cur;
    if (kKb == 4) {  // 32-bit gains stay within 2^30: the same comparisons, room for D + 1 and differences
      constexpr long long lim = 1LL << 30;
      D64 = D64 > lim ? lim : (D64 < -lim - 1 ? -lim - 1 : D64);
    }
    const KeyT D = (KeyT)D64;

    // ---- 1. maxima: slice, then cluster
    CandMax<KeyT> q4[4];
    cand_scan<PROB == P_MDP, KeyT>(val, stamp, nr, row0, now, q4[0], q4[1]);
    cand_scan<false, KeyT>(val + rpc, stamp + rpc, nc, col0, now, q4[2], q4[3]);
    {
      const CandMax<KeyT> r = warp_max4(q4);
      if ((lane & 7) == 0) sh.wmax[lane >> 3][warp] = r;
    }
    if (tid == 0) { sh.nrow = 0; sh.ncol = 0; sh.nheavy = 0; sh.nhits = 0; }
    __syncthreads();
    const int q = lane >> 3, t8 = lane & 7;  // warp 0: eight lanes for each maximum
    CandMax<KeyT> top = CandMax<KeyT>::none();
    int32_t topv = -1;
    if (warp == 0) {
      if (t8 < nw) top = sh.wmax[q][t8];
      if (t8 + 8 < nw) top = max_of(top, sh.wmax[q][t8 + 8]);
      top = octet_max(top);
      if (top.pos() >= 0) {  // the entry of the quad
        const KeyT k = top.key();
        const int32_t x = q < 2 ? top.pos() - row0 : top.pos() - col0 + rpc;
        const KeyT raw = PROB == P_MDP && q < 2 ? -k : k;
        const bool any = q & 1;
        int32_t e = 3;  // entries past the slice's end lie behind a match
        if (val[x + 2] == raw && (any || stamp[x + 2] <= now)) e = 2;
        if (val[x + 1] == raw && (any || stamp[x + 1] <= now)) e = 1;
        if (val[x] == raw && (any || stamp[x] <= now)) e = 0;
        topv = ids[x + e];
        top = CandMax<KeyT>::of(k, top.pos() + e);
      }
      if (nb > 1)
#pragma unroll 1
        for (int o = t8; o < nb; o += 8) {
          CandTop<KeyT>* d = cl.map_shared_rank(&sh.top[rank], o);
          d->m[q] = top;
          d->v[q] = topv;
        }
    }
    if (nb > 1) cl.sync();
    if (warp == 0) {
      if (nb > 1) {
        top = CandMax<KeyT>::none();
        topv = -1;
        for (int o = t8; o < nb; o += 8) {
          const CandMax<KeyT> x = sh.top[o].m[q];
          if (top.below(x)) { top = x; topv = sh.top[o].v[q]; }
        }
        const int32_t own = top.pos();
        top = octet_max(top);
        const unsigned mine = __ballot_sync(0xffffffffu, own >= 0 && own == top.pos());
        const unsigned oct = (mine >> (q * 8)) & 0xffu;
        topv = __shfl_sync(0xffffffffu, topv, oct ? q * 8 + __ffs(oct) - 1 : lane);
      }
      KeyT gk[4];
      int32_t gi[4], gv[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const CandMax<KeyT> x = top.lane(k * 8);
        gk[k] = x.key();
        gi[k] = x.pos();
        gv[k] = __shfl_sync(0xffffffffu, topv, k * 8);
      }
      // the four vertices' CSR rows: two words each, one round trip
      long long rp = 0;
      {
        const int32_t x = __shfl_sync(0xffffffffu, topv, (lane >> 1 & 3) * 8);
        if (lane < 8 && x >= 0) rp = __ldg(g.rowptr + x + (lane & 1));
      }
      const KeyT Am = gk[0], AA = gk[1], Bm = gk[2], BA = gk[3];
      const bool nt_ok = gi[0] >= 0 && gi[2] >= 0;

      // ---- 2. seeds and thresholds
      CandGoal<KeyT> G;
      G.best.j = kPairNone;
      KeyT c2w[2] = {0, 0};  // c*w of the non-tabu and of the overall seed pair
      const bool one_seed = nt_ok && gi[0] == gi[1] && gi[2] == gi[3];
      const bool asp = AA + BA + plus > D;  // some tabu pair might be aspirated
      if (!fav) {
#pragma unroll 1
        for (int k = nt_ok ? 0 : 1; k < (one_seed || !asp ? 1 : 2); k++) {
          const long long ru = __shfl_sync(0xffffffffu, rp, 2 * k), ru1 = __shfl_sync(0xffffffffu, rp, 2 * k + 1);
          const long long rv = __shfl_sync(0xffffffffu, rp, 2 * k + 4), rv1 = __shfl_sync(0xffffffffu, rp, 2 * k + 5);
          const int32_t w = cand_warp_w<ST, KeyT>(g, s, k ? gi[1] : gi[0], k ? gi[3] : gi[2], k ? gv[1] : gv[0],
                                                  k ? gv[3] : gv[2], ru, (int32_t)(ru1 - ru), rv, (int32_t)(rv1 - rv));
          const KeyT c = PROB == P_MDP ? -(KeyT)w : (KeyT)2 * (KeyT)w;
          if (k) c2w[1] = c;
          else c2w[0] = c;
        }
        if (one_seed) c2w[1] = c2w[0];
      }
      const KeyT c1 = c2w[0], c2 = c2w[1];
      KeyT LB = kNoKey;
      int from = 0;  // which seed is the better one
      if (nt_ok) {
        G.best.key = LB = Am + Bm + c1;
        G.best.i = gi[0]; G.best.j = gi[2]; G.best.u = gv[0]; G.best.v = gv[2];
        G.best.a = PROB == P_MDP ? -Am : Am;
        G.best.b = Bm;
      }
      if (!one_seed && AA + BA + c2 > D) {
        CandBest<KeyT> y;
        y.key = AA + BA + c2;
        y.i = gi[1]; y.j = gi[3]; y.u = gv[1]; y.v = gv[3];
        y.a = PROB == P_MDP ? -AA : AA;
        y.b = BA;
        if (y.key > LB) LB = y.key;
        cand_better(G.best, y);
        from = G.best.i == y.i && G.best.j == y.j;
      }
      const KeyT LT = LB > D ? LB : D + 1;
      G.Am = Am; G.AA = AA; G.Bm = Bm; G.BA = BA; G.LB = LB; G.LT = LT;
      G.nt_ok = nt_ok;
      // N: non-adjacent pairs, and adjacent ones with c*w <= 0, bounded by A + B
      G.need_n = !fav && ((nt_ok && c1 < 0 && Am + Bm >= LB) || (c2 < 0 && asp && AA + BA >= LT));
      // E: adjacent pairs with c*w > 0, bounded by A + B + plus
      G.s_nt = nt_ok ? LB - Am - Bm : (KeyT)0;
      G.s_all = LT - AA - BA;
      G.need_e = plus > 0 && ((nt_ok && plus >= G.s_nt) || plus >= G.s_all);
      const long long ru1 = __shfl_sync(0xffffffffu, rp, 2 * from + 1), rv1 = __shfl_sync(0xffffffffu, rp, 2 * from + 5);
      G.row_u = __shfl_sync(0xffffffffu, rp, 2 * from);
      G.row_v = __shfl_sync(0xffffffffu, rp, 2 * from + 4);
      G.len_u = (int32_t)(ru1 - G.row_u);
      G.len_v = (int32_t)(rv1 - G.row_v);
      if (lane == 0) sh.goal = G;
    }
    __syncthreads();
    CandBest<KeyT> best = sh.goal.best;

    // ---- 3. candidates
    if (sh.goal.need_n || sh.goal.need_e) {
      const KeyT LB = sh.goal.LB, LT = sh.goal.LT;
      const KeyT Am = sh.goal.Am, AA = sh.goal.AA, Bm = sh.goal.Bm, BA = sh.goal.BA;
      const bool nt_ok = sh.goal.nt_ok != 0;
      CandBest<KeyT> mine;
      mine.j = kPairNone;
      bool bail = false;
      if (sh.goal.need_n) {
        // rows with A + Bm >= LB, columns with Am + B >= LB (tabu ones: LT)
#pragma unroll 1
        for (int32_t x = tid; x < rpc + cpc; x += T) {
          const bool row = x < rpc;
          if (row ? x >= nr : x - rpc >= nc) continue;
          const KeyT y = PROB == P_MDP && row ? -val[x] : val[x];
          if ((nt_ok && stamp[x] <= now && y + (row ? Bm : Am) >= LB) || y + (row ? BA : AA) >= LT) {
            const int32_t at = atomicAdd(row ? &sh.nrow : &sh.ncol, 1);
            if (at < L.rcap) (row ? rl : cll)[at] = x;
          }
        }
        barrier();
        // counts of the cluster: column prefix, largest lists
        const int32_t cr = lane < nb ? *cl.map_shared_rank(&sh.nrow, lane) : 0;
        const int32_t cc = lane < nb ? *cl.map_shared_rank(&sh.ncol, lane) : 0;
        int32_t incl = cc;
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) {
          const int32_t t = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += t;
        }
        if (warp == 0 && lane < nb) sh.pre[lane + 1] = incl;
        if (tid == 0) sh.pre[0] = 0;
        const int32_t mr = __reduce_max_sync(0xffffffffu, cr), mc = __reduce_max_sync(0xffffffffu, cc);
        const int32_t tc = __shfl_sync(0xffffffffu, incl, nb - 1);
        bail = mr > L.rcap || mc > L.ccap || (long long)mr * tc > s.cand_pairs;
        __syncthreads();
        if (!bail) {
          KeyT* sb = reinterpret_cast<KeyT*>(smem + L.stage);
          int32_t* sj = reinterpret_cast<int32_t*>(sb + kCandStage);
          int32_t* sv = sj + kCandStage;  // vertex, bit 31: tabu
          const int32_t lr = sh.nrow;
#pragma unroll 1
          for (int32_t e0 = 0; e0 < tc; e0 += kCandStage) {
            const int32_t ec = min(kCandStage, tc - e0);
#pragma unroll 1
            for (int32_t e = tid; e < ec; e += T) {
              int32_t r = 0;
              while (e0 + e >= sh.pre[r + 1]) r++;
              const uint32_t base = cta_smem(sbase, r);
              const int32_t x = ld_cta32(base + L.cl + 4u * (uint32_t)(e0 + e - sh.pre[r]));
              ld_cta(base + L.va + (uint32_t)(kKb * x), sb[e]);
              sj[e] = r * cpc + x - rpc;
              sv[e] = ld_cta32(base + L.ua + 4u * (uint32_t)x) |
                      (ld_cta32(base + L.ta + 4u * (uint32_t)x) > now ? INT_MIN : 0);
            }
            __syncthreads();
            const int32_t pairs = lr * ec;
            // Few pairs: eight lanes each, eight probes of the row per step
            // (a row of 2,000 entries: 4 loads one after another instead of
            // 11); many: a thread each.  Hash and WSwap answer a thread in one
            // or two loads.
            const int width = ST != S_HASH && ST != S_WSWAP && pairs <= kCandGroupPairs * nw ? 8 : 1;
#pragma unroll 1
            for (int32_t p0 = tid / width; p0 - lane / width < pairs; p0 += T / width) {
              const int32_t p = min(p0, pairs - 1);  // all lanes of a warp search together
              const int32_t i = rl[p / ec], e = p % ec;
              const KeyT a = val[i], A = PROB == P_MDP ? -a : a, b = sb[e];
              const bool tabu = sv[e] < 0 || stamp[i] > now;
              const bool reach = p0 < pairs && A + b >= (tabu ? LT : LB);
              CandBest<KeyT> y;
              y.a = a; y.b = b; y.i = row0 + i; y.j = sj[e]; y.u = ids[i]; y.v = sv[e] & INT_MAX;
              int32_t w = 0;
              if (width == 8) w = cand_octet_w<ST, KeyT>(g, s, y.i, y.j, y.u, y.v, reach);
              else if (reach) w = cand_pair_w<ST, KeyT>(g, s, y.i, y.j, y.u, y.v);
              y.key = pair_gain<PROB, KeyT>(a, b, w);
              if (reach && !(tabu && !(y.key > D)) && lane % width == 0) cand_better(mine, y);
            }
            __syncthreads();
          }
        }
        if (sh.goal.need_e && !bail) {
          barrier();  // the lists are rewritten
          if (tid == 0) { sh.nrow = 0; sh.ncol = 0; }
          __syncthreads();
        }
      }
      if (sh.goal.need_e && !bail) {
        // A pair of gain >= LB has d_i + d_j <= c*w - s, with d the distance
        // of an end from its side's maximum and s = LB - Am - Bm (for pairs
        // with a tabu side LT - AA - BA).  So d <= p - s at both ends (the
        // bitmap), and at the end with the smaller d even 2d <= c*w - s: only
        // the entries of such ends, of at least that weight, are looked at.
        const KeyT q_nt = plus - sh.goal.s_nt, q_all = plus - sh.goal.s_all;
        // Thresholds of the value itself: non-tabu positions may pair as
        // either kind, tabu ones as the second only.
        auto bar = [&](KeyT Mn, KeyT Ma, bool nt) {
          const KeyT a = Ma - q_all, n = Mn - q_nt;
          return nt && nt_ok && q_nt >= 0 && (q_all < 0 || n < a) ? n : (q_all >= 0 ? a : KeyLim<KeyT>::high);
        };
        const KeyT row_n = bar(Am, AA, true), row_t = bar(Am, AA, false);
        const KeyT col_n = bar(Bm, BA, true), col_t = bar(Bm, BA, false);
        // distances of a candidate, doubled; what does not apply is past its slack
        auto twice = [&](int32_t x, KeyT& dn, KeyT& da) {
          const bool row = x < rpc;
          const KeyT y = PROB == P_MDP && row ? -val[x] : val[x];
          da = (row ? AA : BA) - y;
          dn = nt_ok && stamp[x] <= now ? (row ? Am : Bm) - y : q_nt / 2 + 1;
          dn = dn > q_nt ? q_nt + 1 : 2 * dn;
          da = da > q_all ? q_all + 1 : 2 * da;
        };
        // A thread marks its candidates among up to 32 positions, then the
        // warp takes list space once: the two counts travel in one word.
#pragma unroll 1
        for (int32_t base = 0; base < rpc + cpc; base += 32 * T) {
          unsigned full = 0, half = 0;
#pragma unroll 4
          for (int32_t k = 0; k < 32; k++) {
            const int32_t x = base + k * T + tid;
            if (x >= rpc + cpc) break;
            const bool row = x < rpc;
            if (row ? x >= nr : x - rpc >= nc) continue;
            const KeyT y = PROB == P_MDP && row ? -val[x] : val[x];
            if (y >= (stamp[x] <= now ? (row ? row_n : col_n) : (row ? row_t : col_t))) full |= 1u << k;
          }
          if (!__any_sync(0xffffffffu, full)) continue;
#pragma unroll 1
          for (unsigned left = full; left; left &= left - 1) {
            const int b = __ffs(left) - 1;
            KeyT dn, da;
            twice(base + b * T + tid, dn, da);
            if (dn <= q_nt || da <= q_all) half |= 1u << b;
          }
          const unsigned own = (unsigned)__popc(nb > 1 ? full : 0u) << 16 | (unsigned)__popc(half);
          unsigned incl = own;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
          }
          int32_t af = 0, ah = 0;
          if (lane == 31) {
            if (nb > 1) af = atomicAdd(&sh.ncol, (int32_t)(incl >> 16));
            ah = atomicAdd(&sh.nrow, (int32_t)(incl & 0xffffu));
          }
          af = __shfl_sync(0xffffffffu, af, 31) + (int32_t)((incl - own) >> 16);
          ah = __shfl_sync(0xffffffffu, ah, 31) + (int32_t)((incl - own) & 0xffffu);
#pragma unroll 1
          for (unsigned left = full; left; left &= left - 1) {
            const int b = __ffs(left) - 1;
            const int32_t x = base + b * T + tid, v = ids[x];
            if (nb == 1) {
              atomicOr(&map[v >> 5], 1u << (v & 31));
            } else {
              if (af < L.ccap) cll[af] = v;
              af++;
            }
            if (half >> b & 1u) {
              if (ah < L.rcap) rl[ah] = x;
              ah++;
            }
          }
        }
        __syncthreads();
        const int32_t items = sh.nrow;
        bool over = items > L.rcap;
        int32_t* lst = reinterpret_cast<int32_t*>(smem + L.stage);  // a round's rows: slice index, length,
        int32_t* len = lst + kCandTPB;                              // start and smallest c*w of interest
        long long* rs = reinterpret_cast<long long*>(len + kCandTPB);
        KeyT* least = reinterpret_cast<KeyT*>(rs + kCandTPB);
        int32_t* hits = reinterpret_cast<int32_t*>(smem + L.hits);
        // the first round's rows are fetched while the other CTAs' lists settle
        if (nb > 1) cl.barrier_arrive();
#pragma unroll 1
        for (int32_t base = 0; base < items || base == 0; base += T) {
          int32_t l = 0;
          if (base + tid < items && !over) {
            const int32_t x = rl[base + tid], u = ids[x];
            const int2 wr = __ldg(g.wrange + u);
            long long start;
            l = row_of(u, start);
            KeyT dn, da;
            twice(x, dn, da);
            const KeyT fn = dn + sh.goal.s_nt, fa = da + sh.goal.s_all;
            const KeyT f = dn <= q_nt && (da > q_all || fn < fa) ? fn : fa;
            if ((PROB == P_MDP ? -(KeyT)wr.x : (KeyT)2 * (KeyT)wr.y) < f) l = 0;  // no entry weighs enough
            if (l > 1 << kCandRowBits) {  // (parallel edges) counts as too many kept entries: a sweep
              atomicAdd(&sh.nhits, kCandHits + 1);
              l = 0;
            }
            if (l > kCandHeavy) {
              const int32_t at = atomicAdd(&sh.nheavy, 1);
              if (at < kCandHeavyList) {
                sh.heavy[at] = tid;
                l = -l;  // left out by the warps
              }
            }
            lst[tid] = x;
            rs[tid] = start;
            least[tid] = f;
          }
          len[tid] = l;
          if (nb > 1 && base == 0) {
            cl.barrier_wait();
            // every CTA sets the bits of all lists, a list to a few warps
            const int32_t cc = lane < nb ? *cl.map_shared_rank(&sh.ncol, lane) : 0;
            over |= __reduce_max_sync(0xffffffffu, cc) > L.ccap;
            const int per = nw / nb > 0 ? nw / nb : 1;
            if (!over)
#pragma unroll 1
              for (int r = warp % nb; r < nb && warp < per * nb; r += nw) {
                const int32_t cnt = __shfl_sync(0xffffffffu, cc, r);
                const uint32_t src = cta_smem(sbase, r) + L.cl;
#pragma unroll 1
                for (int32_t e = (warp / nb) * 128 + lane; e - lane < cnt; e += per * 128) {
                  int32_t v[4];
#pragma unroll
                  for (int k = 0; k < 4; k++) v[k] = e + k * 32 < cnt ? ld_cta32(src + 4u * (uint32_t)(e + k * 32)) : -1;
#pragma unroll
                  for (int k = 0; k < 4; k++)
                    if (v[k] >= 0) atomicOr(&map[v[k] >> 5], 1u << (v[k] & 31));
                }
              }
          }
          __syncthreads();
          if (over) break;
          // Eight rows a warp, 32 entries (a chunk) at a time, eight chunks in
          // flight whether they are of long rows or of short ones; then the
          // long rows' chunks, shared by all warps.
          const int32_t cnt = min(T, items - base), nh = min(sh.nheavy, kCandHeavyList);
          int32_t g0 = 0, c0 = 0, chunks = -1, incl = 0, mylen = 0, h = 0, k0 = warp;
          for (;;) {
            int32_t r[8], k[8];
            int2 e[8];
            if (g0 < cnt) {
              if (chunks < 0) {
                const int32_t own = g0 + lane * nw + warp;
                mylen = lane < 8 && own < cnt ? max(len[own], 0) : 0;
                incl = (mylen + 31) >> 5;
#pragma unroll
                for (int o = 1; o < 8; o <<= 1) {
                  const int32_t t = __shfl_up_sync(0xffffffffu, incl, o);
                  if (lane >= o) incl += t;
                }
                chunks = __shfl_sync(0xffffffffu, incl, 7);
                c0 = 0;
              }
#pragma unroll
              for (int x = 0; x < 8; x++) {
                const int r8 = __popc(__ballot_sync(0xffffffffu, lane < 8 && incl <= c0 + x));
                const int32_t before = __shfl_sync(0xffffffffu, incl, (r8 - 1) & 7);
                const int32_t lr = __shfl_sync(0xffffffffu, mylen, r8 & 7);
                r[x] = g0 + (r8 & 7) * nw + warp;
                k[x] = (c0 + x - (r8 ? before : 0)) * 32 + lane;
                if (c0 + x >= chunks || k[x] >= lr) r[x] = -1;
              }
              c0 += 8;
              if (c0 >= chunks) { g0 += 8 * nw; chunks = -1; }
            } else if (h < nh) {
              const int32_t row = sh.heavy[h], lr = -len[row];
#pragma unroll
              for (int x = 0; x < 8; x++) {
                k[x] = (k0 + x * nw) * 32 + lane;
                r[x] = k[x] < lr ? row : -1;
              }
              k0 += 8 * nw;
              if (k0 * 32 >= lr) { h++; k0 = warp; }
            } else {
              break;
            }
#pragma unroll
            for (int x = 0; x < 8; x++) {
              e[x] = make_int2(-1, 0);
              if (r[x] >= 0) e[x] = __ldg(g.adj + rs[r[x]] + k[x]);
            }
            // kept: entries that weigh enough and end at a candidate
            unsigned keep = 0;
#pragma unroll
            for (int x = 0; x < 8; x++) {
              if (e[x].x < 0) continue;
              const KeyT c = PROB == P_MDP ? -(KeyT)e[x].y : (KeyT)2 * (KeyT)e[x].y;
              if (c >= least[r[x]] && (map[e[x].x >> 5] >> (e[x].x & 31) & 1u)) keep |= 1u << x;
            }
            if (!__any_sync(0xffffffffu, keep)) continue;
            int32_t pre = __popc(keep);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
              const int32_t t = __shfl_up_sync(0xffffffffu, pre, o);
              if (lane >= o) pre += t;
            }
            int32_t at = 0;
            if (lane == 31) at = atomicAdd(&sh.nhits, pre);
            at = __shfl_sync(0xffffffffu, at, 31) + pre - __popc(keep);
#pragma unroll
            for (int x = 0; x < 8; x++)
              if (keep >> x & 1u) {
                if (at < kCandHits) hits[at] = r[x] | k[x] << 9;
                at++;
              }
          }
          __syncthreads();
          // the kept entries, evaluated exactly
          if (sh.nhits > kCandHits) over = true;
          const int32_t kept = over ? 0 : sh.nhits;
#pragma unroll 1
          for (int32_t f = tid; f < kept; f += T) {
            const int32_t w = hits[f], r = w & 511, x = lst[r];
            const long long at = rs[r] + (w >> 9);
            const int2 e = __ldg(g.adj + at);
            const int32_t p = pos_of(e.x);
            const bool row = x < rpc;
            if (row == (p < m)) continue;  // both ends on one side
            uint32_t base2;
            const int32_t x2 = place(p, base2);
            KeyT other;
            ld_cta(base2 + L.va + (uint32_t)(kKb * x2), other);
            CandBest<KeyT> y;
            y.a = row ? val[x] : other;
            y.b = row ? other : val[x];
            y.key = pair_gain<PROB, KeyT>(y.a, y.b, e.y);
            if (y.key < LB) continue;
            const bool tabu = stamp[x] > now || ld_cta32(base2 + L.ta + 4u * (uint32_t)x2) > now;
            if (tabu && !(y.key > D)) continue;
            if (at > rs[r] && __ldg(&g.adj[at - 1].x) == e.x) continue;  // duplicated pair: first entry
            y.i = row ? row0 + x : p;
            y.j = row ? p - m : col0 + x - rpc;
            y.u = row ? ids[x] : e.x;
            y.v = row ? e.x : ids[x];
            cand_better(mine, y);
          }
          if (over || base + T >= items) break;
          __syncthreads();  // the round's arrays are reused
          if (tid == 0) { sh.nheavy = 0; sh.nhits = 0; }
          __syncthreads();
        }
        if (over) mine.j = kPairOverflow;
        __syncthreads();  // bits set and read before they are cleared
#pragma unroll 1
        for (uint32_t x = tid; x < L.map_bytes / 16; x += T) reinterpret_cast<uint4*>(map)[x] = make_uint4(0, 0, 0, 0);
      }
      if (bail) { status = kCandBail; break; }
      // ---- block, then cluster best
      const bool over = mine.j == kPairOverflow;
      warp_best<KeyT>(mine);
      if (lane == 0) {
        if (over) mine.j = kPairOverflow;
        sh.wbest[warp] = mine;
      }
      __syncthreads();
      CandBest<KeyT> b;
      b.j = kPairNone;
      if (nb > 1) {
        if (warp == 0) {
          if (lane < nw) b = sh.wbest[lane];
          const bool o = __ballot_sync(0xffffffffu, b.j == kPairOverflow) != 0;
          warp_best<KeyT>(b);
          if (o) b.j = kPairOverflow;
          if (lane < nb) *cl.map_shared_rank(&sh.rec[rank], lane) = b;
        }
        cl.sync();
        b.j = kPairNone;
      }
      if (lane < (nb > 1 ? nb : nw)) b = nb > 1 ? sh.rec[lane] : sh.wbest[lane];
      if (__ballot_sync(0xffffffffu, b.j == kPairOverflow)) { status = kCandBail; break; }
      warp_best<KeyT>(b);
      cand_better(best, b);
    }

    // ---- 4. decision (decide_apply's rules)
    if (best.j < 0 || (PROB == P_MDP && (long long)best.key <= kMdpSentinel)) {
      __syncthreads();
      if (tid == 0) sh.sc.mode = 1;  // no allowed pair above the sentinel: the exact pass decides
      __syncthreads();
      status = kCandBail;
      break;
    }
    budget--;
    const int scribe = T - 64;  // keeps the scalars while the others apply the move
    int32_t t_u = 0, t_v = 0;
    if (tid == T - 1 || tid == scribe) {  // the threads that stamp and trace
      if (PROB == P_MDP) {
        const int32_t c = s.tenure_policy == 0 ? mdp_ref_tenure(iter) : s.tenure;
        t_u = c;
        t_v = s.tenure_policy == 0 ? s.c2_tab[c == 15 ? 0 : c == 30 ? 1 : c == 60 ? 2 : 3] : s.c2_fixed;
      } else {
        t_u = t_v = s.tenure_policy == 0 ? maxbs_ref_tenure(iter, s.maxt) : s.tenure;
      }
    }
    int32_t iu = best.i, jv = best.j, u = best.u, v = best.v;
    KeyT a = best.a, b0 = best.b;
    long long su = sh.goal.row_u, sv = sh.goal.row_v;
    int32_t nu = sh.goal.len_u, nv2 = sh.goal.len_v;
    if (best.i != sh.goal.best.i || best.j != sh.goal.best.j) { nu = row_of(u, su); nv2 = row_of(v, sv); }
    // ---- 5. the move, then the moves of a perturbation where one is due
    long long mv = -1;  // perturbation: the flat index
    for (int32_t turn = 0;; turn++) {
      // bookkeeping: read by the other threads again after the barrier below
      if (tid == scribe) {
        CandScalars& c = sh.sc;
        if (c.log_n < s.log_cap) {
          if (rank == 0) s.movelog[c.log_n] = make_int2(iu, jv);
        } else {
          c.err |= E_LOG_FULL;
        }
        c.log_n++;
        if (turn == 0) {
          const long long key = (long long)best.key;
          c.cur += (PROB == P_MAXBS && key < kMaxbsRecoverBelow) ? key + kMaxbsInf : key;
          c.evaluations += s.P;
          if (c.cur > c.best) {
            c.best = c.cur;
            c.best_log_n = c.log_n;
            c.isi = 0;
          } else {
            c.isi += 1;
          }
          c.iter = iter + 1;
          c.perturb = PROB == P_MAXBS && c.isi >= s.piter;
          if (rank == 0 && s.trace && c.trace_n < s.trace_cap) {
            TraceRec r;
            r.iter = iter; r.idx = (long long)iu * delta + jv; r.key = key; r.cur = c.cur; r.best = c.best;
            r.kind = 0; r.tenure = t_u; r.tenure2 = PROB == P_MDP ? t_v : 0; r.pad = 0;
            s.trace[c.trace_n] = r;
          }
          c.trace_n++;
        }
      }
      // Updates of the swap by the whole cluster: contributions along the rows
      // of u and v (shared-memory atomics on the owners), the swapped slots,
      // positions, CSR cpos and the clearing half of the WSwap patch.  Four
      // entries per thread are in flight (a dense or hub row is several
      // rounds of the CTA).
      constexpr int kBatch = 4;
      const int32_t total = nu + nv2, step = nb * T;
#pragma unroll 1
      for (int32_t base = rank * T + tid; base < total; base += kBatch * step) {
        int2 e[kBatch];
        int32_t p[kBatch];
        long long mirror[ST == S_CSR ? kBatch : 1];
#pragma unroll
        for (int x = 0; x < kBatch; x++) {
          const int32_t k = base + x * step;
          e[x] = make_int2(-1, 0);
          if (k < total) {
            const long long at = k < nu ? su + k : sv + (k - nu);
            e[x] = __ldg(g.adj + at);
            if constexpr (ST == S_CSR) mirror[x] = __ldg(g.rev + at);
          }
        }
#pragma unroll
        for (int x = 0; x < kBatch; x++) p[x] = e[x].x >= 0 ? pos_of(e[x].x) : 0;
#pragma unroll
        for (int x = 0; x < kBatch; x++) {
          const int32_t k = base + x * step, z = e[x].x, w = e[x].y;
          if (k >= total) break;
          const bool from_u = k < nu;
          if constexpr (ST == S_CSR) s.cpos[mirror[x]] = from_u ? m + jv : iu;  // new position of u / v
          if (PROB == P_MAXBS && from_u && z == v && (k == 0 || __ldg(&g.adj[su + k - 1].x) != z))
            *cl.map_shared_rank(&sh.wuv, 0) = w;
          const bool moved = z == u || z == v;  // their slots after the swap, negated with them in Max Bisection
          const bool z_in = moved ? z == u : p[x] < m;
          KeyT d;
          if (PROB == P_MDP) {
            d = from_u ? -(KeyT)w : (KeyT)w;
          } else {
            d = (from_u == z_in) != moved ? -(KeyT)2 * (KeyT)w : (KeyT)2 * (KeyT)w;
          }
          uint32_t base2;
          const int32_t x2 = place(moved ? (z == u ? m + jv : iu) : p[x], base2);
          add_cta(base2 + L.va + (uint32_t)(kKb * x2), d);
          if (ST == S_WSWAP && !moved) {
            // row iu stops being u's, column jv stops being v's
            if (from_u && !z_in) w_set(s, (long long)iu * s.ldc + (p[x] - m), 0);
            if (!from_u && z_in) w_set(s, (long long)p[x] * s.ldc + jv, 0);
          }
        }
      }
      if (rank == 0 && tid == T - 1) {
        // v takes slot iu, u takes slot jv; added as a difference, so that it
        // commutes with the entries' updates of the two slots
        const KeyT fa = PROB == P_MDP ? a : -a, fb = PROB == P_MDP ? b0 : -b0;
        uint32_t bi, bj;
        const int32_t xi = place(iu, bi), xj = place(m + jv, bj);
        add_cta(bi + L.va + (uint32_t)(kKb * xi), fb - a);
        add_cta(bj + L.va + (uint32_t)(kKb * xj), fa - b0);
        st_cta32(bi + L.ua + 4u * (uint32_t)xi, v);
        st_cta32(bj + L.ua + 4u * (uint32_t)xj, u);
        const uint32_t ri = bi + L.ta + 4u * (uint32_t)xi, rj = bj + L.ta + 4u * (uint32_t)xj;
        // a perturbation's stamps travel with the vertices
        const int32_t ni = turn == 0 ? (int32_t)(iter + t_v) : ld_cta32(rj);
        const int32_t nj = turn == 0 ? (int32_t)(iter + t_u) : ld_cta32(ri);
        st_cta32(ri, ni);
        st_cta32(rj, nj);
        if (L.vpc) {
          const int32_t ou = div_by(u, inv_v), ov = div_by(v, inv_v);
          st_cta32(cta_smem(sbase, ou) + L.pv + 4u * (uint32_t)(u - ou * L.vpc), m + jv);
          st_cta32(cta_smem(sbase, ov) + L.pv + 4u * (uint32_t)(v - ov * L.vpc), iu);
        } else {
          s.pos[u] = m + jv;
          s.pos[v] = iu;
        }
      }
      barrier();
      if (ST == S_WSWAP) {
        // the setting half: row iu at v's outside neighbours, column jv at u's
        // inside ones, first entry of a duplicated pair, (iu, jv) left alone
#pragma unroll 1
        for (int32_t k = rank * T + tid; k < total; k += step) {
          const bool from_u = k < nu;
          const long long at = from_u ? su + k : sv + (k - nu);
          const int2 e = __ldg(g.adj + at);
          if (e.x == u || e.x == v) continue;
          if (at != (from_u ? su : sv) && __ldg(&g.adj[at - 1].x) == e.x) continue;
          const int32_t p = pos_of(e.x);
          if (!from_u && p >= m) w_set(s, (long long)iu * s.ldc + (p - m), e.y);
          if (from_u && p < m) w_set(s, (long long)p * s.ldc + jv, e.y);
        }
      }
      if (PROB != P_MAXBS || !sh.sc.perturb) break;
      // ---- perturbation: turn 0 only looks the event up, turn q applied its
      // q-th move
      const long long ev = sh.sc.pert_events - pert_base;
      const bool in_window = ev >= 0 && ev < s.draw_events && ev < pert_limit;
      uint32_t bi, bj;
      if (turn > 0 && tid == scribe) {
        CandScalars& c = sh.sc;
        // the slots now hold the negated contributions after the update
        const int32_t xi = place(iu, bi), xj = place(m + jv, bj);
        KeyT na, ob;
        ld_cta(bj + L.va + (uint32_t)(kKb * xj), na);
        ld_cta(bi + L.va + (uint32_t)(kKb * xi), ob);
        const long long aux = -(long long)na - (long long)ob - 2LL * *cl.map_shared_rank(&sh.wuv, 0);
        c.cur += aux;
        c.pert_moves += 1;
        if (rank == 0 && s.trace && c.trace_n < s.trace_cap) {
          TraceRec r;
          r.iter = iter + 1; r.idx = mv; r.key = aux; r.cur = c.cur; r.best = c.best;
          r.kind = 2; r.tenure = 0; r.tenure2 = 0; r.pad = 0;
          s.trace[c.trace_n] = r;
        }
        c.trace_n++;
      }
      bool bad = false;
      if (in_window && turn < s.num_pert) {
        mv = __ldg(s.draws + ev * s.num_pert + turn);
        bad = mv < 0 || mv >= s.P;
      }
      if (!in_window || turn >= s.num_pert || bad) {
        barrier();  // slots and wuv read, scalars of the last move written
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
        break;
      }
      barrier();  // wuv and the last move's slots read before the next move's updates
      iu = (int32_t)(mv / delta);
      jv = (int32_t)(mv % delta);
      const int32_t xi = place(iu, bi), xj = place(m + jv, bj);
      u = ld_cta32(bi + L.ua + 4u * (uint32_t)xi);
      v = ld_cta32(bj + L.ua + 4u * (uint32_t)xj);
      ld_cta(bi + L.va + (uint32_t)(kKb * xi), a);
      ld_cta(bj + L.va + (uint32_t)(kKb * xj), b0);
      nu = row_of(u, su);
      nv2 = row_of(v, sv);
      if (rank == 0 && tid == 0) sh.wuv = 0;
      barrier();  // slots read before anyone updates them
    }
  }

#pragma unroll 1
  for (int32_t x = tid; x < rpc + cpc; x += T) {
    const bool row = x < rpc;
    const int32_t i = row ? x : x - rpc;
    if (i >= (row ? nr : nc)) continue;
    (row ? s.vg_in + row0 : s.vg_out + col0)[i] = val[x];
    (row ? s.tab_in + row0 : s.tab_out + col0)[i] = stamp[x];
    (row ? s.sol_in + row0 : s.sol_out + col0)[i] = ids[x];
  }
#pragma unroll 1
  for (int32_t v = tid; v < nv; v += T) s.pos[v0 + v] = pv[v];
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
