// graph.cu -- device-side graph builders for the six lookup structures and
// the single lookup interface.
//
// Reference builders replaced: read_instance/createCSR (src/mdp/GPU-MDP-CSR.cu:
// 210-367, host sort + H2D), load/createCSR (src/maxbisection/GPU-MAXBS-CSR.cu:
// 112-173), the host bitmap (src/mdp/GPU-MDP-CSR-Bitset-BuscaBinaria.cu:321-378),
// and the uint32-keyed global hash table (src/mdp/GPU-MDP-Hash.cu:140-217,413-440),
// whose (u<<16)|v key aliases once n > 65,536.  Here everything is built on the
// device from the edge list: one stable radix sort of 64-bit (row, neighbour)
// keys produces the CSR; bitset rows and per-vertex hash tables are filled from
// it.  The hash tables are keyed by (row vertex, neighbour) -- the row selects
// the table, the neighbour id is the key -- so no aliasing at any n; keys and
// weights are stored as separate arrays so a probe reads 4 bytes.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>

#include "ts_host.h"

namespace tsb {

static thread_local std::string g_last_error;

void set_error(const std::string& msg) { g_last_error = msg; }
const char* last_error() { return g_last_error.c_str(); }

ts_status cuda_fail(cudaError_t e, const char* what) {
  std::string m = std::string(what) + ": " + cudaGetErrorString(e);
  set_error(m);
  cudaGetLastError();  // clear sticky-free errors
  return e == cudaErrorMemoryAllocation ? TS_ERR_OUT_OF_MEMORY : TS_ERR_CUDA;
}

uint64_t context_id() {
  // Reached through the runtime, so that the library needs no link-time
  // dependency on the driver library.
  using GetCurrent = int (*)(void**);
  using GetId = int (*)(void*, unsigned long long*);
  struct Driver {
    GetCurrent current = nullptr;
    GetId id = nullptr;
  };
  static const Driver d = [] {
    Driver f;
    auto find = [](const char* name) {
      void* fn = nullptr;
      cudaDriverEntryPointQueryResult q;
      if (cudaGetDriverEntryPoint(name, &fn, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) {
        cudaGetLastError();
        fn = nullptr;
      }
      return fn;
    };
    f.current = reinterpret_cast<GetCurrent>(find("cuCtxGetCurrent"));
    f.id = reinterpret_cast<GetId>(find("cuCtxGetId"));
    return f;
  }();
  void* ctx = nullptr;
  unsigned long long id = 0;
  if (!d.current || !d.id || d.current(&ctx) != 0) return 0;
  if (!ctx || d.id(ctx, &id) != 0) {
    // none bound to this thread yet, or one that a reset has ended: the
    // device's primary context, the one the runtime would use
    int dev = 0;
    id = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaSetDevice(dev) != cudaSuccess || d.current(&ctx) != 0 || !ctx ||
        d.id(ctx, &id) != 0) {
      cudaGetLastError();
      return 0;
    }
  }
  return id;
}

// One pool per context: a context that ends (a device reset) takes its pool,
// stream and memory along, and the next one gets a pool of its own.  Entries
// of ended contexts stay, so that an entry's address says which context a
// block belongs to.
struct Pool {
  uint64_t ctx = 0;
  cudaMemPool_t pool = nullptr;
  cudaStream_t stream = nullptr;  // allocations and frees for any stream
  int users = 0;
};

namespace {
constexpr int kMaxPools = 64;
std::mutex g_pool_mu;
Pool g_pool[kMaxPools];
int g_pools = 0;

// The current context's pool; null (no context ids, no pool to be had, or 64
// contexts before this one): plain allocations.
Pool* context_pool() {
  const uint64_t ctx = context_id();
  if (!ctx) return nullptr;
  std::lock_guard<std::mutex> lock(g_pool_mu);
  for (int k = 0; k < g_pools; k++)
    if (g_pool[k].ctx == ctx) return g_pool[k].pool ? &g_pool[k] : nullptr;
  if (g_pools == kMaxPools) return nullptr;
  Pool& t = g_pool[g_pools++];
  t.ctx = ctx;
  int dev = 0;
  cudaMemPoolProps props = {};
  props.allocType = cudaMemAllocationTypePinned;
  props.handleTypes = cudaMemHandleTypeNone;
  props.location.type = cudaMemLocationTypeDevice;
  uint64_t keep = kPoolKeep;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaStreamCreateWithFlags(&t.stream, cudaStreamNonBlocking) != cudaSuccess ||
      (props.location.id = dev, cudaMemPoolCreate(&t.pool, &props)) != cudaSuccess) {
    t.pool = nullptr;
    cudaGetLastError();
    return nullptr;
  }
  cudaMemPoolSetAttribute(t.pool, cudaMemPoolAttrReleaseThreshold, &keep);
  return &t;
}

// Tried again once what the pool holds unused has been given back; a pool that
// still does not get what it needs gives back what it got.
template <class Get>
cudaError_t with_trim(Get&& get) {
  for (int attempt = 0;; attempt++) {
    const cudaError_t e = get();
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    pool_trim();
    if (attempt) return e;
  }
}
}  // namespace

cudaError_t pool_get(PoolBlock& b, size_t bytes, bool ordered, cudaStream_t st) {
  b = PoolBlock{};
  b.ctx = context_id();
  b.ordered = ordered;
  b.stream = st;
  Pool* t = context_pool();
  cudaError_t e;
  if (!t || (!ordered && bytes > kPoolBlock)) {
    e = with_trim([&] { return cudaMalloc(&b.p, bytes); });
  } else {
    b.pool = t;
    if (!ordered) b.stream = t->stream;
    e = with_trim([&] { return cudaMallocFromPoolAsync(&b.p, bytes, t->pool, b.stream); });
    if (e == cudaSuccess && !ordered) e = cudaStreamSynchronize(b.stream);
  }
  if (e != cudaSuccess) b.p = nullptr;
  return e;
}
void pool_put(PoolBlock& b) {
  if (b.p && context_id() == b.ctx) {  // else its context has ended, and the memory with it
    if (!b.pool) {
      if (b.ordered) cudaStreamSynchronize(b.stream);
      cudaFree(b.p);
    } else {
      if (!b.ordered) cudaDeviceSynchronize();
      cudaFreeAsync(b.p, b.stream);
    }
  }
  b = PoolBlock{};
}
void pool_trim() {
  Pool* t = context_pool();
  if (!t) return;
  cudaDeviceSynchronize();  // frees still queued on a stream
  cudaMemPoolTrimTo(t->pool, 0);
}
Pool* pool_enter() {
  Pool* t = context_pool();
  if (!t) return nullptr;
  std::lock_guard<std::mutex> lock(g_pool_mu);
  t->users++;
  return t;
}
void pool_leave(Pool* t) {
  if (!t) return;
  {
    std::lock_guard<std::mutex> lock(g_pool_mu);
    if (--t->users > 0) return;
  }
  if (context_id() == t->ctx) cudaMemPoolTrimTo(t->pool, kPoolIdle);
}

cudaError_t allow_dyn_smem(const void* fn, size_t smem) {
  // The default limit is 48 KB minus the kernel's static shared memory, so
  // even a request below 48 KB may need the attribute raised.
  static std::mutex mu;
  std::lock_guard<std::mutex> lock(mu);
  cudaFuncAttributes fa;
  cudaError_t e = cudaFuncGetAttributes(&fa, fn);
  if (e != cudaSuccess) return e;
  if ((size_t)fa.maxDynamicSharedSizeBytes >= smem) return cudaSuccess;
  return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

namespace {

constexpr int kTPB = 256;

inline int blocks_for(int64_t n, int tpb = kTPB) {
  int64_t b = (n + tpb - 1) / tpb;
  if (b < 1) b = 1;
  if (b > 148LL * 64) b = 148 * 64;  // grid-stride loops cover the rest
  return (int)b;
}

// Directed entries: 2 per edge ((u,v) at 2e, (v,u) at 2e+1), key = row<<cb|col
// with cb the bits of a column, so that the sort has no idle bits to pass over.
// Dropped self-loops and out-of-range endpoints get row n (sorted past the end).
__global__ void k_make_keys(int32_t n, int cb, int64_t E, const int32_t* __restrict__ u,
                            const int32_t* __restrict__ v, const int32_t* __restrict__ w,
                            int drop_self, unsigned long long* __restrict__ keys,
                            int32_t* __restrict__ vals, int32_t* __restrict__ err) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < E;
       e += (int64_t)gridDim.x * blockDim.x) {
    int32_t a = u[e], b = v[e];
    bool bad = a < 0 || a >= n || b < 0 || b >= n;
    if (bad) atomicOr(err, E_BAD_EDGE);
    bool skip = bad || (drop_self && a == b);
    unsigned long long ra = skip ? (unsigned long long)n : (unsigned long long)a;
    unsigned long long rb = skip ? (unsigned long long)n : (unsigned long long)b;
    const int32_t x = w[e];
    reinterpret_cast<ulonglong2*>(keys)[e] =
        make_ulonglong2((ra << cb) | (unsigned)(skip ? 0 : b), (rb << cb) | (unsigned)(skip ? 0 : a));
    reinterpret_cast<int2*>(vals)[e] = make_int2(x, x);
  }
}

// rowptr[r] = first sorted entry whose row >= r; entries with row == n are past the end.
__global__ void k_rowptr(int32_t n, int cb, int64_t N, const unsigned long long* __restrict__ keys,
                         int64_t* __restrict__ rowptr) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k <= N;
       k += (int64_t)gridDim.x * blockDim.x) {
    int64_t rp = k == 0 ? -1 : (int64_t)(keys[k - 1] >> cb);
    int64_t rc = k == N ? n : (int64_t)(keys[k] >> cb);
    if (rp > n) rp = n;
    if (rc > n) rc = n;
    for (int64_t r = rp + 1; r <= rc; r++) rowptr[r] = k;
  }
}

// The kernels over entries run over all sorted keys and leave out those of row
// n: how many there are is not known on the host yet.
__global__ void k_pack_adj(int32_t n, int cb, int64_t N2, const unsigned long long* __restrict__ keys,
                           const int32_t* __restrict__ vals, int2* __restrict__ adj) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < N2;
       k += (int64_t)gridDim.x * blockDim.x) {
    const unsigned long long key = keys[k];
    if ((int64_t)(key >> cb) < n) adj[k] = make_int2((int32_t)(key & ((1ull << cb) - 1)), vals[k]);
  }
}

// Per-row sum |w|: bounds |contribution| and decides the 32-bit key path
// (out[0]); out[1] != 0 when some weight is negative; out[2] = max |w| (the
// WSwap matrix holds 16-bit weights when it fits); the range of each row's
// weights (the candidate pass leaves rows out by it).  A warp per row, one
// atomic per block and result.
__global__ void __launch_bounds__(kTPB)
k_max_wdeg(int32_t n, const int64_t* __restrict__ rowptr, const int2* __restrict__ adj,
           unsigned long long* __restrict__ out, int2* __restrict__ wrange) {
  __shared__ unsigned long long s_sum, s_abs;
  __shared__ int s_neg;
  if (threadIdx.x == 0) { s_sum = 0; s_abs = 0; s_neg = 0; }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  unsigned long long best = 0;
  int32_t lo = 0, hi = 0;  // of all the warp's rows
  for (int32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n; r += (gridDim.x * blockDim.x) >> 5) {
    unsigned long long sum = 0;
    int2 wr = make_int2(0, 0);  // of the row's weights and 0
    for (int64_t k = rowptr[r] + lane; k < rowptr[r + 1]; k += 32) {
      const int32_t x = adj[k].y;
      sum += (unsigned long long)(x < 0 ? -(long long)x : (long long)x);
      wr.x = min(wr.x, x);
      wr.y = max(wr.y, x);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sum += __shfl_xor_sync(0xffffffffu, sum, o);
      wr.x = min(wr.x, __shfl_xor_sync(0xffffffffu, wr.x, o));
      wr.y = max(wr.y, __shfl_xor_sync(0xffffffffu, wr.y, o));
    }
    if (lane == 0) wrange[r] = wr;
    best = sum > best ? sum : best;
    lo = min(lo, wr.x);
    hi = max(hi, wr.y);
  }
  if (lane == 0) {
    const unsigned long long a = (unsigned long long)(-(long long)lo), b = (unsigned long long)hi;
    atomicMax(&s_sum, best);
    atomicMax(&s_abs, a > b ? a : b);
    if (lo < 0) atomicOr(&s_neg, 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (s_sum) atomicMax(out, s_sum);
    if (s_neg) atomicMax(out + 1, 1ull);
    if (s_abs) atomicMax(out + 2, s_abs);
  }
}

// Row of entry k: from its sorted key, or, where the keys had to make room for
// the graph (keys null), the last row that starts at or before k.
__device__ __forceinline__ int64_t row_of(int32_t n, int cb, const unsigned long long* __restrict__ keys,
                                          const int64_t* __restrict__ rowptr, int64_t k) {
  if (keys) return (int64_t)(keys[k] >> cb);
  int32_t lo = 0, hi = n - 1;
  while (lo < hi) {
    const int32_t mid = (lo + hi + 1) >> 1;
    if (rowptr[mid] <= k) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__global__ void k_fill_bits(int32_t n, int cb, int64_t N2, const unsigned long long* __restrict__ keys,
                            const int64_t* __restrict__ rowptr, const int2* __restrict__ adj, int64_t wpr,
                            unsigned long long* __restrict__ bits) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < N2;
       k += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = row_of(n, cb, keys, rowptr, k);
    if (r >= n) continue;
    const int32_t c = keys ? (int32_t)(keys[k] & ((1ull << cb) - 1)) : adj[k].x;
    atomicOr(&bits[r * wpr + (c >> 6)], 1ull << (c & 63));
  }
}

__global__ void k_hash_caps(int32_t n, const int64_t* __restrict__ rowptr, int64_t* __restrict__ caps) {
  for (int32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x)
    caps[r] = hash_capacity(rowptr[r + 1] - rowptr[r]);
  if (blockIdx.x == 0 && threadIdx.x == 0) caps[n] = 0;
}

// Inserts the first entry of every (row, neighbour) pair with linear probing.
__global__ void k_hash_insert(int32_t n, int cb, int64_t N, const unsigned long long* __restrict__ sorted,
                              const int64_t* __restrict__ rowptr, const int2* __restrict__ adj, const int64_t* __restrict__ hoff,
                              int32_t* __restrict__ keys, int32_t* __restrict__ vals,
                              int32_t* __restrict__ err) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < N;
       k += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = row_of(n, cb, sorted, rowptr, k);
    int2 e = adj[k];
    if (k > rowptr[r] && adj[k - 1].x == e.x) continue;  // duplicate pair: first wins
    const int64_t base = hoff[r];
    const int64_t cap = hoff[r + 1] - base;
    const uint32_t gmask = (uint32_t)(cap / 4 - 1);
    uint32_t grp = hash_group(e.x, hash_gshift(cap));
    bool ok = false;
    for (uint32_t t = 0; t <= gmask && !ok; t++) {
      for (int sl = 0; sl < 4; sl++) {
        const int64_t at = base + 4LL * grp + sl;
        if (atomicCAS(&keys[at], kHashEmpty, e.x) == kHashEmpty) {
          vals[at] = e.y;
          ok = true;
          break;
        }
      }
      grp = (grp + 1) & gmask;
    }
    if (!ok) atomicOr(err, E_HASH_FULL);
  }
}

// rev[k] for entry k = (y -> z): the entry (z -> y) in row z with the same
// duplicate rank (a self-loop's entries map to themselves).
__global__ void k_reverse_index(int32_t n, int cb, int64_t N2, const unsigned long long* __restrict__ keys,
                                const int64_t* __restrict__ rowptr, const int2* __restrict__ adj,
                                int64_t* __restrict__ rev) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < N2;
       k += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = row_of(n, cb, keys, rowptr, k);
    if (row >= n) continue;
    const int32_t y = (int32_t)row;
    const int32_t z = adj[k].x;
    auto lower = [&](int32_t row, int32_t key) {
      int64_t lo = rowptr[row], len = rowptr[row + 1] - lo;
      while (len > 0) {
        int64_t half = len >> 1;
        if (adj[lo + half].x < key) { lo += half + 1; len -= half + 1; }
        else len = half;
      }
      return lo;
    };
    const int64_t t = k - lower(y, z);
    rev[k] = lower(z, y) + t;
  }
}

}  // namespace

// ------------------------------------------------------------- lookups
// First entry of row u with neighbour v (gpu_edge semantics, GPU-MDP-CSR.cu:555-564).
__device__ __forceinline__ int32_t csr_scan(const DevGraph& g, int32_t u, int32_t v) {
  for (int64_t k = g.rowptr[u]; k < g.rowptr[u + 1]; k++) {
    int2 e = g.adj[k];
    if (e.x == v) return e.y;
  }
  return 0;
}

// lower_bound over the sorted row (binary-search variant,
// GPU-MDP-CSR-BuscaBinaria.cu:554-566, returning the first duplicate).
__device__ __forceinline__ int32_t csr_bsearch(const DevGraph& g, int32_t u, int32_t v) {
  int64_t lo = g.rowptr[u], len = g.rowptr[u + 1] - lo;
  while (len > 0) {
    int64_t half = len >> 1;
    if (g.adj[lo + half].x < v) { lo += half + 1; len -= half + 1; }
    else len = half;
  }
  if (lo < g.rowptr[u + 1] && g.adj[lo].x == v) return g.adj[lo].y;
  return 0;
}

__device__ __forceinline__ int32_t lookup_any(const DevGraph& g, int32_t u, int32_t v) {
  switch (g.kind) {
    case S_HASH: {
      const int64_t base = g.hoff[u];
      const int64_t cap = g.hoff[u + 1] - base;
      const uint32_t gmask = (uint32_t)(cap / 4 - 1);
      uint32_t grp = hash_group(v, hash_gshift(cap));
      for (uint32_t t = 0; t <= gmask; t++) {
        const int4 k4 = *reinterpret_cast<const int4*>(g.hkey + base + 4LL * grp);
        const int32_t ks[4] = {k4.x, k4.y, k4.z, k4.w};
        bool empty = false;
        for (int sl = 0; sl < 4; sl++) {
          if (ks[sl] == v) return g.hval[base + 4LL * grp + sl];
          empty |= ks[sl] == kHashEmpty;
        }
        if (empty) return 0;
        grp = (grp + 1) & gmask;
      }
      return 0;
    }
    case S_BITSET:
    case S_BITSET_BB: {
      uint64_t word = g.bits[u * g.wpr + (v >> 6)];
      if (!((word >> (v & 63)) & 1ull)) return 0;
      return g.kind == S_BITSET ? csr_scan(g, u, v) : csr_bsearch(g, u, v);
    }
    case S_BB:
      return csr_bsearch(g, u, v);
    default:  // CSR and WSwap (whose matrix belongs to a solver)
      return csr_scan(g, u, v);
  }
}

__global__ void k_lookup(DevGraph g, int64_t count, const int32_t* __restrict__ u,
                         const int32_t* __restrict__ v, int32_t* __restrict__ w) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < count;
       k += (int64_t)gridDim.x * blockDim.x) {
    int32_t a = u[k], b = v[k];
    w[k] = (a >= 0 && a < g.n && b >= 0 && b < g.n) ? lookup_any(g, a, b) : 0;
  }
}

// ------------------------------------------------------------- build
// Builds from device arrays, or from host arrays (copied first).  All
// temporaries are one allocation (pooled) and so are the graph's arrays (the
// hash tables, whose size needs the degrees, another): an allocation or a free
// synchronises and takes 50 us to milliseconds, and a build had 12 to 20 of
// each.  One host round trip, two for Hash.  Conflict graph, n = 100,000, 3.4M
// edges, from host arrays: Hash 11.2 -> 4.2 to 5.6 ms (2.3 of them the copies;
// the tables' plain allocation varies), CSR 8.7 -> 4.0; a million lookups 3.3 ->
// 1.1 ms.
// Where the device has no room for the temporaries (48 bytes an edge) beside
// all of the graph, only what the sort fills is allocated with them, and the
// bitmap, the reverse index or the hash tables once they are gone; these are
// then filled from the rows, with a search for each entry's row.
static ts_status build_graph(ts_graph* G, int64_t E, const int32_t* u, const int32_t* v, const int32_t* w,
                             bool on_host) {
  cudaStream_t st = G->stream;
  const int32_t n = G->n;
  const int64_t N2 = 2 * E;
  const bool hash = G->kind == TS_STRUCT_HASH;
  const bool bitset = G->kind == TS_STRUCT_CSR_BITSET || G->kind == TS_STRUCT_CSR_BITSET_BB;
  TS_CUDA(cudaSetDevice(G->device));
  int row_bits = 1, cb = 1;
  while ((1LL << row_bits) <= (int64_t)n) row_bits++;
  while ((1LL << cb) < (int64_t)n) cb++;
  ts_status s;
  auto temp = std::make_unique<DevParts>();
  DevPart keys, keys_alt, vals, vals_alt, sum, tmp, caps, full;
  const size_t eb = sizeof(int32_t) * (size_t)E;
  temp->add(keys, sizeof(unsigned long long) * N2);
  temp->add(keys_alt, sizeof(unsigned long long) * N2);
  temp->add(vals, sizeof(int32_t) * N2);
  temp->add(vals_alt, sizeof(int32_t) * N2);
  // sum: wdeg results (3 words), then the error word
  temp->add(sum, 4 * sizeof(unsigned long long));
  if (hash) temp->add(caps, sizeof(int64_t) * (n + 1));
  size_t sort_bytes = 0, scan_bytes = 0;
  {
    cub::DoubleBuffer<unsigned long long> dk;
    cub::DoubleBuffer<int32_t> dv;
    if (N2 > 0) TS_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, dk, dv, N2, 0, cb + row_bits, st));
    int64_t* none = nullptr;
    if (hash) TS_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, none, none, n + 1, st));
  }
  temp->add(tmp, sort_bytes > scan_bytes ? sort_bytes : scan_bytes);
  if ((s = temp->alloc_temp("alloc build temporaries", st)) != TS_OK) return s;

  auto rows = [&] {
    G->mem.add(G->rowptr, sizeof(int64_t) * (n + 1));
    // Two spare entries: the sweep bulk-copies rows from an even entry to an
    // even end (16-byte aligned), which can reach one entry past the last row.
    G->mem.add(G->adj, sizeof(int2) * (N2 + 2));
    G->mem.add(G->wrange, sizeof(int2) * (size_t)n);
    if (hash) G->mem.add(G->hoff, sizeof(int64_t) * (n + 1));
  };
  auto filled = [&](DevParts& mem) {  // from the rows; with the hash tables' turn below
    if (bitset) {
      const int64_t words = ((int64_t)n + 63) / 64;
      G->wpr = (words + 1) & ~1LL;  // even: every row starts on a 16 B boundary
      mem.add(G->bits, sizeof(uint64_t) * (size_t)n * (size_t)G->wpr);
    }
    if (G->kind == TS_STRUCT_CSR) mem.add(G->rev, sizeof(int64_t) * (size_t)(N2 > 0 ? N2 : 1));
  };
  bool later = false;
  rows();
  filled(G->mem);
  s = G->mem.alloc("alloc graph");
  if (s == TS_ERR_OUT_OF_MEMORY && (bitset || G->kind == TS_STRUCT_CSR)) {
    later = true;
    rows();
    s = G->mem.alloc("alloc graph");
  }
  if (s != TS_OK) return s;

  auto* d_sum = sum.as<unsigned long long>();
  auto* d_err = reinterpret_cast<int32_t*>(d_sum + 3);
  TS_CUDA(cudaMemsetAsync(d_sum, 0, 4 * sizeof(unsigned long long), st));
  if (on_host && E > 0) {
    // the sort's second buffers hold the edge arrays until the keys are made
    int32_t* hu = keys_alt.as<int32_t>();  // 4 words per edge: u, v
    int32_t* hw = vals_alt.as<int32_t>();
    TS_CUDA(cudaMemcpyAsync(hu, u, eb, cudaMemcpyHostToDevice, st));
    TS_CUDA(cudaMemcpyAsync(hu + E, v, eb, cudaMemcpyHostToDevice, st));
    TS_CUDA(cudaMemcpyAsync(hw, w, eb, cudaMemcpyHostToDevice, st));
    u = hu;
    v = hu + E;
    w = hw;
  }
  cub::DoubleBuffer<unsigned long long> dk(keys.as<unsigned long long>(), keys_alt.as<unsigned long long>());
  cub::DoubleBuffer<int32_t> dv(vals.as<int32_t>(), vals_alt.as<int32_t>());
  if (E > 0) {
    k_make_keys<<<blocks_for(E), kTPB, 0, st>>>(n, cb, E, u, v, w, G->drop_self_loops, keys.as<unsigned long long>(),
                                                vals.as<int32_t>(), d_err);
    TS_CUDA(cudaGetLastError());
    TS_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, sort_bytes, dk, dv, N2, 0, cb + row_bits, st));
  }
  k_rowptr<<<blocks_for(N2 + 1), kTPB, 0, st>>>(n, cb, N2, dk.Current(), G->rowptr.as<int64_t>());
  TS_CUDA(cudaGetLastError());
  if (E > 0) {
    k_pack_adj<<<blocks_for(N2), kTPB, 0, st>>>(n, cb, N2, dk.Current(), dv.Current(), G->adj.as<int2>());
    TS_CUDA(cudaGetLastError());
  }
  k_max_wdeg<<<blocks_for((int64_t)n * 32), kTPB, 0, st>>>(n, G->rowptr.as<int64_t>(), G->adj.as<int2>(), d_sum,
                                                            G->wrange.as<int2>());
  TS_CUDA(cudaGetLastError());
  auto fill = [&](int64_t count, const unsigned long long* sorted) -> ts_status {
    if (bitset) {
      TS_CUDA(cudaMemsetAsync(G->bits.p, 0, G->bits.bytes, st));
      if (count > 0) {
        k_fill_bits<<<blocks_for(count), kTPB, 0, st>>>(n, cb, count, sorted, G->rowptr.as<int64_t>(), G->adj.as<int2>(),
                                                        G->wpr, G->bits.as<unsigned long long>());
        TS_CUDA(cudaGetLastError());
      }
    }
    if (G->kind == TS_STRUCT_CSR && count > 0) {
      k_reverse_index<<<blocks_for(count), kTPB, 0, st>>>(n, cb, count, sorted, G->rowptr.as<int64_t>(),
                                                          G->adj.as<int2>(), G->rev.as<int64_t>());
      TS_CUDA(cudaGetLastError());
    }
    return TS_OK;
  };
  if (!later && (s = fill(N2, dk.Current())) != TS_OK) return s;
  int64_t slots = 0;
  if (hash) {
    k_hash_caps<<<blocks_for(n), kTPB, 0, st>>>(n, G->rowptr.as<int64_t>(), caps.as<int64_t>());
    TS_CUDA(cudaGetLastError());
    TS_CUDA(cub::DeviceScan::ExclusiveSum(tmp.p, scan_bytes, caps.as<int64_t>(), G->hoff.as<int64_t>(), n + 1, st));
    TS_CUDA(cudaMemcpyAsync(&slots, G->hoff.as<int64_t>() + n, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  }
  G->h_rowptr.resize(n + 1);
  unsigned long long got[4] = {0, 0, 0, 0};
  TS_CUDA(cudaMemcpyAsync(G->h_rowptr.data(), G->rowptr.p, sizeof(int64_t) * (n + 1), cudaMemcpyDeviceToHost, st));
  TS_CUDA(cudaMemcpyAsync(got, d_sum, sizeof(got), cudaMemcpyDeviceToHost, st));
  TS_CUDA(cudaStreamSynchronize(st));
  if ((int32_t)got[3] & E_BAD_EDGE) {
    set_error("ts_graph_create: edge endpoint outside [0, n)");
    return TS_ERR_INVALID_ARG;
  }
  const int64_t N = G->h_rowptr[n];
  G->entries = N;
  G->num_edges = N / 2;
  G->max_wdeg = (int64_t)got[0];
  G->neg_w = got[1] != 0;
  G->max_abs_w = (int64_t)got[2];
  if (hash) {
    G->hash_slots = slots;
    auto tables = [&] {
      G->tables.add(G->hkey, sizeof(int32_t) * slots);
      G->tables.add(G->hval, sizeof(int32_t) * slots);
      G->tables.add(full, sizeof(int32_t));
      return G->tables.alloc("alloc hash tables");
    };
    const unsigned long long* sorted = dk.Current();
    s = tables();
    if (s == TS_ERR_OUT_OF_MEMORY) {
      temp.reset();
      sorted = nullptr;
      s = tables();
    }
    if (s != TS_OK) return s;
    TS_CUDA(cudaMemsetAsync(G->hkey.p, 0xff, G->hkey.bytes, st));  // kHashEmpty
    TS_CUDA(cudaMemsetAsync(G->hval.p, 0, G->hval.bytes, st));
    TS_CUDA(cudaMemsetAsync(full.p, 0, full.bytes, st));
    if (N > 0) {
      k_hash_insert<<<blocks_for(N), kTPB, 0, st>>>(n, cb, N, sorted, G->rowptr.as<int64_t>(), G->adj.as<int2>(),
                                                    G->hoff.as<int64_t>(), G->hkey.as<int32_t>(),
                                                    G->hval.as<int32_t>(), full.as<int32_t>());
      TS_CUDA(cudaGetLastError());
    }
    int32_t err = 0;
    TS_CUDA(cudaMemcpyAsync(&err, full.p, sizeof(err), cudaMemcpyDeviceToHost, st));
    TS_CUDA(cudaStreamSynchronize(st));
    if (err & E_HASH_FULL) {
      set_error("ts_graph_create: hash table overflow");
      return TS_ERR_DEVICE;
    }
  }
  if (later) {
    temp.reset();
    filled(G->tables);
    if ((s = G->tables.alloc("alloc graph")) != TS_OK) return s;
    if ((s = fill(N, nullptr)) != TS_OK) return s;
    TS_CUDA(cudaStreamSynchronize(st));
  }
  return TS_OK;
}

}  // namespace tsb

using namespace tsb;

static ts_status make_graph(int32_t n, int64_t E, const int32_t* u, const int32_t* v, const int32_t* w, int32_t kind,
                            int32_t drop, void* stream, bool on_host, ts_graph** out) {
  if (!out) { set_error("ts_graph_create: out is NULL"); return TS_ERR_INVALID_ARG; }
  *out = nullptr;
  if (on_host && (E < 0 || (E > 0 && (!u || !v || !w)))) {
    set_error("ts_graph_create: bad edge arrays");
    return TS_ERR_INVALID_ARG;
  }
  int ndev = 0;
  if (on_host && (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)) {
    cudaGetLastError();
    set_error("no CUDA device visible");
    return TS_ERR_NO_DEVICE;
  }
  if (n < 2 || E < 0 || kind < 0 || kind >= TS_STRUCT_COUNT) {
    set_error("ts_graph_create: need n >= 2, num_edges >= 0 and a valid structure");
    return TS_ERR_INVALID_ARG;
  }
  if (E > 0 && (!u || !v || !w)) { set_error("ts_graph_create: NULL edge array"); return TS_ERR_INVALID_ARG; }
  if (!on_host && (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)) {
    cudaGetLastError();
    set_error("no CUDA device visible");
    return TS_ERR_NO_DEVICE;
  }
  auto* G = new ts_graph;
  G->n = n;
  G->kind = kind;
  G->drop_self_loops = drop ? 1 : 0;
  G->stream = (cudaStream_t)stream;
  cudaGetDevice(&G->device);
  ts_status s = build_graph(G, E, u, v, w, on_host);
  if (s != TS_OK) { delete G; return s; }
  G->pool = pool_enter();
  *out = G;
  return TS_OK;
}

extern "C" {

int32_t ts_abi_version(void) { return TS_ABI_VERSION; }

const char* ts_status_string(ts_status s) {
  switch (s) {
    case TS_OK: return "ok";
    case TS_ERR_INVALID_ARG: return "invalid argument";
    case TS_ERR_CUDA: return "CUDA error";
    case TS_ERR_OUT_OF_MEMORY: return "out of device memory";
    case TS_ERR_UNSUPPORTED: return "unsupported";
    case TS_ERR_DEVICE: return "device-side error";
    case TS_ERR_STATE: return "invalid call order";
    case TS_ERR_NO_DEVICE: return "no CUDA device";
  }
  return "unknown status";
}

const char* ts_last_error(void) { return tsb::last_error(); }

static const char* kNames[TS_STRUCT_COUNT] = {"csr", "hash", "wswap", "csr-bitset", "csr-bb", "csr-bitset-bb"};

int32_t ts_struct_from_name(const char* name) {
  if (!name) return -1;
  for (int i = 0; i < TS_STRUCT_COUNT; i++)
    if (std::strcmp(name, kNames[i]) == 0) return i;
  return -1;
}

const char* ts_struct_name(int32_t kind) {
  return (kind >= 0 && kind < TS_STRUCT_COUNT) ? kNames[kind] : "unknown";
}

ts_status ts_graph_create_device(int32_t n, int64_t num_edges, const int32_t* d_u, const int32_t* d_v,
                                 const int32_t* d_w, int32_t kind, int32_t drop_self_loops,
                                 void* stream, ts_graph** out) {
  tsb::TraceRange tr_("ts_graph_create_device");
  return make_graph(n, num_edges, d_u, d_v, d_w, kind, drop_self_loops, stream, false, out);
}

ts_status ts_graph_create(int32_t n, int64_t num_edges, const int32_t* u, const int32_t* v,
                          const int32_t* w, int32_t kind, int32_t drop_self_loops, void* stream,
                          ts_graph** out) {
  tsb::TraceRange tr_("ts_graph_create");
  return make_graph(n, num_edges, u, v, w, kind, drop_self_loops, stream, true, out);
}

ts_status ts_graph_info_get(const ts_graph* g, ts_graph_info* out) {
  if (!g || !out) { set_error("ts_graph_info_get: NULL argument"); return TS_ERR_INVALID_ARG; }
  std::memset(out, 0, sizeof(*out));
  out->n = g->n;
  out->kind = g->kind;
  out->num_edges = g->num_edges;
  out->num_entries = g->entries;
  out->max_weighted_degree = g->max_wdeg;
  out->device_bytes = g->device_bytes();
  out->hash_slots = g->hash_slots;
  out->bitset_words_per_row = g->wpr;
  return TS_OK;
}

ts_status ts_graph_destroy(ts_graph* g) {
  if (!g) return TS_OK;
  cudaSetDevice(g->device);
  cudaStreamSynchronize(g->stream);
  Pool* pool = g->pool;
  delete g;
  pool_leave(pool);
  cudaGetLastError();  // a context that ended before its graph: no error for the next call to find
  return TS_OK;
}

ts_status ts_lookup(const ts_graph* g, int64_t count, const int32_t* d_u, const int32_t* d_v,
                    int32_t* d_w_out) {
  tsb::TraceRange tr_("ts_lookup");
  if (!g || count < 0 || (count > 0 && (!d_u || !d_v || !d_w_out))) {
    set_error("ts_lookup: bad argument");
    return TS_ERR_INVALID_ARG;
  }
  if (count == 0) return TS_OK;
  TS_CUDA(cudaSetDevice(g->device));
  int64_t b = (count + 255) / 256;
  if (b > 148 * 64) b = 148 * 64;
  k_lookup<<<(int)b, 256, 0, g->stream>>>(g->dev(), count, d_u, d_v, d_w_out);
  TS_CUDA(cudaGetLastError());
  return TS_OK;
}

ts_status ts_lookup_host(const ts_graph* g, int64_t count, const int32_t* u, const int32_t* v,
                         int32_t* w_out) {
  if (!g || count < 0 || (count > 0 && (!u || !v || !w_out))) {
    set_error("ts_lookup_host: bad argument");
    return TS_ERR_INVALID_ARG;
  }
  if (count == 0) return TS_OK;
  TS_CUDA(cudaSetDevice(g->device));
  DevParts mem;
  DevPart a, b, c;
  size_t bytes = sizeof(int32_t) * (size_t)count;
  ts_status s;
  mem.add(a, bytes);
  mem.add(b, bytes);
  mem.add(c, bytes);
  if ((s = mem.alloc_temp("alloc lookup", g->stream)) != TS_OK) return s;
  TS_CUDA(cudaMemcpyAsync(a.p, u, bytes, cudaMemcpyHostToDevice, g->stream));
  TS_CUDA(cudaMemcpyAsync(b.p, v, bytes, cudaMemcpyHostToDevice, g->stream));
  s = ts_lookup(g, count, a.as<int32_t>(), b.as<int32_t>(), c.as<int32_t>());
  if (s != TS_OK) return s;
  TS_CUDA(cudaMemcpyAsync(w_out, c.p, bytes, cudaMemcpyDeviceToHost, g->stream));
  TS_CUDA(cudaStreamSynchronize(g->stream));
  return TS_OK;
}

}  // extern "C"
