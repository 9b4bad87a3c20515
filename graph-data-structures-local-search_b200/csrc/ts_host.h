// ts_host.h -- host-side objects behind the C-ABI handles.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <memory>
#include <random>
#include <string>
#include <utility>
#include <vector>

#include <nvtx3/nvToolsExt.h>

#include "ts_b200.h"
#include "ts_internal.cuh"

namespace tsb {

// Names the span of a C-ABI call on a profiler's timeline (NVTX range: ncu
// --nvtx filters, Nsight Systems); a no-op unless a tool is attached.
struct TraceRange {
  explicit TraceRange(const char* name) { nvtxRangePushA(name); }
  ~TraceRange() { nvtxRangePop(); }
  TraceRange(const TraceRange&) = delete;
  TraceRange& operator=(const TraceRange&) = delete;
};

// Thread-local message of the last failing call.
void set_error(const std::string& msg);
const char* last_error();

// Records the failure and returns TS_ERR_CUDA (or TS_ERR_OUT_OF_MEMORY).
ts_status cuda_fail(cudaError_t e, const char* what);

#define TS_CUDA(call)                                     \
  do {                                                    \
    cudaError_t e_ = (call);                              \
    if (e_ != cudaSuccess) return ::tsb::cuda_fail(e_, #call); \
  } while (0)

// Identity of the context current on the calling thread (the device's primary
// context if none is); 0 when the driver does not tell.  Unlike the context's
// address it does not come back after a device reset.
uint64_t context_id();

// Device memory of graphs, solvers and calls comes from a memory pool of the
// library's own per context: outside a pool an allocation or free of megabytes
// costs 50 us to milliseconds and stalls every stream (ER n = 2,000: graph
// 650 -> 150 us, its and its solver's end 450 -> 30 us).  The pool keeps at
// most kPoolKeep unused bytes, kPoolIdle once the last graph is gone, and
// gives them back before an allocation of the library fails.  Blocks above
// kPoolBlock that outlive a call are plain allocations: the pool grows and
// shrinks by many small mappings (a matrix of 1.8 GB: 10 ms and more, 0.5 ms
// plain).
constexpr size_t kPoolKeep = 512u << 20;
constexpr size_t kPoolIdle = 256u << 20;
constexpr size_t kPoolBlock = 64u << 20;
struct Pool;
struct PoolBlock {
  void* p = nullptr;
  uint64_t ctx = 0;      // the context it lives in
  Pool* pool = nullptr;  // null: a plain allocation
  bool ordered = false;  // for work on `stream` alone, freed in its order
  cudaStream_t stream = nullptr;
};
// ordered: for work on `st` alone (temporaries of one call); else for any
// stream: ready on return, and pool_put waits for the device, as a plain free
// does.
cudaError_t pool_get(PoolBlock& b, size_t bytes, bool ordered, cudaStream_t st);
void pool_put(PoolBlock& b);
void pool_trim();           // current context: unused bytes back to the driver
Pool* pool_enter();         // a graph begins: the current context's pool
void pool_leave(Pool* pool);  // and ends

// Owning device buffer.
struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  ~DevBuf() { release(); }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
  }
  ts_status alloc(size_t nbytes, const char* what) {
    release();
    if (nbytes == 0) nbytes = 16;
    cudaError_t e = cudaMalloc(&p, nbytes);
    if (e == cudaErrorMemoryAllocation) {
      cudaGetLastError();
      pool_trim();
      e = cudaMalloc(&p, nbytes);
    }
    if (e != cudaSuccess) {
      p = nullptr;
      return cuda_fail(e, what);
    }
    bytes = nbytes;
    return TS_OK;
  }
  template <class T> T* as() const { return static_cast<T*>(p); }
};

// Part of a device allocation that something else owns.
struct DevPart {
  void* p = nullptr;
  size_t bytes = 0;
  template <class T> T* as() const { return static_cast<T*>(p); }
};
// Parts of one pool allocation: sizes are registered first, then placed
// together (every part starts on 256 bytes).
struct DevParts {
  PoolBlock mem;
  std::vector<std::pair<DevPart*, size_t>> parts;
  DevParts() = default;
  DevParts(const DevParts&) = delete;
  DevParts& operator=(const DevParts&) = delete;
  ~DevParts() { pool_put(mem); }
  void add(DevPart& part, size_t n) {
    part.bytes = n;
    parts.emplace_back(&part, n);
  }
  // For any stream, until the object goes.
  ts_status alloc(const char* what) { return place(what, false, nullptr); }
  // For work on `st` alone.
  ts_status alloc_temp(const char* what, cudaStream_t st) { return place(what, true, st); }

 private:
  ts_status place(const char* what, bool ordered, cudaStream_t st) {
    auto pad = [](size_t b) { return b ? (b + 255) & ~(size_t)255 : (size_t)256; };
    size_t bytes = 0;
    for (auto& x : parts) bytes += pad(x.second);
    const cudaError_t e = pool_get(mem, bytes, ordered, st);
    if (e != cudaSuccess) {
      parts.clear();
      return cuda_fail(e, what);
    }
    unsigned char* p = static_cast<unsigned char*>(mem.p);
    for (auto& x : parts) {
      x.first->p = p;
      p += pad(x.second);
    }
    parts.clear();
    return TS_OK;
  }
};

}  // namespace tsb

struct ts_graph {
  int32_t n = 0;
  int32_t kind = 0;
  int32_t drop_self_loops = 0;
  int32_t device = 0;
  cudaStream_t stream = nullptr;
  int64_t num_edges = 0;
  int64_t entries = 0;
  int64_t max_wdeg = 0;
  bool neg_w = false;  // some edge weight is negative
  int64_t max_abs_w = 0;  // largest |w| of an entry
  int64_t wpr = 0;
  int64_t hash_slots = 0;
  tsb::Pool* pool = nullptr;  // entered by the graph
  tsb::DevParts mem, tables;  // what is known before the sort; the hash tables, or what had to wait for room
  tsb::DevPart rowptr, adj, bits, hoff, hkey, hval, rev, wrange;
  // Host copy of the CSR row pointers/degrees (for footprint planning and the
  // solver's staging budgets); small: n+1 int64.
  std::vector<int64_t> h_rowptr;
  tsb::DevGraph dev() const {
    tsb::DevGraph g;
    g.n = n;
    g.kind = kind;
    g.entries = entries;
    g.rowptr = rowptr.as<int64_t>();
    g.adj = adj.as<int2>();
    g.bits = bits.as<uint64_t>();
    g.wpr = wpr;
    g.hoff = hoff.as<int64_t>();
    g.hkey = hkey.as<int32_t>();
    g.hval = hval.as<int32_t>();
    g.rev = rev.as<int64_t>();
    g.wrange = wrange.as<int2>();
    return g;
  }
  int64_t device_bytes() const {
    return (int64_t)(rowptr.bytes + adj.bytes + bits.bytes + hoff.bytes + hkey.bytes + hval.bytes + rev.bytes + wrange.bytes);
  }
  mutable int64_t max_degree = -1;  // computed on first use
  mutable int64_t deg90 = -1;  // 90th-percentile degree, computed on first use
};

namespace tsb {

// Shared by the plain solver and the batched form (solver.cu).
// Reference-compatible random streams: the MDP start (srand/rand rejection),
// the MaxBS shuffle partition (side0[v] = 1: part 0) and one perturbation
// event of k distinct flat move indices.
void mdp_random_set(int32_t n, int32_t m, uint32_t seed, std::vector<int32_t>& ids);
void maxbs_random_part(std::mt19937& rng, int32_t n, std::vector<uint8_t>& side0);
void draw_event(std::mt19937& rng, int64_t P, int k, std::vector<long long>& out);
// Dynamic shared memory for staging R rows of a lookup structure (the pass
// with per-row registers).
int32_t staging_bytes(const ts_graph* g, int R);

// Tile shape of a solve, shared by the plain and the persistent (batched,
// served; `persist`: 256-thread CTAs) forms: rows per tile, whether the fast pass runs (32-bit keys) and its index capacity,
// the CSR adjacency mask, column chunks (a multiple of one pass of the CTA, at
// least `min_tiles` tiles where the columns allow) and the dynamic shared
// memory one tile needs.
struct TileGeom {
  int32_t rows = 0, n_row_blocks = 0, chunk_cols = 0, n_chunks = 0;
  int32_t fast = 0, fast_ecap = 0, adj_mask = 0, stage_bytes = 0;
  size_t smem = 16;
};
TileGeom tile_geometry(const ts_graph* g, int32_t problem, int32_t m, bool wide, int64_t min_tiles,
                       int32_t pass, bool persist);
// WSwap: the matrix holds 16-bit weights when every |w| fits (the patch of a
// move clears and sets elements, so an element only ever holds one weight).
bool wswap_w16(const ts_graph* g);
// Opts kernel `fn` in to `smem` bytes of dynamic shared memory on the current
// device.  The limit only grows (under a lock), so a launch planned earlier
// with a larger size stays valid when a smaller one is planned later.
cudaError_t allow_dyn_smem(const void* fn, size_t smem);

// A round of a served solve.  begin admits up to k iterations and launches them,
// after the event `before` (null: none).  next waits for the launches, says how
// many iterations the round has made, and, where the candidate pass left one to
// the sweeps (which take many times longer) and go_on is set, launches what comes
// next.  Unlike ts_solver_sync it need not complete them.
ts_status solver_round_begin(ts_solver* s, int64_t k, int64_t* admitted, cudaEvent_t before);
ts_status solver_round_next(ts_solver* s, bool go_on, bool* running, int64_t* advanced);

}  // namespace tsb
