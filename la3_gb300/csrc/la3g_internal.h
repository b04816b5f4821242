// Internal declarations shared by the library's translation units.
#ifndef LA3G_INTERNAL_H
#define LA3G_INTERNAL_H

#include <cstdint>
#include <cstdio>
#include <new>
#include <string>
#include <utility>
#include <vector>

#include "la3g.h"

#ifdef __CUDACC__
#include <cuda_runtime.h>
#endif

namespace la3g {

// Records `code` and a printf-style message as the thread's last error and
// returns `code`.
int set_error(int code, const char* fmt, ...) __attribute__((format(printf, 2, 3)));
unsigned host_threads();

// Hashing of vertex ids: SimpleBucketHasher at one rank
// (src/matrix/hashers.h:39-68) or the identity (NullHasher) for bipartite
// graphs.
struct Hasher
{
  uint64_t height = 0, max_range = 0;
  bool null_hash = false;
#ifdef __CUDACC__
  __host__ __device__
#endif
  inline uint32_t hash(uint64_t v) const
  {
    if (null_hash || v >= max_range) return (uint32_t) v;
    return (uint32_t) (v / 128u + ((uint32_t) v % 128u) * height);
  }
#ifdef __CUDACC__
  __host__ __device__
#endif
  inline uint32_t unhash(uint64_t v) const
  {
    if (null_hash || v >= max_range) return (uint32_t) v;
    return (uint32_t) (v / height + (v % height) * 128u);
  }
};

}  // namespace la3g

#ifdef __CUDACC__

namespace la3g {

#define LA3G_CUDA(call)                                                                         \
  do {                                                                                          \
    cudaError_t err_ = (call);                                                                  \
    if (err_ != cudaSuccess)                                                                    \
      return ::la3g::set_error(LA3G_ECUDA, "%s:%d %s: %s", __FILE__, __LINE__, #call,           \
                               cudaGetErrorString(err_));                                       \
  } while (0)

#define LA3G_TRY(expr)                \
  do {                                \
    int rc_ = (expr);                 \
    if (rc_ != LA3G_OK) return rc_;   \
  } while (0)

// Checks the launch that was just made (configuration errors only; the
// kernel itself is checked at the next synchronisation).
#define LA3G_LAUNCHED() LA3G_CUDA(cudaGetLastError())

// Streaming multiprocessors of the current device (152 on a GB300: 2 dies
// x 76), queried once per device; grid sizes are multiples of it.
int num_sms();

inline unsigned grid_for(uint64_t n, unsigned block, unsigned max_blocks = num_sms() * 16)
{
  uint64_t g = (n + block - 1) / block;
  if (g < 1) g = 1;
  if (g > max_blocks) g = max_blocks;
  return (unsigned) g;
}

// Block-wide reductions for kernels that add their partial counts into one
// global counter: one atomic per block instead of one per warp (thousands of
// same-address atomics serialise in L2).  Every thread of the block must
// call them; the result is valid in thread 0.
__device__ __forceinline__ unsigned long long block_sum_u64(unsigned long long v)
{
  __shared__ unsigned long long s_part[32];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();  // s_part may still be read from a previous call
  if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32)
  {
    v = threadIdx.x < (blockDim.x + 31) / 32 ? s_part[threadIdx.x] : 0ull;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  }
  return v;
}

__device__ __forceinline__ uint32_t block_min_u32(uint32_t v)
{
  __shared__ uint32_t s_part[32];
  for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32)
  {
    v = threadIdx.x < (blockDim.x + 31) / 32 ? s_part[threadIdx.x] : 0xFFFFFFFFu;
    for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
  }
  return v;
}

// Barrier over the blocks of a cooperative launch.  `count` starts at zero and
// takes 2 per arrival (it may wrap).  A block that waits more than `limit` polls
// gives up: sync() returns false in all its threads, which then leave the
// kernel, and so does every other block's.  A barrier is passed by every block or
// by none, so that what lies between two of them is done whole or the kernel does
// not get past it: giving up sets the count's bit 0, only while the count is
// below the barrier's target.  No block then gets to the next barrier, so a count
// above the target, which only blocks at the next one can have made, says that
// the bit was set there.  (A 64-bit count took 0.3 us more a barrier.)
// Every thread of every block calls sync() the same number of times.  Like
// cooperative groups' grid barrier it is a fence at device scope, after which
// ordinary loads see what the other blocks wrote before it.
struct GridBarrier
{
  unsigned int* count;
  long long limit;
  unsigned int target = 0;
  __device__ bool sync()
  {
    __shared__ int s_ok;
    target += 2 * gridDim.x;
    __syncthreads();
    if (threadIdx.x == 0)
    {
      __threadfence();
      atomicAdd(count, 2u);
      volatile unsigned int* c = count;
      long long left = limit;
      unsigned int x;
      int ok = 1;
      while ((int) ((x = *c) - target) < 0 || (x & 1u))  // not all here, or one gave up
      {
        if (x & 1u)
        {
          ok = (int) ((x & ~1u) - target) > 0;
          break;
        }
        if (--left < 0 && atomicCAS(count, x, x | 1u) == x)
        {
          ok = 0;
          break;
        }
      }
      __threadfence();
      s_ok = ok;
    }
    __syncthreads();
    return s_ok;
  }
};

// Polls of a barrier before it gives up, by default: 2^26 (ten seconds; a poll
// takes 0.15 us) and kEntryPolls for each entry of the matrix, since a lane may
// walk a whole list between two barriers (the neighbours of a vertex in a
// bottom-up level, a sink's in-edges: 0.05 and 0.14 us an entry out of L2; eight
// polls leave room for reads that miss it): work that is only long is waited for.
static constexpr long long kBarrierPolls = 1ll << 26, kEntryPolls = 8;
__host__ __device__ inline long long barrier_polls(long long set, uint64_t entries)
{
  return set < 0 ? kBarrierPolls + kEntryPolls * (long long) entries : set;
}

// Blocks of a cooperative launch of `f`: enough for `want` threads, at most
// as many as are resident at once (and max_per_sm per SM).
int cooperative_blocks(const void* f, int threads, uint64_t want, int max_per_sm, unsigned* out);

// Kernel-level profiling: when on, a launch is bracketed by events on its
// stream and its time accumulated under `name` with `bytes` algorithmic
// bytes.  Always counts the launch.
struct ProfileScope
{
  const char* name;
  cudaStream_t stream;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  double bytes;
  ProfileScope(const char* name, cudaStream_t s, double bytes);
  ~ProfileScope();
};

// Adds algorithmic bytes to a kernel's profile entry when they are known
// only after its launches (e.g. from a count the kernels produced).
void profile_add_bytes(const char* name, double bytes);

extern thread_local uint32_t tls_launches;

// cudaMalloc, or LA3G_ENOMEM (also as la3g_fail_allocation asks).
int device_alloc(void** p, size_t bytes);

// Scoped device buffer for temporaries.
struct DevBuf
{
  void* p = nullptr;
  size_t bytes = 0;
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  ~DevBuf() { if (p) cudaFree(p); }
  int alloc(size_t n)
  {
    if (n <= bytes && p) return LA3G_OK;
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
    LA3G_TRY(device_alloc(&p, n));
    bytes = n;
    return LA3G_OK;
  }
  template <class T>
  T* as() const { return (T*) p; }
};

// The device image of a graph in internal order.
struct DevGraph
{
  uint32_t flags = 0;
  uint32_t nvertices = 0, nslots = 0, nleft = 0;
  uint64_t nrecords = 0, nent = 0;
  uint32_t nreg = 0, nsink = 0, nsrc = 0;
  Hasher hasher;
  bool directed() const { return flags & LA3G_DIRECTED; }
  bool weighted() const { return flags & LA3G_WEIGHTED; }
  uint32_t src_base() const { return nreg + nsink; }
  uint32_t iso_base() const { return nreg + nsink + nsrc; }
  uint32_t nrows() const { return nreg + nsink; }

  uint32_t* id_of_pos = nullptr;    // [nslots] original id of each position
  uint32_t* pos_of_id = nullptr;    // [nslots]
  uint32_t* hash_of_pos = nullptr;  // [nslots] hashed id (Edge::src / Edge::dst)

  // Pull CSR over rows = positions [0, nreg + nsink): in-neighbours (column
  // positions) in the reference's order: source columns first, then regular
  // columns, each ascending.  For undirected graphs this is the only CSR.
  uint32_t* in_ptr = nullptr;  // [nslots + 1]
  uint32_t* in_col = nullptr;  // [nent]
  uint32_t* in_w = nullptr;    // [nent] when weighted

  // Push CSR over columns = positions: out-neighbours (row positions),
  // ascending, so regular rows come before sink rows.  Built on demand for
  // directed graphs; the same arrays as the pull CSR for undirected graphs.
  uint32_t* out_ptr = nullptr;  // [nslots + 1]
  uint32_t* out_row = nullptr;
  uint32_t* out_w = nullptr;
};

// Per-app device scratch cached on a graph handle (allocated on first use).
enum AppSlot { kSlotPr = 0, kSlotBfs, kSlotSssp, kSlotCc, kSlotTc, kSlotBm25, kSlotBatch, kSlotVp, kSlotLm, kSlotCount };

}  // namespace la3g

struct la3g_graph
{
  la3g::DevGraph g;
  cudaStream_t stream = nullptr;       // stream the calls run on
  cudaStream_t own_stream = nullptr;   // the graph's own stream
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  long long wait_polls = -1;           // la3g_set_wait_limit; < 0: the default
  std::vector<std::pair<void*, uint64_t>> allocations;  // and their bytes
  uint64_t device_bytes = 0;
  void* slot[la3g::kSlotCount] = {};
  void (*slot_free[la3g::kSlotCount])(void*) = {};
};

namespace la3g {

// Graph-owned device allocation (freed by la3g_graph_free).
int galloc_bytes(la3g_graph* G, void** p, size_t bytes);
template <class T>
int galloc(la3g_graph* G, T** p, size_t count)
{
  return galloc_bytes(G, (void**) p, count * sizeof(T));
}

// Graph allocations made while it lives are released again unless keep() is
// called: what is built in several allocations stands whole or not at all.
struct GallocScope
{
  la3g_graph* G;
  size_t from;
  bool kept = false;
  explicit GallocScope(la3g_graph* G_) : G(G_), from(G_->allocations.size()) {}
  GallocScope(const GallocScope&) = delete;
  GallocScope& operator=(const GallocScope&) = delete;
  ~GallocScope();
  int keep()
  {
    kept = true;
    return LA3G_OK;
  }
};

// An app's scratch on the graph, made by build(scratch) on first use.  It is put
// in its slot only when it is complete: a call after a failed one builds it anew.
template <class S, class Build>
int graph_scratch(la3g_graph* G, AppSlot slot, void (*free_scratch)(void*), S** out, Build build)
{
  if (!G->slot[slot])
  {
    S* s = new (std::nothrow) S();
    if (!s) return set_error(LA3G_ENOMEM, "out of host memory");
    GallocScope scope(G);
    const int rc = build(s);
    if (rc != LA3G_OK)
    {
      cudaStreamSynchronize(G->stream);  // kernels that write to it
      free_scratch(s);
      return rc;
    }
    scope.keep();
    G->slot[slot] = s;
    G->slot_free[slot] = free_scratch;
  }
  *out = (S*) G->slot[slot];
  return LA3G_OK;
}

// Releases a graph allocation that another one replaces (null: nothing).
void galloc_release(la3g_graph* G, void* p);

int build_push_csr(la3g_graph* G);
// la3g_sssp; order: if they are not there yet, the in-edges are first ordered for
// its pull steps (sssp.cu).
int sssp_run(la3g_graph* G, uint32_t root, uint32_t* dist_out, la3g_stats* st, bool order);
// Bipartite corpus: the position of the first term row (docs come first).
int bipartite_first_term_row(la3g_graph* G, uint32_t* out);

// Bracket an app call: events on the graph's stream and the host clock.
struct CallTimer
{
  la3g_graph* G;
  la3g_stats* st;
  double t0;
  uint32_t launches0;
  CallTimer(la3g_graph* G, la3g_stats* st);
  void device_begin();
  void device_end();
  int finish();  // synchronises and fills st
};

double now_ms();

}  // namespace la3g

#endif  // __CUDACC__

#endif
