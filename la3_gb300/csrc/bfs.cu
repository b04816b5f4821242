// BFS: the reference bfs app (src/apps/graph_analytics/bfs.cpp:11-37,
// bfs.h:11-49) on the device, direction-optimising.
//
// Reference semantics kept exactly (np = 1):
//   * hops are uint8 with 255 = unvisited; apply at iteration i sets
//     hops = (uint8)(i + 1) on a touched vertex whose hops are 255
//     (bfs.h:41-48); the loop stops after the first iteration that activates
//     nothing (execute_non_opt, vertex_program_execute.hpp:166-248);
//   * parent: gather returns edge.src (the hashed id of the column) and
//     combine keeps the last value written (bfs.h:39-40).  The SpMV walks the
//     active columns in ascending position = ascending hashed id, so the
//     last writer of a row is its frontier neighbour with the LARGEST hashed
//     id.  Top-down keeps it with atomicMax; bottom-up scans a vertex's
//     neighbours from the highest position down and stops at the first one
//     in the frontier, which is that same neighbour.
//
// Direction switching follows Beamer et al. (alpha = 14, beta = 24): go
// bottom-up when the frontier's edges exceed the unvisited edges / alpha,
// back top-down when the frontier holds fewer than n / beta vertices.
//
// All levels run in one cooperative kernel, the direction decided by every
// block for itself from counters in global memory, one grid barrier per level
// (one more where the frontier changes form).  A host- or graph-driven loop
// spent its time between the kernels: 10 us a level on a graph whose levels
// take 3 us of work.
#include <algorithm>
#include <cstring>

#include "frontier.cuh"
#include "la3g_internal.h"

namespace la3g {

// A frontier is kept as two lists, vertices of degree <= kBigDeg ("small",
// one warp each) and hubs ("big", whose edges the whole grid shares), so that
// no warp serialises on a hub; both sit in one array, small from the front,
// hubs from the back.
struct FrontierCounters
{
  unsigned long long raw;      // vertices found by a bottom-up level
  unsigned long long degsum;   // degrees of the next frontier
  unsigned long long nsmall;   // next frontier: small list length
  unsigned long long packed;   // next frontier: hub slots and hub tasks (frontier.cuh)
};

struct BfsStats  // written by the kernel at its end
{
  unsigned long long iterations, pulls, examined, status, reached_deg;
};

static constexpr unsigned long long kBfsRunning = 2;  // status until the kernel has ended properly

struct BfsArgs
{
  const uint32_t *ptr, *col, *key;  // CSR by position, rows ascending by key; key: hashed id
  uint32_t N, nrows;
  uint64_t nent, limit;  // entries (CHECK: read from ptr); most levels
  uint32_t root;
  uint8_t* hops;
  // [N] while the hops fit a byte (the first 254 levels): 0, or the parent's
  // key + 1 (bfs_code), which a level's visitors raise by atomicMax; later: a
  // level's candidate, moved to `parent` at its end
  uint32_t* cand;
  uint32_t* parent;                 // [N] later levels' parents
  uint32_t* list[2];                // [N] frontier lists
  uint32_t* task0;                  // [N] first task numbers of the hubs: even levels from the front, odd from the back
  uint32_t* bits[2];                // [N / 32 + 1] frontier bitmaps
  FrontierCounters* ctr;            // [3]
  unsigned int* bar;                // barrier count
  long long wait_polls;             // < 0: the default
  const uint32_t* pos_of_id;        // null: ids are positions
  uint8_t* hops_out;                // by id, or null
  uint32_t* parent_out;             // by id, or null
  BfsStats* stats;
};

static constexpr double kAlpha = 14.0, kBeta = 24.0;
static constexpr int kBfsThreads = 512;

__global__ void k_bfs_none(uint32_t N, uint8_t* hops, uint32_t* parent)
{
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < N; p += gridDim.x * blockDim.x)
  {
    if (hops) hops[p] = 255;
    if (parent) parent[p] = 0;
  }
}

// The hub lists of the level with parity c.
struct HubList
{
  uint32_t *big, *task0;  // slot k at big[-k], task0[k * dir]
  int dir;
  __device__ HubList(const BfsArgs& A, int c)
      : big(A.list[c] + (A.N - 1)), task0(c ? A.task0 + (A.N - 1) : A.task0), dir(c ? -1 : 1)
  {
  }
  __device__ void append(uint32_t v, uint32_t deg, unsigned long long* packed) const
  {
    const unsigned long long old = atomicAdd(packed, hub_pack_inc((deg + kHubTask - 1) / kHubTask));
    const int64_t slot = (int64_t) (old >> kHubSlotShift);
    big[-slot] = v;
    task0[slot * dir] = (uint32_t) (old & ((1ull << kHubSlotShift) - 1));
  }
  __device__ uint32_t of_task(uint32_t nbig, uint32_t t) const
  {
    uint32_t lo = 0, hi = nbig;
    while (hi - lo > 1)
    {
      const uint32_t mid = (lo + hi) >> 1;
      if (task0[(int64_t) mid * dir] <= t) lo = mid;
      else hi = mid;
    }
    return lo;
  }
};

__device__ __forceinline__ FrontierCounters bfs_counters(const FrontierCounters* c)
{
  return {__ldcg(&c->raw), __ldcg(&c->degsum), __ldcg(&c->nsmall), __ldcg(&c->packed)};
}

// A parent's key as cand holds it: above 0, ascending with the key.  A caller's
// keys (CHECK) may be any 32-bit numbers; the two largest share a code.
template <bool CHECK>
__device__ __forceinline__ uint32_t bfs_code(uint32_t key)
{
  return CHECK ? key + (key != 0xFFFFFFFFu) : key + 1;
}

// The key behind the code x of v, which was reached at `hop`: where two keys
// share it, the larger one if a neighbour with that key was in the frontier.
template <bool CHECK>
__device__ __forceinline__ uint32_t bfs_key_of(const BfsArgs& A, uint32_t v, uint32_t x, uint8_t hop)
{
  if (CHECK && x == 0xFFFFFFFFu)
    for (uint32_t i = A.ptr[v + 1]; i > A.ptr[v]; i--)
    {
      const uint32_t u = A.col[i - 1];
      if (u < A.N && A.key[u] == x && A.hops[u] == (uint8_t) (hop - 1)) return x;
    }
  return x - 1;
}

// CHECK: the CSR comes from the caller; neighbour ids outside the graph are
// skipped.
template <bool CHECK>
__global__ void __launch_bounds__(kBfsThreads, 3) k_bfs_run(BfsArgs A)
{
  __shared__ FrontierCounters s_next;
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
  const uint32_t lane = threadIdx.x & 31, warp = tid >> 5, nwarps = nth >> 5;
  const uint32_t words = (A.N + 31) / 32;
  const uint32_t rp = A.pos_of_id ? A.pos_of_id[A.root] : A.root;
  const uint64_t nent = CHECK ? A.ptr[A.N] : A.nent;
  GridBarrier bar{A.bar, barrier_polls(A.wait_polls, nent)};
  const uint32_t rdeg = rp < A.nrows ? A.ptr[rp + 1] - A.ptr[rp] : 0;

  // everything unvisited, the root at 0 and in the first frontier
  for (uint32_t p = tid; p < A.N; p += nth)
  {
    A.hops[p] = p == rp ? 0 : 255;
    A.cand[p] = 0;
  }
  for (uint32_t w = tid; w < words; w += nth) A.bits[0][w] = A.bits[1][w] = 0;
  if (tid == 0)
  {
    for (int k = 0; k < 3; k++) A.ctr[k] = FrontierCounters{0, 0, 0, 0};
    if (rdeg > kBigDeg)
    {
      const HubList H(A, 0);
      H.big[0] = rp;
      H.task0[0] = 0;
      A.ctr[0].packed = hub_pack_inc((rdeg + kHubTask - 1) / kHubTask);
    }
    else if (rdeg)
    {
      A.list[0][0] = rp;
      A.ctr[0].nsmall = 1;
    }
  }
  if (!bar.sync()) return;

  // the loop's state, the same in every thread
  unsigned long long iter = 0, pulls = 0, examined = 0;
  unsigned long long fdeg = rdeg, nfront = rdeg != 0, unv = nent - rdeg;
  uint32_t nsmall = rdeg && rdeg <= kBigDeg, nbig = rdeg > kBigDeg;
  uint32_t ntasks = nbig ? (rdeg + kHubTask - 1) / kHubTask : 0;
  bool bottom_up = false, in_list = true, wide = false, failed = false;  // wide: hops no longer fit a byte
  if (!nfront) iter = 1;
  while (nfront)
  {
    if (iter > A.limit)
    {
      failed = true;
      break;
    }
    // Beamer's test, as the reference counts: the frontier's degrees against
    // the unvisited ones', then its size against the graph's
    if (!bottom_up && (double) fdeg > (double) unv / kAlpha) bottom_up = true;
    else if (bottom_up && (double) nfront < (double) A.N / kBeta) bottom_up = false;
    const int c = (int) (iter & 1);
    FrontierCounters* const cur = A.ctr + iter % 3;
    FrontierCounters* const next = A.ctr + (iter + 1) % 3;
    if (tid == 0) A.ctr[(iter + 2) % 3] = FrontierCounters{0, 0, 0, 0};  // read last before the barrier just passed
    const uint8_t hop = (uint8_t) (iter + 1);
    if (!wide && iter + 1 >= 255)
    {
      // hop 255 is "unvisited" too, and later hops repeat earlier ones, so from
      // here on a level's vertices are marked only after all of its visits;
      // hubs go a warp each (their task numbers may lie in `parent`)
      wide = true;
      for (uint32_t p = tid; p < A.N; p += nth) A.parent[p] = 0;
      if (!bar.sync()) return;
    }
    if (!bottom_up && !in_list)
    {
      // bitmap -> lists; the bitmaps are left empty
      const HubList H(A, c);
      for (uint32_t w = tid; w < words; w += nth)
      {
        uint32_t x = A.bits[c][w];
        A.bits[c][w] = A.bits[c ^ 1][w] = 0;
        while (x)
        {
          const uint32_t v = w * 32 + (__ffs(x) - 1);
          x &= x - 1;
          const uint32_t d = A.ptr[v + 1] - A.ptr[v];
          if (d > kBigDeg && !wide) H.append(v, d, &cur->packed);
          else A.list[c][atomicAdd(&cur->nsmall, 1ull)] = v;
        }
      }
      if (!bar.sync()) return;
      if (threadIdx.x == 0) s_next = bfs_counters(cur);
      __syncthreads();
      nsmall = (uint32_t) s_next.nsmall;
      nbig = hub_count(s_next.packed);
      ntasks = hub_tasks(s_next.packed);
      in_list = true;
    }
    else if (bottom_up && in_list)
    {
      const HubList H(A, c);
      for (uint32_t i = tid; i < nsmall + nbig; i += nth)
      {
        const uint32_t v = i < nsmall ? A.list[c][i] : H.big[-(int64_t) (i - nsmall)];
        atomicOr(&A.bits[c][v >> 5], 1u << (v & 31));
      }
      if (!bar.sync()) return;
      in_list = false;
    }
    unsigned long long deg = 0;
    if (bottom_up)
    {
      pulls++;
      examined += unv;
      // a lane per vertex, a warp per word of the bitmap; neighbours from the
      // highest key down, four at a time, the first one in the frontier is
      // the parent
      const uint32_t* fbits = A.bits[c];
      uint32_t cnt = 0;
      for (uint32_t w = warp; w < words; w += nwarps)
      {
        const uint32_t v = w * 32 + lane;
        bool found = false;
        if (v < A.nrows && A.hops[v] == 255)
        {
          const uint32_t b = A.ptr[v], e = A.ptr[v + 1];
          uint32_t i = e;
          while (i > b && !found)
          {
            uint32_t u[4], from = 0;
            bool in[4];
#pragma unroll
            for (int k = 0; k < 4; k++)
            {
              in[k] = i - b > (uint32_t) k;
              u[k] = in[k] ? __ldg(&A.col[i - 1 - k]) : 0;
              if (CHECK) in[k] = in[k] && u[k] < A.N;
              if (CHECK && !in[k]) u[k] = 0;
            }
#pragma unroll
            for (int k = 0; k < 4; k++) in[k] = in[k] && (fbits[u[k] >> 5] >> (u[k] & 31) & 1);
#pragma unroll
            for (int k = 3; k >= 0; k--)
              if (in[k])
              {
                found = true;
                from = u[k];
              }
            if (found)
            {
              A.hops[v] = hop;
              if (wide) A.parent[v] = A.key[from];
              else A.cand[v] = bfs_code<CHECK>(A.key[from]);
              deg += e - b;
              cnt++;
            }
            i -= min(4u, i - b);
          }
        }
        const unsigned m = __ballot_sync(0xffffffffu, found);
        if (lane == 0) A.bits[c ^ 1][w] = m;
      }
      const unsigned long long total = block_sum_u64(cnt);
      if (threadIdx.x == 0 && total) atomicAdd(&next->raw, total);
    }
    else
    {
      examined += fdeg;
      // an edge's target that no earlier level has visited keeps the largest
      // key + 1; the first visitor marks it and appends it to the next frontier
      const HubList H(A, c), Hn(A, c ^ 1);
      auto visit = [&](uint32_t i, uint32_t e, uint32_t hu) {
        uint32_t v = 0, d = 0;
        bool add = false;
        if (i < e)
        {
          v = __ldg(&A.col[i]);
          if (!CHECK || v < A.N)
          {
            const uint8_t h = A.hops[v];
            if (h == 255 || (h == hop && !wide)) add = atomicMax(&A.cand[v], hu) == 0;
          }
        }
        bool small = add;
        if (add && !wide)
        {
          A.hops[v] = hop;
          d = A.ptr[v + 1] - A.ptr[v];
          deg += d;
          if (d > kBigDeg)
          {
            Hn.append(v, d, &next->packed);
            small = false;
          }
        }
        const unsigned m = __ballot_sync(0xffffffffu, small);
        if (m)
        {
          uint32_t base = 0;
          if (lane == 0) base = (uint32_t) atomicAdd(&next->nsmall, (unsigned long long) __popc(m));
          base = __shfl_sync(0xffffffffu, base, 0);
          if (small) A.list[c ^ 1][base + __popc(m & ((1u << lane) - 1))] = v;
        }
      };
      if (!wide)
        for (uint32_t t = warp; t < ntasks; t += nwarps)
        {
          const uint32_t slot = H.of_task(nbig, t), u = H.big[-(int64_t) slot], hu = bfs_code<CHECK>(A.key[u]);
          const uint32_t b = A.ptr[u] + (t - H.task0[(int64_t) slot * H.dir]) * kHubTask;
          const uint32_t e = min(b + kHubTask, A.ptr[u + 1]);
          for (uint32_t i0 = b; i0 < e; i0 += 32) visit(i0 + lane, e, hu);
        }
      for (uint32_t f = warp; f < nsmall + (wide ? nbig : 0); f += nwarps)
      {
        const uint32_t u = f < nsmall ? A.list[c][f] : H.big[-(int64_t) (f - nsmall)], hu = bfs_code<CHECK>(A.key[u]);
        const uint32_t b = A.ptr[u], e = A.ptr[u + 1];
        for (uint32_t i0 = b; i0 < e; i0 += 32) visit(i0 + lane, e, hu);
      }
      if (wide)
      {
        if (!bar.sync()) return;
        const uint32_t n = (uint32_t) __ldcg(&next->nsmall);
        for (uint32_t i = tid; i < n; i += nth)
        {
          const uint32_t v = A.list[c ^ 1][i];
          A.hops[v] = hop;
          A.parent[v] = bfs_key_of<CHECK>(A, v, A.cand[v], hop);
          A.cand[v] = 0;
          deg += A.ptr[v + 1] - A.ptr[v];
        }
      }
    }
    deg = block_sum_u64(deg);
    if (threadIdx.x == 0 && deg) atomicAdd(&next->degsum, deg);
    if (!bar.sync()) return;
    if (threadIdx.x == 0) s_next = bfs_counters(next);
    __syncthreads();
    nsmall = (uint32_t) s_next.nsmall;
    nbig = hub_count(s_next.packed);
    ntasks = hub_tasks(s_next.packed);
    fdeg = s_next.degsum;
    nfront = bottom_up ? s_next.raw : (unsigned long long) nsmall + nbig;
    unv -= min(unv, fdeg);
    iter++;
    __syncthreads();  // s_next is free
  }
  for (uint32_t i = tid; i < A.N; i += nth)
  {
    const uint32_t p = A.pos_of_id ? A.pos_of_id[i] : i;
    if (A.hops_out && A.hops_out != A.hops) A.hops_out[i] = A.hops[p];
    if (A.parent_out)
    {
      const uint32_t x = A.cand[p];
      A.parent_out[i] = x ? bfs_key_of<CHECK>(A, p, x, A.hops[p]) : wide ? A.parent[p] : 0;
    }
  }
  if (wide)
  {
    // a vertex may be visited again at hop 255: count the reached ones' degrees
    unsigned long long d = 0;
    for (uint32_t v = tid; v < A.nrows; v += nth)
      if (A.hops[v] != 255) d += A.ptr[v + 1] - A.ptr[v];
    d = block_sum_u64(d);
    if (tid == 0) A.ctr[0].degsum = 0;
    if (!bar.sync()) return;
    if (threadIdx.x == 0 && d) atomicAdd(&A.ctr[0].degsum, d);
    if (!bar.sync()) return;
    unv = nent - __ldcg(&A.ctr[0].degsum);
  }
  if (tid == 0 && A.stats) *A.stats = BfsStats{iter, pulls, examined, failed ? 1ull : 0ull, nent - unv};
}

template <bool CHECK>
static int bfs_launch(BfsArgs& A, unsigned* grid, cudaStream_t s)
{
  // few blocks for a small graph: a barrier takes longer the more there are
  if (!*grid) LA3G_TRY(cooperative_blocks((const void*) k_bfs_run<CHECK>, kBfsThreads, std::max<uint64_t>(A.N, A.nent / 8), 3, grid));
  LA3G_CUDA(cudaMemsetAsync(A.bar, 0, sizeof *A.bar, s));
  void* args[] = {(void*) &A};
  LA3G_CUDA(cudaLaunchCooperativeKernel((const void*) k_bfs_run<CHECK>, *grid, kBfsThreads, args, 0, s));
  return LA3G_OK;
}

// Up to this many vertices the kernel writes the outputs by id straight into
// pinned host memory, copied to the caller's once it has ended.  Two copies from
// the device take longer up to about twice this (R-MAT x 8, hops and parents: 2^12
// 79 us copied, 65 direct; 2^14 87 and 77; 2^16 155 and 154; 2^18 200 and 262).
static constexpr uint32_t kBfsDirect = 1u << 15;
static_assert(sizeof(BfsStats) <= 256, "the outputs start 256 bytes behind");

struct BfsScratch
{
  BfsArgs A{};
  BfsStats* stats = nullptr;   // pinned
  uint8_t* hops_id = nullptr;  // [nslots] outputs by id
  uint32_t* parent_id = nullptr;
  bool direct = false;         // they are in pinned host memory, behind stats
  unsigned grid = 0;
};

static void bfs_scratch_free(void* p)
{
  BfsScratch* s = (BfsScratch*) p;
  if (s->stats) cudaFreeHost(s->stats);
  delete s;
}

static int bfs_scratch_build(la3g_graph* G, BfsScratch* bs)
{
  DevGraph& g = G->g;
  const uint32_t N = g.nslots;
  // one allocation: six arrays of a word per vertex, two of a byte, two bitmaps
  auto round = [](size_t b) { return (b + 255) & ~(size_t) 255; };
  const size_t n4 = round((size_t) N * 4), n1 = round(N), nb = round(((size_t) N / 32 + 1) * 4);
  char* p = nullptr;
  LA3G_TRY(galloc(G, &p, 6 * n4 + 2 * n1 + 2 * nb + 512));
  auto take = [&](size_t b) { char* r = p; p += b; return r; };
  BfsArgs& A = bs->A;
  A.cand = (uint32_t*) take(n4);
  A.parent = (uint32_t*) take(n4);
  A.list[0] = (uint32_t*) take(n4);
  A.list[1] = (uint32_t*) take(n4);
  A.task0 = (uint32_t*) take(n4);
  bs->parent_id = (uint32_t*) take(n4);
  A.hops = (uint8_t*) take(n1);
  bs->hops_id = (uint8_t*) take(n1);
  A.bits[0] = (uint32_t*) take(nb);
  A.bits[1] = (uint32_t*) take(nb);
  A.ctr = (FrontierCounters*) take(256);
  A.bar = (unsigned int*) take(256);
  A.ptr = g.in_ptr;
  A.col = g.in_col;
  A.key = g.hash_of_pos;
  A.N = N;
  A.nrows = g.nrows();
  A.nent = g.nent;
  A.limit = (uint64_t) N + 2;  // every level visits at least one new vertex: more is a fault
  A.pos_of_id = g.pos_of_id;
  bs->direct = N <= kBfsDirect;
  LA3G_CUDA(cudaHostAlloc(&bs->stats, bs->direct ? 256 + n4 + n1 : sizeof(BfsStats), cudaHostAllocMapped));
  A.stats = bs->stats;
  if (bs->direct)
  {
    bs->parent_id = (uint32_t*) ((char*) bs->stats + 256);
    bs->hops_id = (uint8_t*) bs->parent_id + n4;
  }
  return LA3G_OK;
}

static int bfs_scratch(la3g_graph* G, BfsScratch** out)
{
  return graph_scratch(G, kSlotBfs, bfs_scratch_free, out, [&](BfsScratch* bs) { return bfs_scratch_build(G, bs); });
}

}  // namespace la3g

using namespace la3g;

extern "C" int la3g_bfs(la3g_graph* G, uint32_t root, uint8_t* hops_out, uint32_t* parent_out, la3g_stats* st)
{
  if (!G) return set_error(LA3G_EINVAL, "null graph");
  DevGraph& g = G->g;
  if (g.directed()) return set_error(LA3G_EINVAL, "bfs needs an undirected graph (load without LA3G_DIRECTED)");
  CallTimer T(G, st);
  BfsScratch* bs = nullptr;
  LA3G_TRY(bfs_scratch(G, &bs));
  cudaStream_t s = G->stream;
  const uint32_t N = g.nslots;
  const bool none = root >= N;  // no vertex matches the root: every hop stays 255
  T.device_begin();
  if (none)
  {
    k_bfs_none<<<grid_for(N, 256), 256, 0, s>>>(N, bs->hops_id, bs->parent_id);
    LA3G_LAUNCHED();
    tls_launches++;
  }
  else
  {
    BfsArgs A = bs->A;
    A.root = root;
    A.wait_polls = G->wait_polls;
    bs->stats->status = kBfsRunning;
    A.hops_out = hops_out ? bs->hops_id : nullptr;
    A.parent_out = parent_out ? bs->parent_id : nullptr;
    // row offsets and hops of every vertex; the edges examined are added below
    ProfileScope p("bfs", s, 9.0 * N);
    LA3G_TRY(bfs_launch<false>(A, &bs->grid, s));
  }
  T.device_end();
  if (hops_out && !bs->direct) LA3G_CUDA(cudaMemcpyAsync(hops_out, bs->hops_id, N, cudaMemcpyDeviceToHost, s));
  if (parent_out && !bs->direct)
    LA3G_CUDA(cudaMemcpyAsync(parent_out, bs->parent_id, (size_t) N * 4, cudaMemcpyDeviceToHost, s));
  LA3G_TRY(T.finish());
  if (bs->direct)
  {
    if (hops_out) std::memcpy(hops_out, bs->hops_id, N);
    if (parent_out) std::memcpy(parent_out, bs->parent_id, (size_t) N * 4);
  }
  if (none)
  {
    if (st) st->iterations = 1;
    return LA3G_OK;
  }
  const BfsStats r = *bs->stats;
  if (r.status == kBfsRunning) return set_error(LA3G_ETIMEOUT, "bfs: a grid barrier wait ran out");
  if (r.status) return set_error(LA3G_ETIMEOUT, "bfs did not converge");
  profile_add_bytes("bfs", 4.0 * (double) r.examined);
  if (st)
  {
    st->iterations = (uint32_t) r.iterations;
    st->pull_iterations = (uint32_t) r.pulls;
    st->edges_examined = r.examined;
    st->teps_edges = r.reached_deg / 2;
    st->algo_bytes = r.examined * 4 + (uint64_t) N * 6;
  }
  return LA3G_OK;
}

// ---------------------------------------------------------------------------
// la3g_bfs_noalloc: the same BFS kernel over a CSR the caller already holds
// in device memory, with every temporary in one fixed device array, so the
// call itself never allocates.
//
// The scratch lives in `g_bfs_noalloc_scratch`, a file-scope __device__
// array: each GPU that loads this library holds it (kNoAllocScratchBytes,
// about 12.8 MB) until the process exits.  Host code must not hand the
// array's name to a kernel (on the host it only names a stand-in object);
// every call looks up its device address on the current device with
// cudaGetSymbolAddress (which allocates nothing), so the address stays right
// for whichever device and context is current.
//
// All calls share the one array and it keeps whatever the last call left in
// it; the call clears what has to start at zero.  Two calls whose work
// overlaps on the GPU (different streams, or different host threads on one
// device) race on the array: serialise them.  The call waits for its stream
// before it returns, on success and on every error after its first launch, so
// no work of a finished call is left running on the array.
// ---------------------------------------------------------------------------

namespace la3g {

static constexpr uint32_t kNoAllocMaxVertices = 1u << 20;
static constexpr size_t kNaAlign = 256;
static constexpr size_t na_round(size_t b) { return (b + kNaAlign - 1) / kNaAlign * kNaAlign; }
static constexpr uint32_t kNaWords = kNoAllocMaxVertices / 32 + 1;
static constexpr size_t kNaCandOff = 0;
static constexpr size_t kNaList0Off = kNaCandOff + na_round(sizeof(uint32_t) * kNoAllocMaxVertices);
static constexpr size_t kNaList1Off = kNaList0Off + na_round(sizeof(uint32_t) * kNoAllocMaxVertices);
static constexpr size_t kNaBits0Off = kNaList1Off + na_round(sizeof(uint32_t) * kNoAllocMaxVertices);
static constexpr size_t kNaBits1Off = kNaBits0Off + na_round(sizeof(uint32_t) * kNaWords);
static constexpr size_t kNaCtrOff = kNaBits1Off + na_round(sizeof(uint32_t) * kNaWords);
static constexpr size_t kNaBarOff = kNaCtrOff + na_round(3 * sizeof(FrontierCounters));
static constexpr size_t kNaStatsOff = kNaBarOff + na_round(sizeof(unsigned int));
static constexpr size_t kNoAllocScratchBytes = kNaStatsOff + na_round(sizeof(BfsStats));

static __device__ __align__(256) unsigned char g_bfs_noalloc_scratch[kNoAllocScratchBytes];

// Device address of the scratch array on the current device.
static int noalloc_scratch(unsigned char** out)
{
  void* p = nullptr;
  const cudaError_t e = cudaGetSymbolAddress(&p, g_bfs_noalloc_scratch);
  if (e != cudaSuccess || !p)
  {
    cudaGetLastError();
    return set_error(LA3G_ECUDA, "cudaGetSymbolAddress(scratch) failed: %s", cudaGetErrorString(e));
  }
  *out = (unsigned char*) p;
  return LA3G_OK;
}

}  // namespace la3g

namespace la3g {

static int bfs_noalloc_run(const uint32_t* row_ptr, const uint32_t* col, const uint32_t* key, uint32_t nvertices,
                           uint32_t root, uint8_t* hops, uint32_t* parent, cudaStream_t s, la3g_stats* st,
                           bool* launched);

}  // namespace la3g

extern "C" int la3g_bfs_noalloc(const uint32_t* row_ptr, const uint32_t* col, const uint32_t* key,
                                uint32_t nvertices, uint32_t root, uint8_t* hops, uint32_t* parent,
                                void* cuda_stream, la3g_stats* st)
{
  using namespace la3g;
  if (st) std::memset(st, 0, sizeof *st);
  if (nvertices == 0 || nvertices > kNoAllocMaxVertices)
    return set_error(LA3G_EINVAL,
                     "la3g_bfs_noalloc: nvertices = %u; it must be between 1 and %u (the size of its fixed scratch)",
                     nvertices, kNoAllocMaxVertices);
  if (!row_ptr || !col || !key || !hops || !parent)
    return set_error(LA3G_EINVAL, "la3g_bfs_noalloc: row_ptr, col, key, hops and parent must be device pointers");
  cudaStream_t s = (cudaStream_t) cuda_stream;
  bool launched = false;
  const int rc = bfs_noalloc_run(row_ptr, col, key, nvertices, root, hops, parent, s, st, &launched);
  if (rc != LA3G_OK && launched)
  {
    // let the work already queued finish before the caller may reuse the array
    cudaStreamSynchronize(s);
    cudaGetLastError();
  }
  return rc;
}

namespace la3g {

static int bfs_noalloc_run(const uint32_t* row_ptr, const uint32_t* col, const uint32_t* key, uint32_t nvertices,
                           uint32_t root, uint8_t* hops, uint32_t* parent, cudaStream_t s, la3g_stats* st,
                           bool* launched)
{
  unsigned char* base = nullptr;
  LA3G_TRY(noalloc_scratch(&base));
  const uint32_t N = nvertices;
  const double t0 = now_ms();
  BfsStats r{1, 0, 0, 0, 0};
  *launched = true;
  if (root < N)
  {
    BfsArgs A{};
    A.ptr = row_ptr;
    A.col = col;
    A.key = key;
    A.N = A.nrows = N;
    A.limit = 100000;
    A.root = root;
    A.hops = A.hops_out = hops;
    A.cand = (uint32_t*) (base + kNaCandOff);
    // the parents are written at the end; until then their array holds the
    // hubs' task numbers, and later levels' parents once those are no longer used
    A.parent = A.task0 = A.parent_out = parent;
    A.list[0] = (uint32_t*) (base + kNaList0Off);
    A.list[1] = (uint32_t*) (base + kNaList1Off);
    A.bits[0] = (uint32_t*) (base + kNaBits0Off);
    A.bits[1] = (uint32_t*) (base + kNaBits1Off);
    A.ctr = (FrontierCounters*) (base + kNaCtrOff);
    A.bar = (unsigned int*) (base + kNaBarOff);
    A.wait_polls = -1;
    A.stats = (BfsStats*) (base + kNaStatsOff);
    unsigned grid = 0;
    LA3G_CUDA(cudaMemsetAsync(&A.stats->status, 0xFF, sizeof r.status, s));
    LA3G_TRY(bfs_launch<true>(A, &grid, s));
    LA3G_CUDA(cudaMemcpyAsync(&r, A.stats, sizeof r, cudaMemcpyDeviceToHost, s));
  }
  else
  {
    k_bfs_none<<<grid_for(N, 256), 256, 0, s>>>(N, hops, parent);
    LA3G_LAUNCHED();
  }
  LA3G_CUDA(cudaStreamSynchronize(s));
  if (r.status == 1) return set_error(LA3G_ETIMEOUT, "la3g_bfs_noalloc did not converge");
  if (r.status) return set_error(LA3G_ETIMEOUT, "la3g_bfs_noalloc: a grid barrier wait ran out");
  if (st)
  {
    st->iterations = (uint32_t) r.iterations;
    st->pull_iterations = (uint32_t) r.pulls;
    st->host_ms = now_ms() - t0;
  }
  return LA3G_OK;
}

}  // namespace la3g
