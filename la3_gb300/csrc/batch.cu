// Batched multi-source BFS and SSSP.  The reference runs one root per
// VertexProgram (bfs.cpp:11-37, sssp.cpp:11-37); here a batch of roots runs
// together and every root's result equals what la3g_bfs / la3g_sssp return
// for it alone.
//
// BFS: 64 roots per uint64 word, W = ceil(R / 64) words per vertex (vertex-
// major, so the W words of a vertex are contiguous).  A level is a bit-
// parallel SpMM over the OR semiring:
//     next[v][w] = (OR over neighbours u of front[u][w]) & ~visited[v][w]
// run bottom-up (pull) when the frontier is dense and top-down (push, an
// atomicOr per edge and word) when it is sparse.  Per-word "alive" masks
// record which roots still discovered something; words whose roots are all
// finished are skipped (done-masks).  All levels run inside one cooperative
// kernel with a grid barrier whose waits are bounded (a barrier that waits too
// long makes every block return): with a host round trip per
// level a batch of 64 roots on R-MAT 2^18 spent a third of its time between
// kernels.
// BFS levels are order-free, so hops equal the single-root runs; a batch
// whose BFS would exceed 254 levels (where the reference's uint8 hops wrap)
// is rerun root by root with la3g_bfs.
//
// SSSP: per-root distances, vertex-major ([vertex][root]); a frontier bit
// per (vertex, root); an iteration relaxes the out-edges of every active
// (vertex, root) into regular rows with atomicMin, then the sink rows are
// computed once, as in the single-root run.  With every edge weight at most
// (2^31 - 1) / n no distance can reach INF and no sum can wrap, so the fixed
// point equals the single-root result whatever the relaxation order; batches
// on graphs that do not satisfy that bound are run root by root.
#include <algorithm>
#include <chrono>
#include <cstring>
#include <string>
#include <vector>

#include "la3g_internal.h"
#include "frontier.cuh"
#include "lanes.cuh"

namespace la3g {


struct BatchConfig
{
  int mode = 0;          // 0 = pushing or pulling levels, 1 = pulling levels only
  int block = 256;       // threads per block of the level kernels
  double push_frac = 0.05;  // push when frontier edges * words < push_frac * m * words
  bool tuned = false;
};

struct BatchScratch
{
  long long wait_polls = -1; // grid-barrier poll limit in mode 1 (la3g_batch_set_wait_limit; < 0: the default)
  uint32_t cap_r = 0;        // roots the buffers were sized for
  uint64_t* vis = nullptr;   // [N][W]
  uint64_t* buf[2] = {nullptr, nullptr};  // frontier / next, [N][W]
  uint64_t* alive[3] = {nullptr, nullptr, nullptr};  // [W] per-word "discovered something" masks
  uint8_t* hops = nullptr;   // [N][W * 64] by position (vertex-major)
  uint32_t* rpos = nullptr;  // [R] root ids, then positions
  uint32_t* active = nullptr;  // push: active (vertex, word) pairs of small vertices
  uint32_t* phub = nullptr;    // push: pairs of hub vertices, and their first task numbers
  uint32_t* phub_t0 = nullptr;
  // BFS: [0..2] new bits of the levels in turn, [3] small pairs, [4] hub slots
  // and tasks (packed).  SSSP: [c], [2 + c] list c's small pairs and packed
  // hubs, [4 + c] smallest distance list c holds
  unsigned long long* ctr = nullptr;
  unsigned long long* hctr = nullptr;  // pinned, written by the kernels: [0] levels / iterations, [1] status
  unsigned int* bar = nullptr;         // grid barrier's count
  uint8_t* tpos = nullptr;             // results by root and id, before they leave the device
  size_t tpos_bytes = 0;
  BatchConfig cfg;                           // set by hand, or the default
  std::vector<std::pair<uint32_t, BatchConfig>> tuned;  // autotuned, by words per batch
  // SSSP
  uint32_t cap_sr = 0;
  uint32_t* sdist = nullptr;   // [N][R]
  uint64_t* sfront[2] = {nullptr, nullptr};  // [N][W]
  uint32_t* sact[2] = {nullptr, nullptr};    // active (vertex, word) pairs, N*W each
  uint32_t* shub[2] = {nullptr, nullptr};    // pairs of high-degree vertices, N*W each
  uint32_t* shub_t0[2] = {nullptr, nullptr}; // their first task numbers
  uint32_t* reg_end = nullptr;
  uint32_t max_w = 0;
  uint32_t max_reg_deg = 0;    // most regular out-edges of one vertex
  bool max_w_known = false;
  uint32_t sssp_delta = 0;     // distance window width; 0 = automatic, kNoWindow = none
};

static void batch_scratch_free(void* p)
{
  BatchScratch* b = (BatchScratch*) p;
  if (b->hctr) cudaFreeHost(b->hctr);
  delete b;
}

// ------------------------------------------------------------------ BFS

__global__ void k_ms_init(uint32_t N, uint32_t W, uint32_t R, uint64_t* vis, uint64_t* front, uint64_t* next)
{
  const uint64_t NW = (uint64_t) N * W;
  for (uint64_t i = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x; i < NW; i += (uint64_t) gridDim.x * blockDim.x)
  {
    const uint32_t w = (uint32_t) (i % W);
    // roots beyond R in the last word count as already visited
    const uint32_t lo = w * 64;
    uint64_t pad = 0;
    if (lo + 64 > R) pad = ~0ull << (R - lo);
    vis[i] = pad;
    front[i] = 0;
    next[i] = 0;
  }
}

__global__ void k_ms_roots(const uint32_t* __restrict__ rpos, uint32_t R, uint32_t N, uint32_t W, uint64_t* vis,
                           uint64_t* front, uint8_t* hops, uint64_t* alive)
{
  for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < R; r += gridDim.x * blockDim.x)
  {
    const uint32_t p = rpos[r];
    if (p >= N) continue;  // out-of-range root: nothing matches, all 255
    const uint32_t w = r / 64;
    const uint64_t bit = 1ull << (r % 64);
    atomicOr((unsigned long long*) &vis[(uint64_t) p * W + w], (unsigned long long) bit);
    atomicOr((unsigned long long*) &front[(uint64_t) p * W + w], (unsigned long long) bit);
    atomicOr((unsigned long long*) &alive[w], (unsigned long long) bit);
    hops[((uint64_t) p * W + w) * 64 + r % 64] = 0;
  }
}

struct MsArgs
{
  const uint32_t *ptr, *col;
  uint32_t nrows, N, W, R;
  uint64_t* vis;
  uint64_t* buf[2];    // the frontier of level l in buf[l & 1]
  uint64_t* alive[3];  // the roots still active at level l in alive[l % 3]
  uint8_t* hops;
  PairList list;       // pushing levels: the frontier's pairs
  unsigned long long* ctr;
  unsigned int* bar;
  long long wait_polls;
  // a level pushes when its new bits x mean degree stay below the limit
  double mean_deg, push_limit;
  unsigned long long* out;  // pinned: levels run, status
};

static constexpr uint32_t kMsAliveShared = 256;  // words of the alive mask gathered per block

// What a warp found for 32 consecutive pairs: visited bits, hop bytes, the
// roots still alive (in shared memory first: thousands of pairs would meet at
// a few global words).
__device__ __forceinline__ uint32_t ms_found(const MsArgs& A, uint64_t base, bool ok, uint64_t nb, uint64_t seen, uint8_t hop,
                                             int lane, unsigned long long* s_alive, unsigned long long* alive_next)
{
  const uint64_t i = base + lane;
  if (ok) A.buf[hop & 1][i] = nb;
  if (nb)
  {
    A.vis[i] = seen | nb;
    const uint32_t w = (uint32_t) (i % A.W);
    if (A.W <= kMsAliveShared)
    {
      if ((*(volatile unsigned long long*) &s_alive[w] & nb) != nb) atomicOr(&s_alive[w], (unsigned long long) nb);
    }
    else if ((__ldcg(&alive_next[w]) & nb) != nb) atomicOr(&alive_next[w], (unsigned long long) nb);
  }
  hops_record_warp(A.hops + base * 64, nb, hop, lane);
  return __popcll(nb);
}

// All levels of a batch.  A pulling level (pull_scan: a lane per (vertex,
// word) pair, the warp for long in-edge lists) writes every word of the next
// frontier; a pushing one lists the frontier's nonzero words and clears the
// next, pushes them to the neighbours (masked by visited), then applies.
__global__ void __launch_bounds__(512) k_ms_run(MsArgs A)
{
  __shared__ unsigned long long s_alive[kMsAliveShared], s_got[3];
  GridBarrier bar{A.bar, A.wait_polls};
  const int lane = threadIdx.x & 31;
  const uint64_t tid = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x, nth = (uint64_t) gridDim.x * blockDim.x;
  const uint64_t NW = (uint64_t) A.nrows * A.W;
  unsigned long long found = A.R;  // level 0: every root
  uint32_t level = 0;
  for (; level < 255 && found; level++)
  {
    const uint64_t* front = A.buf[level & 1];
    uint64_t* next = A.buf[(level + 1) & 1];
    const uint64_t* alive_now = A.alive[level % 3];
    unsigned long long* alive_next = (unsigned long long*) A.alive[(level + 1) % 3];
    const uint8_t hop = (uint8_t) (level + 1);
    for (uint64_t w = tid; w < A.W; w += nth) A.alive[(level + 2) % 3][w] = 0;
    if (tid == 0) A.ctr[(level + 2) % 3] = 0;
    for (uint32_t w = threadIdx.x; w < kMsAliveShared; w += blockDim.x) s_alive[w] = 0;
    const bool push = (double) found * A.mean_deg < A.push_limit;
    if (push)
    {
      for (uint64_t i = tid; i < NW; i += nth)
      {
        next[i] = 0;
        if (front[i])
        {
          const uint32_t v = (uint32_t) (i / A.W);
          bs_list_pair((uint32_t) i, A.ptr[v + 1] - A.ptr[v], A.list);
        }
      }
      if (!bar.sync()) return;
      if (threadIdx.x == 0)
      {
        s_got[0] = __ldcg(A.list.nsmall);
        s_got[1] = __ldcg(A.list.packed);
      }
      __syncthreads();
      ms_push_pairs(A.ptr, A.col, A.W, front, A.vis, next, A.list, (uint32_t) s_got[0], s_got[1]);
      if (!bar.sync()) return;
      if (tid == 0) *A.list.nsmall = *A.list.packed = 0;
    }
    else __syncthreads();
    uint32_t cnt = 0;
    for (uint64_t base = (tid >> 5) * 32; base < NW; base += (nth >> 5) * 32)
    {
      const uint64_t i = base + lane;
      const bool ok = i < NW;
      const uint64_t seen = ok ? A.vis[i] : ~0ull;
      uint64_t nb;
      if (push) nb = ok ? next[i] & ~seen : 0;
      else
      {
        const uint32_t v = ok ? (uint32_t) (i / A.W) : 0, w = ok ? (uint32_t) (i % A.W) : 0;
        nb = pull_scan(v, w, A.W, ok ? ~seen & alive_now[w] : 0, A.ptr, A.col, front, lane);
      }
      cnt += ms_found(A, base, ok, nb, seen, hop, lane, s_alive, alive_next);
    }
    const unsigned long long total = block_sum_u64(cnt);  // (its barriers order s_alive too)
    if (threadIdx.x == 0 && total) atomicAdd(&A.ctr[(level + 1) % 3], total);
    if (A.W <= kMsAliveShared)
      for (uint32_t w = threadIdx.x; w < A.W; w += blockDim.x)
        if (s_alive[w]) atomicOr(&alive_next[w], s_alive[w]);
    if (!bar.sync()) return;
    if (threadIdx.x == 0) s_got[2] = __ldcg(&A.ctr[(level + 1) % 3]);
    __syncthreads();
    found = s_got[2];
  }
  if (tid == 0)
  {
    A.out[0] = level;
    A.out[1] = found ? 2 : 1;  // 2: more levels than a byte of hops holds
  }
}

// Hops to out[root][id]: a block takes 128 ids and the 64 roots of a word, reads
// each id's 64 bytes (16 lanes, 4 bytes each), transposes them in shared memory
// and writes runs of 128 bytes.  (A transpose by position and a gather by id
// took 36 + 54 us for 64 roots on R-MAT 2^18; this takes 14 us.)
__global__ void __launch_bounds__(256) k_ms_out(uint32_t N, uint32_t R, uint32_t W, const uint32_t* __restrict__ pos_of_id,
                                                const uint8_t* __restrict__ hops, uint8_t* __restrict__ out)
{
  __shared__ uint8_t t[64][132];
  const uint32_t tid = threadIdx.x, nid = (N + 127) / 128;
  for (uint64_t tile = blockIdx.x; tile < (uint64_t) nid * W; tile += gridDim.x)
  {
    const uint32_t id0 = (uint32_t) (tile % nid) * 128, w = (uint32_t) (tile / nid);
    uint32_t v[8];
#pragma unroll
    for (int k = 0; k < 8; k++)
    {
      const uint32_t id = id0 + k * 16 + (tid >> 4);
      v[k] = id < N ? *reinterpret_cast<const uint32_t*>(hops + ((uint64_t) pos_of_id[id] * W + w) * 64 + 4 * (tid & 15)) : 0;
    }
#pragma unroll
    for (int k = 0; k < 8; k++)
#pragma unroll
      for (int q = 0; q < 4; q++) t[4 * (tid & 15) + q][k * 16 + (tid >> 4)] = (uint8_t) (v[k] >> (8 * q));
    __syncthreads();
    const uint32_t nr = min(64u, R - w * 64), x = tid & 127;
    if (id0 + x < N)
      for (uint32_t r = tid >> 7; r < nr; r += 2) out[(uint64_t) (w * 64 + r) * N + id0 + x] = t[r][x];
    __syncthreads();
  }
}

// The buffer results are put in order in before they leave the device: one, of
// the largest size asked for.
static int batch_out_buffer(la3g_graph* G, BatchScratch* b, size_t bytes)
{
  if (bytes <= b->tpos_bytes) return LA3G_OK;
  galloc_release(G, b->tpos);
  b->tpos = nullptr;
  b->tpos_bytes = 0;
  LA3G_TRY(galloc(G, &b->tpos, bytes));
  b->tpos_bytes = bytes;
  return LA3G_OK;
}

static int batch_scratch(la3g_graph* G, BatchScratch** out)
{
  return graph_scratch(G, kSlotBatch, batch_scratch_free, out, [&](BatchScratch* b) -> int {
    LA3G_TRY(galloc(G, &b->ctr, 8));
    LA3G_TRY(galloc(G, &b->bar, 1));
    LA3G_CUDA(cudaHostAlloc(&b->hctr, 2 * sizeof(unsigned long long), cudaHostAllocMapped));
    return LA3G_OK;
  });
}

// Larger buffers take the place of those in use when all of them are there.
static int ms_bfs_alloc(la3g_graph* G, BatchScratch* b, uint32_t R)
{
  if (R <= b->cap_r) return LA3G_OK;
  const uint32_t N = G->g.nslots, W = (R + 63) / 64;
  GallocScope scope(G);
  BatchScratch t = *b;
  LA3G_TRY(galloc(G, &t.vis, (size_t) N * W));
  LA3G_TRY(galloc(G, &t.buf[0], (size_t) N * W));
  LA3G_TRY(galloc(G, &t.buf[1], (size_t) N * W));
  for (int k = 0; k < 3; k++) LA3G_TRY(galloc(G, &t.alive[k], W));
  LA3G_TRY(galloc(G, &t.hops, (size_t) N * W * 64));
  LA3G_TRY(galloc(G, &t.rpos, R));
  LA3G_TRY(galloc(G, &t.active, (size_t) N * W));
  LA3G_TRY(galloc(G, &t.phub, (size_t) N * W));
  LA3G_TRY(galloc(G, &t.phub_t0, (size_t) N * W));
  t.cap_r = R;
  scope.keep();
  for (void* p : {(void*) b->vis, (void*) b->buf[0], (void*) b->buf[1], (void*) b->alive[0], (void*) b->alive[1],
                  (void*) b->alive[2], (void*) b->hops, (void*) b->rpos, (void*) b->active, (void*) b->phub,
                  (void*) b->phub_t0})
    galloc_release(G, p);
  *b = t;
  return LA3G_OK;
}

static int bs_alloc(la3g_graph* G, BatchScratch* b, uint32_t R)
{
  if (R <= b->cap_sr) return LA3G_OK;
  const uint32_t N = G->g.nslots, W = (R + 63) / 64;
  GallocScope scope(G);
  BatchScratch t = *b;
  LA3G_TRY(galloc(G, &t.sdist, (size_t) N * R));
  for (int c = 0; c < 2; c++)
  {
    LA3G_TRY(galloc(G, &t.sfront[c], (size_t) N * W));
    LA3G_TRY(galloc(G, &t.sact[c], (size_t) N * W));
    LA3G_TRY(galloc(G, &t.shub[c], (size_t) N * W));
    LA3G_TRY(galloc(G, &t.shub_t0[c], (size_t) N * W));
  }
  t.cap_sr = R;
  scope.keep();
  galloc_release(G, b->sdist);
  for (int c = 0; c < 2; c++)
    for (void* p : {(void*) b->sfront[c], (void*) b->sact[c], (void*) b->shub[c], (void*) b->shub_t0[c]}) galloc_release(G, p);
  *b = t;
  return LA3G_OK;
}

// Root ids -> positions, in place.
__global__ void k_root_pos(uint32_t R, uint32_t N, const uint32_t* __restrict__ pos_of_id, uint32_t* rpos)
{
  for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < R; r += gridDim.x * blockDim.x)
    rpos[r] = rpos[r] < N ? pos_of_id[rpos[r]] : 0xFFFFFFFFu;
}

// Runs one batch; hops by position stay in b->hops.  Returns the level count
// in *levels; *wrap = true when some root would need more than 254 levels.
static int ms_bfs_run(la3g_graph* G, BatchScratch* b, const uint32_t* roots_host, uint32_t R, const BatchConfig& cfg,
                      uint32_t* levels, bool* wrap, uint64_t* edges_words)
{
  DevGraph& g = G->g;
  cudaStream_t s = G->stream;
  const uint32_t N = g.nslots, nrows = g.nrows(), W = (R + 63) / 64;
  LA3G_TRY(ms_bfs_alloc(G, b, R));
  LA3G_CUDA(cudaMemcpyAsync(b->rpos, roots_host, (size_t) R * 4, cudaMemcpyHostToDevice, s));
  k_root_pos<<<grid_for(R, 256), 256, 0, s>>>(R, N, g.pos_of_id, b->rpos);
  LA3G_LAUNCHED();
  k_ms_init<<<num_sms() * 8, 256, 0, s>>>(N, W, R, b->vis, b->buf[0], b->buf[1]);
  LA3G_LAUNCHED();
  LA3G_CUDA(cudaMemsetAsync(b->hops, 0xFF, (size_t) N * W * 64, s));
  for (int k = 0; k < 3; k++) LA3G_CUDA(cudaMemsetAsync(b->alive[k], 0, (size_t) W * 8, s));
  LA3G_CUDA(cudaMemsetAsync(b->ctr, 0, 8 * 8, s));
  LA3G_CUDA(cudaMemsetAsync(b->bar, 0, sizeof *b->bar, s));
  k_ms_roots<<<grid_for(R, 256), 256, 0, s>>>(b->rpos, R, N, W, b->vis, b->buf[0], b->hops, b->alive[0]);
  LA3G_LAUNCHED();
  tls_launches += 3;
  MsArgs A;
  A.ptr = g.in_ptr;
  A.col = g.in_col;
  A.nrows = nrows;
  A.N = N;
  A.W = W;
  A.R = R;
  A.vis = b->vis;
  for (int k = 0; k < 2; k++) A.buf[k] = b->buf[k];
  for (int k = 0; k < 3; k++) A.alive[k] = b->alive[k];
  A.hops = b->hops;
  A.list = PairList{b->active, b->phub, b->phub_t0, b->ctr + 3, b->ctr + 4};
  A.ctr = b->ctr;
  A.bar = b->bar;
  A.wait_polls = barrier_polls(cfg.mode == 1 ? b->wait_polls : -1, g.nent);
  A.mean_deg = (double) g.nent / std::max<uint32_t>(1, nrows);
  A.push_limit = cfg.mode == 1 ? 0.0 : cfg.push_frac * (double) g.nent * 64.0 * W;
  A.out = b->hctr;
  b->hctr[1] = 0;
  unsigned grid = 0;
  LA3G_TRY(cooperative_blocks((const void*) k_ms_run, cfg.block, std::max<uint64_t>((uint64_t) nrows * W, g.nent / 8),
                              2048 / cfg.block, &grid));
  {
    void* args[] = {(void*) &A};
    ProfileScope p("msbfs", s, 0.0);
    LA3G_CUDA(cudaLaunchCooperativeKernel((const void*) k_ms_run, grid, cfg.block, args, 0, s));
  }
  LA3G_CUDA(cudaStreamSynchronize(s));
  if (!b->hctr[1]) return set_error(LA3G_ETIMEOUT, "batched BFS: a grid barrier wait ran out");
  *levels = (uint32_t) b->hctr[0];
  *wrap = b->hctr[1] == 2;
  *edges_words = (uint64_t) *levels * g.nent * W;
  return LA3G_OK;
}

// ------------------------------------------------------------------ SSSP

__global__ void k_bs_init(uint64_t n, uint32_t* dist, uint64_t nw, uint64_t* f0, uint64_t* f1)
{
  for (uint64_t i = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t) gridDim.x * blockDim.x)
    dist[i] = kInfD;
  for (uint64_t i = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x; i < nw; i += (uint64_t) gridDim.x * blockDim.x)
  {
    f0[i] = 0;
    f1[i] = 0;
  }
}

__global__ void k_bs_roots(const uint32_t* __restrict__ rpos, uint32_t R, uint32_t N, uint32_t W, uint32_t nreg,
                           uint32_t src_base, uint32_t iso_base, uint32_t* dist, uint64_t* front)
{
  for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < R; r += gridDim.x * blockDim.x)
  {
    const uint32_t p = rpos[r];
    if (p >= N) continue;
    dist[(uint64_t) p * R + r] = 0;
    if (p < nreg || (p >= src_base && p < iso_base))
      atomicOr((unsigned long long*) &front[(uint64_t) p * W + r / 64], 1ull << (r % 64));
  }
}

// Sink rows once: min over regular in-neighbours' final distances and the
// root's message where the root is a source.
__global__ void k_bs_sinks(const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ col, const uint32_t* __restrict__ wgt,
                           uint32_t nreg, uint32_t nsink, uint32_t R, const uint32_t* __restrict__ rpos,
                           uint32_t src_base, uint32_t iso_base, uint32_t* dist)
{
  const uint64_t n = (uint64_t) nsink * R;
  for (uint64_t i = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t) gridDim.x * blockDim.x)
  {
    const uint32_t v = nreg + (uint32_t) (i / R), r = (uint32_t) (i % R);
    const uint32_t rp = rpos[r];
    uint32_t y = kInfD;
    for (uint32_t e = ptr[v]; e < ptr[v + 1]; e++)
    {
      const uint32_t c = col[e];
      uint32_t cand;
      if (c < nreg) cand = dist[(uint64_t) c * R + r] + wgt[e];
      else if (c == rp && rp >= src_base && rp < iso_base) cand = wgt[e];
      else continue;
      y = min(y, cand);
    }
    uint32_t* d = &dist[(uint64_t) v * R + r];
    *d = min(*d, y);
  }
}

// Distances to out[root][id]: a block takes 32 ids and 32 roots, reads each id's
// 128 bytes and writes runs of 128 bytes by id.
__global__ void __launch_bounds__(256) k_bs_out(uint32_t N, uint32_t R, const uint32_t* __restrict__ pos_of_id,
                                                const uint32_t* __restrict__ dist, uint32_t* __restrict__ out)
{
  __shared__ uint32_t t[32][33];
  const uint32_t tx = threadIdx.x & 31, ty = threadIdx.x >> 5, nid = (N + 31) / 32, nr = (R + 31) / 32;
  for (uint64_t tile = blockIdx.x; tile < (uint64_t) nid * nr; tile += gridDim.x)
  {
    const uint32_t id0 = (uint32_t) (tile % nid) * 32, r0 = (uint32_t) (tile / nid) * 32;
#pragma unroll
    for (int k = 0; k < 4; k++)
    {
      const uint32_t id = id0 + ty + 8 * k;
      t[ty + 8 * k][tx] = id < N && r0 + tx < R ? dist[(uint64_t) pos_of_id[id] * R + r0 + tx] : 0u;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; k++)
    {
      const uint32_t r = r0 + ty + 8 * k;
      if (r < R && id0 + tx < N) out[(uint64_t) r * N + id0 + tx] = t[tx][ty + 8 * k];
    }
    __syncthreads();
  }
}

struct BsArgs
{
  const uint32_t *ptr, *reg_end, *row, *wgt;
  uint32_t N, R, W;
  uint64_t* front[2];
  PairList L[2];            // their counters: ctr[c], ctr[2 + c]
  uint32_t* dist;
  unsigned long long* ctr;
  unsigned int* bar;
  long long wait_polls;
  uint32_t delta;           // kNoWindow: no window
  unsigned long long* out;  // pinned: iterations, status
};

// All iterations of a batch's SSSP: relax the listed pairs, then form the next
// list (see lanes.cuh), a grid barrier after each.  With a window, the smallest
// distance a list holds collects in ctr[4 + c] during the relaxation that
// forms it and sets the next limit.
__global__ void __launch_bounds__(256, 4) k_bs_run(BsArgs A)
{
  __shared__ unsigned long long s_got[3];
  __shared__ unsigned int s_taken;
  GridBarrier bar{A.bar, A.wait_polls};
  const uint64_t tid = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t iters = 0, limit = A.delta;
  int cur = 0;
  if (threadIdx.x == 0) s_taken = 0;
  auto counts = [&]() {
    if (threadIdx.x < 3) s_got[threadIdx.x] = __ldcg(&A.ctr[2 * threadIdx.x + cur]);
    __syncthreads();
  };
  counts();
  for (;;)
  {
    const unsigned long long ns = s_got[0], pk = s_got[1];
    __syncthreads();  // s_got is free
    if (iters > 1000000) break;
    iters++;
    unsigned int* pend = (unsigned int*) &A.ctr[4 + (cur ^ 1)];
    if (tid == 0) A.ctr[cur ^ 1] = A.ctr[2 + (cur ^ 1)] = 0;  // the list formed next
    bs_relax_all(A.ptr, A.reg_end, A.row, A.wgt, A.R, A.W, A.front[cur], A.L[cur], (uint32_t) ns, pk, A.front[cur ^ 1],
                 A.dist, A.delta == kNoWindow ? kNoWindow : limit, A.delta == kNoWindow ? nullptr : pend, &s_taken);
    if (!bar.sync()) return;
    // every block has read this list's smallest distance: it starts over for
    // the list after the next
    if (tid == 0) *(unsigned int*) &A.ctr[4 + cur] = 0xFFFFFFFFu;
    if (threadIdx.x == 0) s_taken = 0;
    bs_apply_all(A.N, A.W, A.ptr, A.reg_end, A.front[cur ^ 1], A.L[cur ^ 1], A.front[cur], A.L[cur], ns, hub_count(pk),
                 nullptr);
    if (!bar.sync()) return;
    cur ^= 1;
    counts();
    if (!s_got[0] && !s_got[1]) break;
    if (A.delta != kNoWindow)
    {
      const uint32_t lo = (uint32_t) s_got[2];
      limit = lo > kNoWindow - 1 - A.delta ? kNoWindow - 1 : lo + A.delta;
    }
  }
  if (tid == 0)
  {
    A.out[0] = iters;
    A.out[1] = iters > 1000000 ? 2 : 1;
  }
}

}  // namespace la3g

using namespace la3g;

extern "C" int la3g_bfs_batch(la3g_graph* G, const uint32_t* roots, uint32_t nroots, uint8_t* hops_out, la3g_stats* st)
{
  if (!G) return set_error(LA3G_EINVAL, "null graph");
  if (nroots == 0) return set_error(LA3G_EINVAL, "nroots must be > 0");
  if (!roots) return set_error(LA3G_EINVAL, "roots is null");
  DevGraph& g = G->g;
  if (g.directed()) return set_error(LA3G_EINVAL, "bfs needs an undirected graph");
  CallTimer T(G, st);
  BatchScratch* b = nullptr;
  LA3G_TRY(batch_scratch(G, &b));
  const uint32_t N = g.nslots;
  uint32_t levels = 0;
  bool wrap = false;
  uint64_t ew = 0;
  T.device_begin();
  // the configuration tuned for this many words if there is one (the nearest
  // tuned word count otherwise), else the hand-set / default one
  BatchConfig cfg = b->cfg;
  {
    const uint32_t W = (nroots + 63) / 64;
    uint32_t best = 0xFFFFFFFFu;
    for (const auto& t : b->tuned)
    {
      const uint32_t dist = t.first > W ? t.first - W : W - t.first;
      if (dist < best) { best = dist; cfg = t.second; }
    }
  }
  LA3G_TRY(ms_bfs_run(G, b, roots, nroots, cfg, &levels, &wrap, &ew));
  T.device_end();
  cudaStream_t s = G->stream;
  if (hops_out)
  {
    LA3G_TRY(batch_out_buffer(G, b, (size_t) nroots * N));
    k_ms_out<<<num_sms() * 8, 256, 0, s>>>(N, nroots, (nroots + 63) / 64, g.pos_of_id, b->hops, b->tpos);
    LA3G_LAUNCHED();
    LA3G_CUDA(cudaMemcpyAsync(hops_out, b->tpos, (size_t) nroots * N, cudaMemcpyDeviceToHost, s));
    LA3G_CUDA(cudaStreamSynchronize(s));
  }
  LA3G_TRY(T.finish());
  if (wrap && hops_out)
  {
    // more than 254 levels: the reference's uint8 hops wrap; rerun the roots
    // one by one with the single-root path, which follows it exactly
    for (uint32_t r = 0; r < nroots; r++) LA3G_TRY(la3g_bfs(G, roots[r], hops_out + (size_t) r * N, nullptr, nullptr));
  }
  if (st)
  {
    st->iterations = levels;
    st->edges_examined = ew * 64;
  }
  return LA3G_OK;
}

// Distances (vertices x roots of a chunk) up to which the iterations run in one
// kernel.  There the host's round trips weigh most (ER 50k, 64 roots: 0.95 ms
// against 1.72; R-MAT 2^19, 64 roots: 3.4 against 3.9); with more, distances
// miss the L2 cache and the four-fold grid of a launch per iteration keeps more
// warps ready than the resident one (R-MAT 2^22, 16 roots: 9.2 ms against 10.2;
// ER 2^22, 64 roots: 64 against 79).
static constexpr uint64_t kBsOneKernel = 40ull << 20;

static constexpr uint32_t kSsspChunk = 256;  // roots per device pass (bounds the [N][R] state)

// Default window width of the batched SSSP.  The window pays where degrees
// are even (ER 2^22 x16, weights 1-128, 256 roots: 248 ms with a window of
// 128 against 272 ms without; 64 and 256 give 257 / 282 ms) and costs where
// hubs already make the frontier converge in few iterations (R-MAT s22: 88
// against 75 ms), so it is on only when no vertex is a hub (more than kBigDeg
// regular out-edges), with the largest weight as its width.
static uint32_t sssp_auto_delta(uint32_t max_w, uint32_t max_reg_deg)
{
  return max_reg_deg <= kBigDeg ? std::max(max_w, 1u) : kNoWindow;
}

__global__ void k_max_reg_deg(const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ reg_end, uint32_t N,
                              unsigned int* out)
{
  unsigned int m = 0;
  for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < N; u += gridDim.x * blockDim.x)
    m = max(m, reg_end[u] - ptr[u]);
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

static int sssp_batch_chunk(la3g_graph* G, BatchScratch* b, const uint32_t* roots, uint32_t R, uint32_t* dist_out,
                            uint32_t* iters_out);

extern "C" int la3g_sssp_batch(la3g_graph* G, const uint32_t* roots, uint32_t nroots, uint32_t* dist_out,
                               la3g_stats* st)
{
  if (!G) return set_error(LA3G_EINVAL, "null graph");
  if (nroots == 0) return set_error(LA3G_EINVAL, "nroots must be > 0");
  if (!roots) return set_error(LA3G_EINVAL, "roots is null");
  DevGraph& g = G->g;
  if (!g.directed() || !g.weighted() || (g.flags & (LA3G_REVERSE | LA3G_ACYCLIC | LA3G_BIPARTITE)))
    return set_error(LA3G_EINVAL, "sssp needs a graph loaded with LA3G_DIRECTED | LA3G_WEIGHTED");
  CallTimer T(G, st);
  LA3G_TRY(build_push_csr(G));
  BatchScratch* b = nullptr;
  LA3G_TRY(batch_scratch(G, &b));
  uint32_t iters = 0;
  T.device_begin();
  for (uint32_t r0 = 0; r0 < nroots; r0 += kSsspChunk)
  {
    const uint32_t R = std::min(kSsspChunk, nroots - r0);
    uint32_t it = 0;
    LA3G_TRY(sssp_batch_chunk(G, b, roots + r0, R, dist_out ? dist_out + (size_t) r0 * g.nslots : nullptr, &it));
    iters = std::max(iters, it);
  }
  T.device_end();
  LA3G_TRY(T.finish());
  if (st) st->iterations = iters;
  return LA3G_OK;
}

// The iterations of k_bs_run stepped from the host.
static int bs_stepped(la3g_graph* G, BatchScratch* b, const BsArgs& A)
{
  cudaStream_t s = G->stream;
  int cur = 0;
  uint32_t limit = A.delta;
  for (uint32_t iters = 1;; iters++)
  {
    unsigned int* pend = A.delta == kNoWindow ? nullptr : (unsigned int*) (b->ctr + 4);
    if (pend) LA3G_CUDA(cudaMemsetAsync(pend, 0xFF, 4, s));
    {
      ProfileScope p("sssp_batch_relax", s, 0.0);
      k_bs_relax<<<num_sms() * 16, 256, 0, s>>>(A.ptr, A.reg_end, A.row, A.wgt, A.R, A.W, A.front[cur], A.L[cur],
                                                A.front[cur ^ 1], A.dist, pend ? limit : kNoWindow, pend);
      LA3G_LAUNCHED();
    }
    LA3G_CUDA(cudaMemsetAsync(b->ctr + (cur ^ 1), 0, 8, s));
    LA3G_CUDA(cudaMemsetAsync(b->ctr + 2 + (cur ^ 1), 0, 8, s));
    k_bs_apply<<<num_sms() * 8, 256, 0, s>>>(A.N, A.W, A.ptr, A.reg_end, A.front[cur ^ 1], A.L[cur ^ 1], A.front[cur], A.L[cur]);
    LA3G_LAUNCHED();
    tls_launches += 2;
    unsigned long long act[5] = {0, 0, 0, 0, 0};
    LA3G_CUDA(cudaMemcpyAsync(act, b->ctr, 5 * 8, cudaMemcpyDeviceToHost, s));
    LA3G_CUDA(cudaStreamSynchronize(s));
    cur ^= 1;
    b->hctr[0] = iters;
    b->hctr[1] = iters > 1000000 ? 2 : 1;
    if ((!act[cur] && !act[2 + cur]) || iters > 1000000) return LA3G_OK;
    const uint32_t lo = (uint32_t) act[4];
    if (pend) limit = lo > kNoWindow - 1 - A.delta ? kNoWindow - 1 : lo + A.delta;
  }
}

static int sssp_batch_chunk(la3g_graph* G, BatchScratch* b, const uint32_t* roots, uint32_t R, uint32_t* dist_out,
                            uint32_t* iters_out)
{
  DevGraph& g = G->g;
  cudaStream_t s = G->stream;
  const uint32_t N = g.nslots, W = (R + 63) / 64;
  if (!b->max_w_known)
  {
    DevBuf m;
    LA3G_TRY(m.alloc(8));
    LA3G_CUDA(cudaMemsetAsync(m.p, 0, 8, s));
    if (g.nent)
    {
      k_max_u32<<<grid_for(g.nent, 256), 256, 0, s>>>(g.out_w, g.nent, m.as<unsigned int>());
      LA3G_LAUNCHED();
    }
    LA3G_TRY(galloc(G, &b->reg_end, N));
    k_reg_end<<<grid_for(N, 256), 256, 0, s>>>(g.out_ptr, g.out_row, N, g.nreg, b->reg_end);
    LA3G_LAUNCHED();
    k_max_reg_deg<<<grid_for(N, 256), 256, 0, s>>>(g.out_ptr, b->reg_end, N, m.as<unsigned int>() + 1);
    LA3G_LAUNCHED();
    uint32_t hm[2] = {0, 0};
    LA3G_CUDA(cudaMemcpyAsync(hm, m.p, 8, cudaMemcpyDeviceToHost, s));
    LA3G_CUDA(cudaStreamSynchronize(s));
    b->max_w = hm[0];
    b->max_reg_deg = hm[1];
    b->max_w_known = true;
  }
  // Exact regardless of relaxation order only if no distance can reach INF.
  if ((uint64_t) b->max_w * (uint64_t) N >= (uint64_t) kInfD)
  {
    for (uint32_t r = 0; r < R; r++)
      LA3G_TRY(la3g_sssp(G, roots[r], dist_out ? dist_out + (size_t) r * N : nullptr, nullptr));
    *iters_out = 0;
    return LA3G_OK;
  }
  LA3G_TRY(bs_alloc(G, b, R));
  LA3G_TRY(ms_bfs_alloc(G, b, R));
  LA3G_CUDA(cudaMemcpyAsync(b->rpos, roots, (size_t) R * 4, cudaMemcpyHostToDevice, s));
  k_root_pos<<<grid_for(R, 256), 256, 0, s>>>(R, N, g.pos_of_id, b->rpos);
  LA3G_LAUNCHED();
  k_bs_init<<<num_sms() * 8, 256, 0, s>>>((uint64_t) N * R, b->sdist, (uint64_t) N * W, b->sfront[0], b->sfront[1]);
  LA3G_LAUNCHED();
  k_bs_roots<<<grid_for(R, 256), 256, 0, s>>>(b->rpos, R, N, W, g.nreg, g.src_base(), g.iso_base(), b->sdist,
                                              b->sfront[0]);
  LA3G_LAUNCHED();
  tls_launches += 3;
  // the distance window: roots at distance <= limit relax, the rest wait;
  // after each iteration limit = (smallest distance left in the frontier) + delta
  const uint32_t delta = b->sssp_delta ? b->sssp_delta : sssp_auto_delta(b->max_w, b->max_reg_deg);
  BsArgs A;
  A.ptr = g.out_ptr;
  A.reg_end = b->reg_end;
  A.row = g.out_row;
  A.wgt = g.out_w;
  A.N = N;
  A.R = R;
  A.W = W;
  for (int c = 0; c < 2; c++)
  {
    A.front[c] = b->sfront[c];
    A.L[c] = PairList{b->sact[c], b->shub[c], b->shub_t0[c], b->ctr + c, b->ctr + 2 + c};
  }
  A.dist = b->sdist;
  A.ctr = b->ctr;
  A.bar = b->bar;
  A.wait_polls = barrier_polls(-1, g.nent);
  A.delta = delta;
  A.out = b->hctr;
  b->hctr[1] = 0;
  LA3G_CUDA(cudaMemsetAsync(b->ctr, 0, 4 * 8, s));
  LA3G_CUDA(cudaMemsetAsync(b->ctr + 4, 0xFF, 2 * 8, s));
  LA3G_CUDA(cudaMemsetAsync(b->bar, 0, sizeof *b->bar, s));
  k_bs_list<<<num_sms() * 8, 256, 0, s>>>((uint64_t) N * W, W, g.out_ptr, b->reg_end, b->sfront[0], A.L[0]);
  LA3G_LAUNCHED();
  tls_launches++;
  if ((uint64_t) N * R <= kBsOneKernel)
  {
    unsigned grid = 0;
    LA3G_TRY(cooperative_blocks((const void*) k_bs_run, 256, std::max<uint64_t>((uint64_t) N * W, g.nent * 2), 4, &grid));
    void* args[] = {(void*) &A};
    ProfileScope p("sssp_batch", s, 0.0);
    LA3G_CUDA(cudaLaunchCooperativeKernel((const void*) k_bs_run, grid, 256, args, 0, s));
  }
  else LA3G_TRY(bs_stepped(G, b, A));
  if (g.nsink)
  {
    k_bs_sinks<<<num_sms() * 8, 256, 0, s>>>(g.in_ptr, g.in_col, g.in_w, g.nreg, g.nsink, R, b->rpos, g.src_base(),
                                        g.iso_base(), b->sdist);
    LA3G_LAUNCHED();
    tls_launches++;
  }
  if (dist_out)
  {
    LA3G_TRY(batch_out_buffer(G, b, (size_t) N * R * 4));
    k_bs_out<<<num_sms() * 8, 256, 0, s>>>(N, R, g.pos_of_id, b->sdist, (uint32_t*) b->tpos);
    LA3G_LAUNCHED();
    LA3G_CUDA(cudaMemcpyAsync(dist_out, b->tpos, (size_t) N * R * 4, cudaMemcpyDeviceToHost, s));
  }
  LA3G_CUDA(cudaStreamSynchronize(s));
  if (b->hctr[1] != 1)
    return set_error(LA3G_ETIMEOUT, b->hctr[1] ? "batched sssp did not converge" : "batched sssp: a grid barrier wait ran out");
  *iters_out = (uint32_t) b->hctr[0];
  return LA3G_OK;
}

// Project autotuner for the batched BFS: times every combination of level
// mode (pushing and pulling levels / pulling only), block size and push
// threshold on the caller's roots and keeps the fastest for this graph.
extern "C" int la3g_batch_autotune(la3g_graph* G, const uint32_t* roots, uint32_t nroots, char* report, size_t cap)
{
  if (!G || !roots || nroots == 0) return set_error(LA3G_EINVAL, "graph and roots are required");
  if (G->g.directed()) return set_error(LA3G_EINVAL, "the batched BFS tunes on an undirected graph");
  BatchScratch* b = nullptr;
  LA3G_TRY(batch_scratch(G, &b));
  std::string rep = "[";
  BatchConfig best;
  double best_ms = 1e300;
  const int modes[] = {0, 1};
  const int blocks[] = {128, 256, 512};
  const double fracs[] = {0.0, 0.001, 0.003, 0.01, 0.02, 0.05, 0.1, 0.2, 0.4};
  for (int mode : modes)
    for (int block : blocks)
      for (double frac : fracs)
      {
        if (mode == 1 && frac != 0.0) continue;  // mode 1 pulls only
        BatchConfig c;
        c.mode = mode;
        c.block = block;
        c.push_frac = frac;
        uint32_t lv = 0;
        bool wrap = false;
        uint64_t ew = 0;
        LA3G_TRY(ms_bfs_run(G, b, roots, nroots, c, &lv, &wrap, &ew));  // warm
        LA3G_CUDA(cudaStreamSynchronize(G->stream));
        double ms = 1e300;
        for (int rep = 0; rep < 2; rep++)  // best of two
        {
          const double t0 = now_ms();
          LA3G_TRY(ms_bfs_run(G, b, roots, nroots, c, &lv, &wrap, &ew));
          LA3G_CUDA(cudaStreamSynchronize(G->stream));
          ms = std::min(ms, now_ms() - t0);
        }
        char buf[160];
        std::snprintf(buf, sizeof buf, "%s{\"mode\": %d, \"block\": %d, \"push_frac\": %.3f, \"ms\": %.4f}",
                      rep.size() > 1 ? ", " : "", mode, block, frac, ms);
        rep += buf;
        if (ms < best_ms) { best_ms = ms; best = c; }
      }
  best.tuned = true;
  const uint32_t W = (nroots + 63) / 64;
  bool found = false;
  for (auto& t : b->tuned)
    if (t.first == W)
    {
      t.second = best;
      found = true;
    }
  if (!found) b->tuned.emplace_back(W, best);
  rep += "]";
  if (report && cap)
  {
    size_t n = std::min(rep.size(), cap - 1);
    std::memcpy(report, rep.data(), n);
    report[n] = 0;
  }
  return LA3G_OK;
}

extern "C" int la3g_batch_set_wait_limit(la3g_graph* G, long long polls)
{
  if (!G) return set_error(LA3G_EINVAL, "null graph");
  BatchScratch* b = nullptr;
  LA3G_TRY(batch_scratch(G, &b));
  b->wait_polls = polls;
  return LA3G_OK;
}

extern "C" int la3g_batch_sssp_window(la3g_graph* G, uint32_t delta)
{
  if (!G) return set_error(LA3G_EINVAL, "null graph");
  BatchScratch* b = nullptr;
  LA3G_TRY(batch_scratch(G, &b));
  b->sssp_delta = delta;
  return LA3G_OK;
}

extern "C" int la3g_batch_config(la3g_graph* G, int mode, int block, double push_frac)
{
  if (!G) return set_error(LA3G_EINVAL, "null graph");
  if ((mode != 0 && mode != 1) || (block != 128 && block != 256 && block != 512) || push_frac < 0 || push_frac > 1)
    return set_error(LA3G_EINVAL, "mode must be 0 or 1, block 128/256/512, push_frac in [0, 1]");
  BatchScratch* b = nullptr;
  LA3G_TRY(batch_scratch(G, &b));
  b->cfg.mode = mode;
  b->cfg.block = block;
  b->cfg.push_frac = push_frac;
  b->cfg.tuned = true;
  b->tuned.clear();  // a hand-set configuration replaces the tuned ones
  return LA3G_OK;
}
