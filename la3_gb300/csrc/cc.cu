// Connected components: the reference cc app (src/apps/graph_analytics/
// cc.cpp:11-31, cc.h:11-38) on the device.
//
// The reference propagates labels (initially the vertex's own id) with
// combine y2 = (y2 == 0) ? y1 : min(y1, y2) until nothing changes.  When
// vertex 0 has no edges no label is ever 0, combine is a plain min, and
// the fixed point is: every vertex with edges carries the least id of its
// component, every isolated vertex its own id.  That fixed point is computed
// here with a lock-free union-find over the rows' positions (a root is only
// ever hooked under a smaller position), full path compression, and the least
// id of each tree.  Edges are processed Afforest-style (Sutton et al.): each row
// first hooks under its least neighbour, without atomics, then its tree is
// linked with a few more neighbours' by one atomicMin each, which may be lost;
// the giant component is found by sampling, and only rows outside it walk
// their edges (all of them: the graph is symmetric, so an edge that leaves the
// giant component is seen from its other end).  Positions, not ids, order the
// trees: the neighbours' ids need not be looked up, and a graph whose
// neighbours have consecutive ids (a path, a road network in order) does not
// hook into one long chain, since the bucket hash spreads them.
//
// When vertex 0 does have edges, label 0 behaves as "no value yet" and the
// outcome depends on the order messages arrive in, so that case runs the
// reference's BSP iterations literally: each row folds the messages of its
// active in-neighbours in ascending column order with the reference's
// combine.
#include <algorithm>
#include <cstring>
#include <vector>

#include "la3g_internal.h"

namespace la3g {

static constexpr int kCcFlags = 8;  // chains left by the compressions, one flag each

struct CcScratch
{
  uint32_t* label = nullptr;   // by original id
  uint32_t* parent = nullptr;  // [rows] union-find by position
  uint32_t* least = nullptr;   // [rows] least id of each root's tree
  uint32_t* deep = nullptr;    // [kCcFlags]
  uint32_t* probe = nullptr;   // roots of sampled vertices
  uint32_t* lab_pos = nullptr; // BSP path: labels by position
  uint32_t* msg = nullptr;
  uint8_t* active[2] = {nullptr, nullptr};
  int* flag = nullptr;
  unsigned long long* walked = nullptr;  // [0] rows, [1] edges k_cc_rest walked
  unsigned long long* hwalked = nullptr; // pinned mirror
  uint32_t* giant = nullptr;   // the sampled giant component's root, and the samples in it
  int zero_has_edges = -1;     // whether vertex 0 has edges (-1: not looked up yet)
};

static void cc_scratch_free(void* p)
{
  CcScratch* s = (CcScratch*) p;
  if (s->hwalked) cudaFreeHost(s->hwalked);
  delete s;
}

__device__ __forceinline__ uint32_t cc_find(uint32_t* parent, uint32_t v)
{
  // path halving; concurrent halving writes only ever point further up
  uint32_t p = parent[v];
  while (p != v)
  {
    uint32_t gp = parent[p];
    if (gp != p) parent[v] = gp;
    v = p;
    p = gp;
  }
  return v;
}

__device__ __forceinline__ void cc_union(uint32_t* parent, uint32_t a, uint32_t b)
{
  uint32_t ru = cc_find(parent, a), rv = cc_find(parent, b);
  while (ru != rv)
  {
    if (ru > rv) { uint32_t t = ru; ru = rv; rv = t; }
    // hook the larger root under the smaller one
    uint32_t old = atomicCAS(&parent[rv], rv, ru);
    if (old == rv) break;
    rv = cc_find(parent, old);
    ru = cc_find(parent, ru);
  }
}

// First round: a row starts under the least of itself and its neighbours, the
// first of its entries.  Parents only ever point to smaller positions, so plain
// stores make a forest; what a row leaves out here the later passes see.
// (Uniting with two neighbours in turn by compare-and-swap took 161 + 280 us on
// R-MAT 2^22; this takes 23 us, the link rounds 41 + 30.)
__global__ void k_cc_hook(const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ col, uint32_t nrows,
                          uint32_t* parent, uint32_t* least, uint32_t* deep)
{
  for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < nrows; u += gridDim.x * blockDim.x)
  {
    parent[u] = min(u, col[ptr[u]]);
    least[u] = 0xFFFFFFFFu;
  }
  if (blockIdx.x == 0 && threadIdx.x < kCcFlags) deep[threadIdx.x] = 0;
}

// Later rounds, each after a full compression: a row's tree and that of one
// more neighbour (spread over the row) are linked by a single atomicMin on the
// larger root, which may lose to a smaller parent set at the same time; no
// retries and no finds, since k_cc_rest unites what is lost.  The rounds after
// the second are for graphs whose giant component is not found by then: with
// it half formed, k_cc_rest would unite most edges one by one (R-MAT 2^22 after
// one round only: 4 ms).  They return at once when *giant_share says that
// kCcEnough of the samples are in it.
static constexpr uint32_t kCcLinks = 2, kCcMoreLinks = 2;
static constexpr uint32_t kCcSamples = 1024, kCcEnough = 900;
__global__ void k_cc_link(const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ col, uint32_t nrows, uint32_t round,
                          const uint32_t* __restrict__ giant_share, uint32_t* parent)
{
  if (giant_share && *giant_share >= kCcEnough) return;
  for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < nrows; u += gridDim.x * blockDim.x)
  {
    const uint32_t b = ptr[u], e = ptr[u + 1];
    // the last entry, the middle one, then the quarters
    const uint32_t c = col[round == 0 ? e - 1 : b + (uint32_t) ((uint64_t) (e - b) * (round == 1 ? 2 : round == 2 ? 1 : 3) / 4)];
    const uint32_t ru = parent[u], rv = parent[c];
    const uint32_t lo = min(ru, rv), hi = max(ru, rv);
    if (lo != hi && parent[hi] > lo) atomicMin(&parent[hi], lo);
  }
}

// The edges of the rows whose root is not the sampled giant root: a lane
// looks at a row each, the warp then walks the edges of those found together.
__global__ void __launch_bounds__(256)
k_cc_rest(const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ col, uint32_t nrows,
          const uint32_t* __restrict__ giant_ptr, uint32_t* parent, unsigned long long* walked)
{
  const uint32_t giant = *giant_ptr;
  const uint32_t lane = threadIdx.x & 31;
  unsigned long long rows = 0, edges = 0;
  for (uint32_t u0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); u0 < nrows; u0 += gridDim.x * blockDim.x)
  {
    const uint32_t u = u0 + lane;
    uint32_t b = 0, e = 0;
    const bool out = u < nrows && cc_find(parent, u) != giant;
    if (out)
    {
      b = ptr[u];
      e = ptr[u + 1];
      rows++;
      edges += e - b;
    }
    for (unsigned m = __ballot_sync(0xffffffffu, out); m; m &= m - 1)
    {
      const int src = __ffs(m) - 1;
      const uint32_t b0 = __shfl_sync(0xffffffffu, b, src), e0 = __shfl_sync(0xffffffffu, e, src);
      for (uint32_t i = b0 + lane; i < e0; i += 32) cc_union(parent, u0 + src, col[i]);
    }
  }
  rows = block_sum_u64(rows);
  edges = block_sum_u64(edges);
  if (threadIdx.x == 0 && rows)
  {
    atomicAdd(&walked[0], rows);
    atomicAdd(&walked[1], edges);
  }
}

__global__ void k_cc_probe(uint32_t nrows, uint32_t nsamples, uint64_t seed, const uint32_t* __restrict__ giant_share,
                           uint32_t* parent, uint32_t* out)
{
  if (giant_share && *giant_share >= kCcEnough) return;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nsamples; i += gridDim.x * blockDim.x)
  {
    uint64_t x = seed + 0x9E3779B97F4A7C15ull * (i + 1);
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    x ^= x >> 31;
    out[i] = cc_find(parent, (uint32_t) (x % nrows));
  }
}

// giant[0]: the most frequent root among the samples (ties: the smallest),
// giant[1]: how many they are.  One block counts them in a hash table in shared
// memory, a warp's equal ones with one addition.  again: after rounds that were
// skipped if the first sample had kCcEnough; nothing to do then.
__global__ void __launch_bounds__(kCcSamples) k_cc_giant(const uint32_t* __restrict__ probe, uint32_t* giant, int again)
{
  constexpr uint32_t kSlots = 2 * kCcSamples;
  __shared__ uint32_t key[kSlots], cnt[kSlots];
  __shared__ unsigned long long best;
  if (again && giant[1] >= kCcEnough) return;
  const uint32_t t = threadIdx.x;
  for (uint32_t i = t; i < kSlots; i += kCcSamples)
  {
    key[i] = 0xFFFFFFFFu;
    cnt[i] = 0;
  }
  if (t == 0) best = 0;
  __syncthreads();
  const uint32_t r = probe[t];
  const unsigned same = __match_any_sync(0xffffffffu, r);
  const bool leads = (int) (t & 31) == __ffs(same) - 1;
  uint32_t slot = (r * 0x9E3779B1u) % kSlots;
  if (leads)
  {
    for (;; slot = (slot + 1) % kSlots)
    {
      const uint32_t k = atomicCAS(&key[slot], 0xFFFFFFFFu, r);
      if (k == 0xFFFFFFFFu || k == r) break;
    }
    atomicAdd(&cnt[slot], __popc(same));
  }
  __syncthreads();
  if (leads) atomicMax(&best, (unsigned long long) cnt[slot] << 32 | (0xFFFFFFFFu - r));
  __syncthreads();
  if (t == 0)
  {
    giant[0] = 0xFFFFFFFFu - (uint32_t) best;
    giant[1] = (uint32_t) (best >> 32);
  }
}

// Full compression.  A chain longer than kCcWalk is cut short at that ancestor
// and reported in *deep; the second pass (second: after the first one) then
// walks what is left, and has nothing to do otherwise.  (Walking every chain to
// its end at once, 2^20 vertices hooked one under the other took 19 ms; finds
// with path halving cannot be used here, since a late halving store may
// overwrite what another thread has compressed already, and leave the vertex
// short of its root.)
static constexpr uint32_t kCcWalk = 512;
__global__ void k_cc_flatten(uint32_t nrows, const uint32_t* __restrict__ giant_share, uint32_t* parent, uint32_t* deep,
                             int second)
{
  if (giant_share && *giant_share >= kCcEnough) return;  // after a round that was skipped
  if (second && !*deep) return;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < nrows; v += gridDim.x * blockDim.x)
  {
    uint32_t r = v, p = parent[v], n = 0;
    while (p != r)
    {
      r = p;
      if (!second && ++n == kCcWalk)
      {
        *deep = 1;
        break;
      }
      p = parent[r];
    }
    parent[v] = r;
  }
}

// The least id of each tree (compressed): the lanes of a warp that share a
// root, most of them under the giant one, first take theirs together.
__global__ void k_cc_least(uint32_t nrows, const uint32_t* __restrict__ id_of_pos, const uint32_t* __restrict__ parent,
                           uint32_t* least)
{
  for (uint32_t u0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); u0 < nrows; u0 += gridDim.x * blockDim.x)
  {
    const uint32_t u = u0 + (threadIdx.x & 31);
    uint32_t r = 0xFFFFFFFFu, id = 0xFFFFFFFFu;
    if (u < nrows)
    {
      r = parent[u];
      id = id_of_pos[u];
    }
    const uint32_t first = __shfl_sync(0xffffffffu, r, 0);
    const uint32_t m = __reduce_min_sync(0xffffffffu, r == first ? id : 0xFFFFFFFFu);
    if (r == first) id = (threadIdx.x & 31) == 0 ? m : 0xFFFFFFFFu;
    if (id != 0xFFFFFFFFu && least[r] > id) atomicMin(&least[r], id);
  }
}

__global__ void k_cc_labels(uint32_t N, uint32_t nrows, const uint32_t* __restrict__ id_of_pos,
                            const uint32_t* __restrict__ parent, const uint32_t* __restrict__ least, uint32_t* label)
{
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < N; p += gridDim.x * blockDim.x)
  {
    const uint32_t id = id_of_pos[p];
    label[id] = p < nrows ? least[parent[p]] : id;
  }
}

// ---- literal BSP path (vertex 0 has edges) ---------------------------------

__global__ void k_ccb_init(uint32_t N, uint32_t nrows, const uint32_t* __restrict__ id_of_pos, uint32_t* lab,
                           uint32_t* msg, uint8_t* act)
{
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < N; p += gridDim.x * blockDim.x)
  {
    lab[p] = id_of_pos[p];  // init: label = vid, returns true (cc.h:28)
    msg[p] = id_of_pos[p];
    act[p] = p < nrows;     // regular vertices scatter
  }
}

// One thread per row: fold active in-neighbours in column order.
__global__ void k_ccb_step(const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ col, uint32_t nrows,
                           const uint8_t* __restrict__ act, uint8_t* next_act, const uint32_t* __restrict__ msg,
                           uint32_t* lab, uint32_t* next_msg, int* flag)
{
  for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < nrows; r += gridDim.x * blockDim.x)
  {
    uint32_t y = 0;
    bool touched = false;
    for (uint32_t i = ptr[r]; i < ptr[r + 1]; i++)
    {
      uint32_t c = col[i];
      if (!act[c]) continue;
      uint32_t m = msg[c];
      y = (y == 0) ? m : min(m, y);
      touched = true;
    }
    bool activated = false;
    if (touched)
    {
      uint32_t f = 0;
      f = (f == 0) ? y : min(y, f);  // combine(partial, A())
      uint32_t old = lab[r];
      uint32_t nl = min(old, f);
      lab[r] = nl;
      activated = nl != old;
    }
    next_act[r] = activated;
    if (activated) { next_msg[r] = lab[r]; *flag = 1; }
  }
}

__global__ void k_ccb_by_id(uint32_t N, const uint32_t* __restrict__ id_of_pos, const uint32_t* __restrict__ lab,
                            uint32_t* out)
{
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < N; p += gridDim.x * blockDim.x) out[id_of_pos[p]] = lab[p];
}

static int cc_scratch_build(la3g_graph* G, CcScratch* cs)
{
  LA3G_TRY(galloc(G, &cs->label, G->g.nslots));
  LA3G_TRY(galloc(G, &cs->flag, 1));
  LA3G_TRY(galloc(G, &cs->walked, 2));
  LA3G_CUDA(cudaHostAlloc(&cs->hwalked, 2 * sizeof(unsigned long long), cudaHostAllocDefault));
  return LA3G_OK;
}

static int cc_scratch(la3g_graph* G, CcScratch** out)
{
  return graph_scratch(G, kSlotCc, cc_scratch_free, out, [&](CcScratch* cs) { return cc_scratch_build(G, cs); });
}

}  // namespace la3g

using namespace la3g;

extern "C" int la3g_cc(la3g_graph* G, uint32_t* label_out, la3g_stats* st)
{
  if (!G) return set_error(LA3G_EINVAL, "null graph");
  DevGraph& g = G->g;
  if (g.directed()) return set_error(LA3G_EINVAL, "cc needs an undirected graph (load without LA3G_DIRECTED)");
  CallTimer T(G, st);
  CcScratch* cs = nullptr;
  LA3G_TRY(cc_scratch(G, &cs));
  cudaStream_t s = G->stream;
  const uint32_t N = g.nslots, nrows = g.nrows();
  if (cs->zero_has_edges < 0)
  {
    uint32_t p0 = 0;  // a property of the graph: looked up once
    LA3G_CUDA(cudaMemcpyAsync(&p0, g.pos_of_id, 4, cudaMemcpyDeviceToHost, s));
    LA3G_CUDA(cudaStreamSynchronize(s));
    cs->zero_has_edges = p0 < nrows ? 1 : 0;
  }
  const bool zero_has_edges = cs->zero_has_edges == 1;
  uint32_t iters = 0;
  bool rest_counted = false;
  uint32_t first = 0;  // link rounds before the first sample
  T.device_begin();
  if (!zero_has_edges && nrows)
  {
    if (!cs->parent)
    {
      GallocScope scope(G);
      LA3G_TRY(galloc(G, &cs->least, nrows));
      LA3G_TRY(galloc(G, &cs->deep, kCcFlags));
      LA3G_TRY(galloc(G, &cs->probe, kCcSamples));
      LA3G_TRY(galloc(G, &cs->giant, 2));
      LA3G_TRY(galloc(G, &cs->parent, nrows));  // last: it says that all are there
      scope.keep();
    }
    int nflat = 0;
    auto flatten = [&](const uint32_t* share) -> int {
      ProfileScope p("cc_flatten", s, 8.0 * nrows);
      for (int second = 0; second < 2; second++)
      {
        k_cc_flatten<<<grid_for(nrows, 256), 256, 0, s>>>(nrows, share, cs->parent, cs->deep + nflat, second);
        LA3G_LAUNCHED();
      }
      tls_launches++;
      nflat++;
      return LA3G_OK;
    };
    auto link = [&](uint32_t r, const uint32_t* share) -> int {
      // row offsets, one index, the two roots
      ProfileScope p("cc_link", s, (8.0 + 4.0 + 8.0) * nrows);
      k_cc_link<<<grid_for(nrows, 256), 256, 0, s>>>(g.in_ptr, g.in_col, nrows, r, share, cs->parent);
      LA3G_LAUNCHED();
      return LA3G_OK;
    };
    auto sample = [&](bool again) -> int {
      k_cc_probe<<<4, 256, 0, s>>>(nrows, kCcSamples, 0x5A3Dull, again ? cs->giant + 1 : nullptr, cs->parent, cs->probe);
      LA3G_LAUNCHED();
      k_cc_giant<<<1, kCcSamples, 0, s>>>(cs->probe, cs->giant, again ? 1 : 0);
      LA3G_LAUNCHED();
      tls_launches += 2;
      return LA3G_OK;
    };
    {
      // row offset, one index, the parent and the least id's start
      ProfileScope p("cc_hook", s, 16.0 * nrows);
      k_cc_hook<<<grid_for(nrows, 256), 256, 0, s>>>(g.in_ptr, g.in_col, nrows, cs->parent, cs->least, cs->deep);
      LA3G_LAUNCHED();
    }
    LA3G_TRY(flatten(nullptr));
    // rows of a few entries have hardly more neighbours to link with
    const bool sparse = g.nent < 3ull * nrows;
    const uint32_t rounds = sparse ? 1 : kCcLinks + kCcMoreLinks;
    first = sparse ? 1 : kCcLinks;
    for (uint32_t r = 0; r < rounds; r++)
    {
      const uint32_t* share = r < first ? nullptr : cs->giant + 1;
      LA3G_TRY(link(r, share));
      LA3G_TRY(flatten(share));
      if (r + 1 == first) LA3G_TRY(sample(false));
    }
    if (rounds > first) LA3G_TRY(sample(true));
    LA3G_CUDA(cudaMemsetAsync(cs->walked, 0, 16, s));
    {
      // every row: its root (4 B); the walked rows: offsets (8 B), and per edge
      // its index and the neighbour's root (8 B each), added once the walked
      // counts are back on the host
      ProfileScope p("cc_rest", s, 4.0 * nrows);
      k_cc_rest<<<grid_for(nrows, 256, num_sms() * 32), 256, 0, s>>>(g.in_ptr, g.in_col, nrows, cs->giant, cs->parent,
                                                                     cs->walked);
      LA3G_LAUNCHED();
    }
    LA3G_CUDA(cudaMemcpyAsync(cs->hwalked, cs->walked, 16, cudaMemcpyDeviceToHost, s));
    rest_counted = true;
    LA3G_TRY(flatten(nullptr));
    {
      // ids, roots and the labels by id
      ProfileScope p("cc_labels", s, 8.0 * nrows + 12.0 * N);
      k_cc_least<<<grid_for(nrows, 256), 256, 0, s>>>(nrows, g.id_of_pos, cs->parent, cs->least);
      LA3G_LAUNCHED();
      k_cc_labels<<<grid_for(N, 256), 256, 0, s>>>(N, nrows, g.id_of_pos, cs->parent, cs->least, cs->label);
      LA3G_LAUNCHED();
      tls_launches++;
    }
    iters = 1;
  }
  else if (!zero_has_edges)
  {
    k_cc_labels<<<grid_for(N, 256), 256, 0, s>>>(N, 0, g.id_of_pos, nullptr, nullptr, cs->label);
    LA3G_LAUNCHED();
    tls_launches++;
    iters = 1;
  }
  else
  {
    if (!cs->lab_pos)
    {
      GallocScope scope(G);
      LA3G_TRY(galloc(G, &cs->msg, 2 * (size_t) N));
      LA3G_TRY(galloc(G, &cs->active[0], N));
      LA3G_TRY(galloc(G, &cs->active[1], N));
      LA3G_TRY(galloc(G, &cs->lab_pos, N));  // last
      scope.keep();
    }
    uint32_t* msg[2] = {cs->msg, cs->msg + N};
    k_ccb_init<<<grid_for(N, 256), 256, 0, s>>>(N, nrows, g.id_of_pos, cs->lab_pos, msg[0], cs->active[0]);
    LA3G_LAUNCHED();
    int cur = 0;
    for (;;)
    {
      if (iters > 10000000) return set_error(LA3G_ETIMEOUT, "cc did not converge");
      LA3G_CUDA(cudaMemsetAsync(cs->flag, 0, 4, s));
      {
        ProfileScope p("cc_bsp_step", s, 4.0 * g.nent);
        k_ccb_step<<<grid_for(nrows, 256), 256, 0, s>>>(g.in_ptr, g.in_col, nrows, cs->active[cur], cs->active[cur ^ 1],
                                                        msg[cur], cs->lab_pos, msg[cur ^ 1], cs->flag);
        LA3G_LAUNCHED();
      }
      iters++;
      int f = 0;
      LA3G_CUDA(cudaMemcpyAsync(&f, cs->flag, 4, cudaMemcpyDeviceToHost, s));
      LA3G_CUDA(cudaStreamSynchronize(s));
      cur ^= 1;
      if (!f) break;
    }
    k_ccb_by_id<<<grid_for(N, 256), 256, 0, s>>>(N, g.id_of_pos, cs->lab_pos, cs->label);
    LA3G_LAUNCHED();
  }
  T.device_end();
  if (st)
  {
    st->iterations = iters;
    st->teps_edges = g.nent;
    st->edges_examined = g.nent;
    st->algo_bytes = (uint64_t) (4.0 * g.nent + 12.0 * N);
  }
  if (label_out) LA3G_CUDA(cudaMemcpyAsync(label_out, cs->label, (size_t) N * 4, cudaMemcpyDeviceToHost, s));
  LA3G_TRY(T.finish());
  if (rest_counted)
  {
    const double rest = 8.0 * (double) cs->hwalked[0] + 8.0 * (double) cs->hwalked[1];
    profile_add_bytes("cc_rest", rest);
    if (st)
    {
      // the hook and link rounds (16 and 20 B per row), a compression after
      // each and at the end (8 B), every row's root test (4 B), the walked
      // edges, the labels
      st->edges_examined = (uint64_t) (1 + first) * nrows + cs->hwalked[1];
      st->algo_bytes = (uint64_t) ((16.0 + 20.0 * first + 8.0 * (first + 2) + 4.0 + 8.0) * nrows + 12.0 * N + rest);
    }
  }
  return LA3G_OK;
}
