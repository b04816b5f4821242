// SSSP: the reference sssp app (src/apps/graph_analytics/sssp.cpp:11-37,
// sssp.h:11-46) on the device.
//
// Reference semantics kept exactly (np = 1, the optimizable path
// execute_, vertex_program_execute.hpp:55-163):
//   * dist is uint32 with INF = 2^31 - 1; gather = msg + weight in uint32
//     arithmetic; combine = min; apply = min and activates on change;
//   * iteration i relaxes the out-edges of the vertices activated in
//     iteration i - 1 (the root in iteration 0, if it has out-edges), with
//     the message each of them scattered when it was activated, into the
//     REGULAR rows only;
//   * after convergence the sink rows are computed once from every regular
//     vertex's final distance (activated or not, INF included) and from the
//     root's message if the root is a source (:131-148).
// Push relaxation uses atomicMin on dist: the value a row holds after the
// iteration is min(old, min over messages) exactly as apply computes it.  A
// row is activated iff some relaxation lowered it, i.e. iff its distance is
// now below its message (the distance it scattered when it was last
// activated; INF if never): one dense pass over the regular rows after each
// iteration finds those rows, scatters their new distance and forms the next
// frontier, so the relaxations themselves only do a non-returning atomicMin.
//
// All iterations run in one cooperative kernel with a grid barrier between its
// phases; every block decides for itself, from counters in global memory,
// whether an iteration pushes or pulls.  (As a graph with conditional nodes an
// iteration was five launches, 18 us on a graph whose iterations take a few us
// of work.)
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <vector>

#include <cub/device/device_radix_sort.cuh>

#include "frontier.cuh"
#include "la3g_internal.h"

namespace la3g {

static constexpr uint32_t kInf = 0x7FFFFFFFu;
static constexpr uint32_t kPullLong = 256;    // pull rows longer than this are cut into tasks
static constexpr uint32_t kPullChunk = 512;   // in-edges per long-row task (one warp)
static constexpr uint32_t kPullLanes = 4;     // lanes per short row in a pull step

struct SsspCounters  // what an iteration activates
{
  unsigned long long count, deg, out, fmin;  // vertices, their regular out-degrees' sum, those that have any, smallest message
};

struct SsspStats  // pinned, written by the kernel at its end
{
  unsigned long long iterations, examined, status, reached_deg;
};
static constexpr unsigned long long kSsspRunning = 2;  // status until the kernel has ended properly

struct SsspArgs
{
  // the graph: push CSR (regular rows first, up to reg_end), pull CSR (columns
  // and weights are read for the sinks, and in plain pull steps)
  const uint32_t *out_ptr, *out_row, *out_w, *reg_end, *in_ptr, *in_col, *in_w, *pos_of_id;
  uint32_t N, nreg, nsink, src_base, iso_base;
  uint64_t reg_in;                // in-edges of the regular rows
  uint32_t min_w, max_w;          // pull steps need INF + max_w to stay in uint32
  uint64_t limit;                 // most iterations
  // ordered pull steps: the regular rows' entries, slot of the column and weight,
  // each row in ascending order of weight >> wshift.  Slots number the columns by
  // descending out-degree: the hot ones' messages share sectors.  (Plain ones go
  // over the pull CSR; a column's slot is its position.)
  const uint32_t* slot;
  const uint2* entry;
  int wshift;
  // rows with more than kPullLong in-edges, cut into tasks of kPullChunk
  const uint32_t *task_row, *task_begin;  // row; [begins | ends]
  uint32_t ntasks;
  uint32_t* dist;
  uint32_t* msg;                  // the distance each vertex scattered at its last activation (INF if never)
  uint32_t* fmsg;                 // by slot: msg of the frontier a pull step reads, INF elsewhere
  uint32_t *fbits, *pbits;        // the current frontier; the one fmsg holds
  // push steps: the frontier's lists, vertices with at most kBigDeg regular
  // out-edges (one warp each) and hubs (their edges shared by the grid)
  uint32_t *small, *big, *big_task0;
  unsigned long long* fctr;       // [0] small-list length, [1] hub slots and tasks
  SsspCounters* ctr;              // [3]
  unsigned long long* reached;
  unsigned int* bar;
  long long wait_polls;
  uint32_t root;
  uint32_t* dist_out;             // by id, or null
  SsspStats* stats;
};

struct SsspScratch
{
  SsspArgs A{};
  SsspStats* stats = nullptr;     // pinned
  uint32_t* by_id = nullptr;      // [nslots] distances reordered by id before they leave the device
  uint32_t* reg_end = nullptr;    // [nslots] end of each vertex's out-edges into regular rows
  uint32_t* long_rows = nullptr;
  uint32_t nlong = 0;
  uint64_t reg_in = 0;
  uint32_t max_w = 0, min_w = 0;  // largest weight; smallest of a regular row's in-edge
  int rbits = 1, wbits = 1, wshift = 0;  // bits of a row, of a weight's leading bits; those below
  bool ordered = false;           // slot and entry are there
  bool order_failed = false;      // there was no memory for them
  unsigned grid[2] = {0, 0};      // plain, ordered
};

static void sssp_scratch_free(void* p)
{
  SsspScratch* s = (SsspScratch*) p;
  if (s->stats) cudaFreeHost(s->stats);
  delete s;
}

// End of the regular-row part of every out-edge list (rows ascend, so the
// sinks come last).
__global__ void k_sssp_reg_end(const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ row, uint32_t N,
                               uint32_t nreg, uint32_t* reg_end)
{
  for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < N; u += gridDim.x * blockDim.x)
  {
    uint32_t lo = ptr[u], hi = ptr[u + 1];
    while (lo < hi)
    {
      uint32_t mid = (lo + hi) >> 1;
      if (row[mid] < nreg) lo = mid + 1;
      else hi = mid;
    }
    reg_end[u] = lo;
  }
}

__device__ __forceinline__ void relax(uint32_t v, uint32_t cand, bool valid, uint32_t* dist)
{
  if (valid && cand < dist[v]) atomicMin(&dist[v], cand);  // result unused: a reduction in L2
}

// Relaxation over a split frontier: hubs first (all warps share each hub's
// edges), then one warp per small vertex.  Messages are the distances the
// frontier vertices held when they were activated (msg), as the reference's
// scatter values are.
__device__ __forceinline__ void sssp_push(const SsspArgs& A, uint32_t nsmall, unsigned long long packed, uint32_t warp,
                                          uint32_t nwarps, uint32_t lane)
{
  const uint32_t nbig = hub_count(packed), ntasks = hub_tasks(packed);
  for (uint32_t t = warp; t < ntasks; t += nwarps)
  {
    const uint32_t slot = hub_of_task(A.big_task0, nbig, t);
    const uint32_t u = A.big[slot], mu = A.msg[u];
    const uint32_t b = A.out_ptr[u] + (t - A.big_task0[slot]) * kHubTask;
    const uint32_t e = min(b + kHubTask, A.reg_end[u]);
    for (uint32_t i = b + lane; i < e; i += 32) relax(__ldg(&A.out_row[i]), mu + __ldg(&A.out_w[i]), true, A.dist);
  }
  for (uint32_t f = warp; f < nsmall; f += nwarps)
  {
    const uint32_t u = A.small[f], mu = A.msg[u];
    const uint32_t b = A.out_ptr[u], e = A.reg_end[u];
    for (uint32_t i = b + lane; i < e; i += 32) relax(__ldg(&A.out_row[i]), mu + __ldg(&A.out_w[i]), true, A.dist);
  }
}

// After an iteration: the regular rows whose distance fell below their
// message were activated.  They scatter (msg = dist) and form the next
// frontier, one bit per vertex (a warp writes a whole word, so every word of
// the bitmap is rewritten); the counters describe it.
__device__ __forceinline__ void sssp_dense_apply(const SsspArgs& A, uint32_t words, SsspCounters* ctr, uint32_t warp,
                                                 uint32_t nwarps, uint32_t lane)
{
  unsigned long long deg = 0;
  uint32_t cnt = 0, out = 0, fmin = 0xFFFFFFFFu;
  for (uint32_t w = warp; w < words; w += nwarps)
  {
    const uint32_t v = w * 32 + lane;
    bool act = false;
    if (v < A.nreg)
    {
      const uint32_t dv = A.dist[v];
      act = dv < A.msg[v];
      if (act)
      {
        A.msg[v] = dv;
        const uint32_t d = A.reg_end[v] - A.out_ptr[v];
        deg += d;
        cnt++;
        out += d != 0;
        fmin = min(fmin, dv);
      }
    }
    const unsigned m = __ballot_sync(0xffffffffu, act);
    if (lane == 0) A.fbits[w] = m;
  }
  const unsigned long long co = block_sum_u64((unsigned long long) cnt << 32 | out);
  deg = block_sum_u64(deg);
  fmin = block_min_u32(fmin);
  if (threadIdx.x == 0 && co)
  {
    atomicAdd(&ctr->count, co >> 32);
    atomicAdd(&ctr->out, co & 0xFFFFFFFFull);
    if (deg) atomicAdd(&ctr->deg, deg);
    atomicMin(&ctr->fmin, (unsigned long long) fmin);
  }
}

// Pull steps only: the frontier's messages by slot, INF again for the frontier
// of the last pull step.
template <bool ORDERED>
__device__ __forceinline__ void sssp_front(const SsspArgs& A, uint32_t words, uint32_t warp, uint32_t nwarps, uint32_t lane)
{
  for (uint32_t w = warp; w < words; w += nwarps)
  {
    const uint32_t now = A.fbits[w], was = A.pbits[w];
    if ((now | was) >> lane & 1)
    {
      const uint32_t v = w * 32 + lane;
      A.fmsg[ORDERED ? A.slot[v] : v] = now >> lane & 1 ? A.msg[v] : kInf;
    }
    __syncwarp();
    if (lane == 0 && now != was) A.pbits[w] = now;
  }
}

// Push steps only: the frontier bitmap into the split lists (vertices with
// up to kBigDeg regular out-edges, appended a warp at a time; hubs with their
// edge tasks).
__device__ __forceinline__ void sssp_split(const SsspArgs& A, uint32_t words, uint32_t warp, uint32_t nwarps, uint32_t lane)
{
  for (uint32_t w0 = warp * 32; w0 < words; w0 += nwarps * 32)
  {
    const uint32_t w = w0 + lane;
    uint32_t bits = w < words ? A.fbits[w] : 0u, c = 0;
    for (uint32_t x = bits; x; x &= x - 1)
    {
      const uint32_t v = w * 32 + (__ffs(x) - 1);
      const uint32_t d = A.reg_end[v] - A.out_ptr[v];
      if (d > kBigDeg) hub_append(v, d, A.big, A.big_task0, &A.fctr[1]);
      else c += d != 0;
    }
    uint32_t incl = c;
    for (int o = 1; o < 32; o <<= 1)
    {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= (uint32_t) o) incl += t;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    if (!total) continue;
    uint32_t base = 0;
    if (lane == 31) base = (uint32_t) atomicAdd(&A.fctr[0], (unsigned long long) total);
    base = __shfl_sync(0xffffffffu, base, 31) + incl - c;
    for (uint32_t x = bits; x; x &= x - 1)
    {
      const uint32_t v = w * 32 + (__ffs(x) - 1);
      const uint32_t d = A.reg_end[v] - A.out_ptr[v];
      if (d && d <= kBigDeg) A.small[base++] = v;
    }
  }
}

// Pull step (for large frontiers; the reference's own SpMV direction):
// every regular row takes the min over its in-neighbours in the frontier
// (the previous iteration's frontier lists) of msg + w, and is activated if
// that lowers it.  fmsg holds msg for the frontier and INF for every other
// vertex, so each edge is one load and one add: INF + w (w <= 2^31) stays
// above INF in uint32 and never lowers a row.  Short rows are owned by one
// lane group, long rows are cut into tasks that lower the row's distance by
// atomicMin; the messages are not written while the step runs.
// Sources are frontier vertices only in the first iteration, which always
// pushes.
//
// Every candidate of a step is at least the frontier's smallest message plus
// its edge's weight, and a row's entries ascend by weight (exactly, or by its
// leading bits), so a row is done as soon as that sum reaches what it already
// has: most of its edges' messages, random reads that bound the step at 240 G a
// second however they are arranged, are never read.  R-MAT 2^22: the five pulls
// of a call 1343 us over the CSR by position, 1095 with the messages by slot,
// 486 with the rows by weight.  The ordered copy takes 8 B per in-edge, and 16
// to 24 more while it is made: where the memory is not there, or not granted (a
// server's budget), the pulls go over the CSR.
__device__ __forceinline__ bool sssp_past(unsigned long long fmin, uint32_t w, int wshift, uint32_t have)
{
  return fmin + ((w >> wshift) << wshift) >= have;
}

__global__ void k_sssp_slot_keys(const uint32_t* __restrict__ ptr, uint32_t N, uint32_t* key, uint32_t* iota)
{
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < N; p += gridDim.x * blockDim.x)
  {
    key[p] = ~(ptr[p + 1] - ptr[p]);
    iota[p] = p;
  }
}

__global__ void k_sssp_slots(const uint32_t* __restrict__ order, uint32_t N, uint32_t* slot)
{
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) slot[order[i]] = i;
}

// Sort keys (row, leading bits of the weight) and values (slot, weight) of the
// regular rows' entries, a warp per row.
template <class K>
__global__ void __launch_bounds__(256)
k_sssp_entries(const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ col, const uint32_t* __restrict__ w,
               uint32_t nreg, const uint32_t* __restrict__ slot, int wbits, int wshift, K* key, uint2* entry)
{
  const uint32_t lane = threadIdx.x & 31, nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < nreg; r += nw)
    for (uint32_t e = ptr[r] + lane; e < ptr[r + 1]; e += 32)
    {
      key[e] = (K) r << wbits | (K) (w[e] >> wshift);
      entry[e] = make_uint2(slot[col[e]], w[e]);
    }
}

template <bool ORDERED>
__device__ __forceinline__ void sssp_pull(const SsspArgs& A, unsigned long long fmin, uint32_t warp, uint32_t nwarps,
                                          uint32_t lane)
{
  // Every candidate of this step is a frontier message plus a weight, so at
  // least fmin + min_w: a row already at or below that cannot be lowered and
  // its in-edges are not read (the result is the same).
  const uint32_t settled =
      fmin == ~0ull ? 0u : (fmin + A.min_w < kInf ? (uint32_t) (fmin + A.min_w) : kInf);
  const uint2* __restrict__ entry = A.entry;
  const uint32_t *__restrict__ col = A.in_col, *__restrict__ wgt = A.in_w;
  auto load = [&](uint32_t i) { return ORDERED ? __ldcs(&entry[i]) : make_uint2(__ldcs(&col[i]), __ldcs(&wgt[i])); };
  const uint32_t* fmsg = A.fmsg;
  // long rows first
  for (uint32_t t = warp; t < A.ntasks; t += nwarps)
  {
    uint32_t* const at = &A.dist[A.task_row[t]];
    // with what the row's other tasks found so far: one lane's read for all, since
    // they lower it meanwhile and the lanes leave the loops below together
    uint32_t y = 0;
    if (lane == 0) y = *(volatile uint32_t*) at;
    y = __shfl_sync(0xffffffffu, y, 0);
    if (y <= settled) continue;
    const uint32_t b = A.task_begin[t], e = A.task_begin[A.ntasks + t], had = y;
    for (uint32_t i0 = b; i0 < e; i0 += 128)
    {
      uint2 x[4];
      uint32_t m[4];
#pragma unroll
      for (int u = 0; u < 4; u++) x[u] = i0 + u * 32 + lane < e ? load(i0 + u * 32 + lane) : make_uint2(0u, kInf);
      if (ORDERED && sssp_past(fmin, __shfl_sync(0xffffffffu, x[0].y, 0), A.wshift, y)) break;
#pragma unroll
      for (int u = 0; u < 4; u++) m[u] = fmsg[x[u].x];
#pragma unroll
      for (int u = 0; u < 4; u++) y = min(y, m[u] + x[u].y);
      y = __reduce_min_sync(0xffffffffu, y);
    }
    if (lane == 0 && y < had) atomicMin(at, y);
  }
  // short rows: a group of kPullLanes lanes per row; each lane keeps four
  // independent loads in flight per step (entries, then messages), since the
  // step is bound by memory latency
  constexpr uint32_t G = kPullLanes;
  const uint32_t sub = lane & (G - 1), group = warp * (32 / G) + lane / G, ngroups = nwarps * (32 / G);
  const unsigned group_mask = ((1u << G) - 1) << (lane & ~(G - 1));
  for (uint32_t v = group; v < A.nreg; v += ngroups)
  {
    const uint32_t b = A.in_ptr[v], dv = A.dist[v];
    uint32_t e = A.in_ptr[v + 1], y = dv;  // y: the same in the group's lanes after each step
    if (e - b > kPullLong || dv <= settled) e = b;
    for (uint32_t i = b; i < e; i += 4 * G)
    {
      uint2 x[4];
      uint32_t m[4];
#pragma unroll
      for (uint32_t u = 0; u < 4; u++) x[u] = i + u * G + sub < e ? load(i + u * G + sub) : make_uint2(0u, kInf);
      if (ORDERED && sssp_past(fmin, __shfl_sync(group_mask, x[0].y, 0, G), A.wshift, y)) break;
#pragma unroll
      for (int u = 0; u < 4; u++) m[u] = fmsg[x[u].x];
#pragma unroll
      for (int u = 0; u < 4; u++) y = min(y, m[u] + x[u].y);
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) y = min(y, __shfl_xor_sync(group_mask, y, o));
    }
    if (sub == 0 && y < dv) A.dist[v] = y;
  }
}

__global__ void k_sssp_long_rows(const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ w, uint32_t nreg,
                                 uint32_t* list, unsigned long long* n, unsigned long long* edges, unsigned int* maxw,
                                 unsigned int* minw)
{
  unsigned long long s = 0;
  unsigned int mw = 0, lw = 0xFFFFFFFFu;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < nreg; v += gridDim.x * blockDim.x)
  {
    const uint32_t d = ptr[v + 1] - ptr[v];
    s += d;
    for (uint32_t i = ptr[v]; i < ptr[v + 1]; i++)
    {
      mw = max(mw, w[i]);
      lw = min(lw, w[i]);
    }
    if (d > kPullLong) list[atomicAdd(n, 1ull)] = v;
  }
  for (int o = 16; o > 0; o >>= 1)
  {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    mw = max(mw, __shfl_xor_sync(0xffffffffu, mw, o));
    lw = min(lw, __shfl_xor_sync(0xffffffffu, lw, o));
  }
  if ((threadIdx.x & 31) == 0)
  {
    if (s) atomicAdd(edges, s);
    if (mw) atomicMax(maxw, mw);
    if (lw != 0xFFFFFFFFu) atomicMin(minw, lw);
  }
}

// A step pulls when its frontier's out-degree sum exceeds the regular rows'
// in-edges / kPullDivisor (8 roots each: R-MAT 2^22 2: 8.2 ms, 4: 7.3, 8: 7.3;
// ER 2^22 2: 34.8, 4: 35.2, 8: 38.8).
static constexpr double kPullDivisor = 4.0;
static constexpr int kSsspThreads = 512;

template <bool ORDERED>
__global__ void __launch_bounds__(kSsspThreads, 3) k_sssp_run(SsspArgs A)
{
  __shared__ SsspCounters s_got;
  __shared__ unsigned long long s_list[2];
  GridBarrier bar{A.bar, A.wait_polls};
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
  const uint32_t lane = threadIdx.x & 31, warp = tid >> 5, nwarps = nth >> 5;
  const uint32_t words = A.N / 32 + 1;
  // The root (none if it is outside the graph): distance 0, scattered (msg 0);
  // regular and source vertices scatter, so they form the first frontier (even
  // with no regular out-edge: the first iteration runs).
  const uint32_t rp = A.root < A.N ? A.pos_of_id[A.root] : 0xFFFFFFFFu;
  const bool src = rp >= A.src_base && rp < A.iso_base, scatters = rp < A.nreg || src;
  for (uint32_t p = tid; p < A.N; p += nth)
  {
    A.dist[p] = A.msg[p] = p == rp ? 0u : kInf;
    A.fmsg[p] = kInf;
  }
  for (uint32_t w = tid; w < words; w += nth)
  {
    A.fbits[w] = scatters && w == rp >> 5 ? 1u << (rp & 31) : 0u;
    A.pbits[w] = 0;
  }
  if (tid == 0)
  {
    for (int k = 0; k < 3; k++) A.ctr[k] = SsspCounters{0, 0, 0, ~0ull};
    A.fctr[0] = A.fctr[1] = *A.reached = 0;
  }
  if (!bar.sync()) return;
  // the loop's state, the same in every thread.  It ends as the reference's
  // execute loop does: nothing activated, or activated vertices with no
  // regular out-edge, which take one more, empty iteration.
  unsigned long long it = 0, examined = 0, nlist = scatters, deg = scatters ? A.reg_end[rp] - A.out_ptr[rp] : 0, fmin = ~0ull;
  bool failed = false;
  for (;;)
  {
    if (it > A.limit)
    {
      failed = true;
      break;
    }
    it++;
    if (!nlist) break;
    SsspCounters* const next = A.ctr + it % 3;
    if (tid == 0) A.ctr[(it + 1) % 3] = SsspCounters{0, 0, 0, ~0ull};  // read last before the barrier just passed
    if (it > 1 && A.max_w <= 0x80000000u && (double) deg * kPullDivisor > (double) A.reg_in)
    {
      examined += A.reg_in;
      sssp_front<ORDERED>(A, words, warp, nwarps, lane);
      if (!bar.sync()) return;
      sssp_pull<ORDERED>(A, fmin, warp, nwarps, lane);
    }
    else
    {
      examined += deg;
      sssp_split(A, words, warp, nwarps, lane);
      if (!bar.sync()) return;
      if (threadIdx.x < 2) s_list[threadIdx.x] = __ldcg(&A.fctr[threadIdx.x]);
      __syncthreads();
      sssp_push(A, (uint32_t) s_list[0], s_list[1], warp, nwarps, lane);
    }
    if (!bar.sync()) return;
    if (tid == 0) A.fctr[0] = A.fctr[1] = 0;
    sssp_dense_apply(A, words, next, warp, nwarps, lane);
    if (!bar.sync()) return;
    if (threadIdx.x == 0) s_got = {__ldcg(&next->count), __ldcg(&next->deg), __ldcg(&next->out), __ldcg(&next->fmin)};
    __syncthreads();
    const unsigned long long count = s_got.count;
    deg = s_got.deg;
    nlist = s_got.out;
    fmin = s_got.fmin;
    __syncthreads();  // s_got is free
    if (!count) break;
  }
  // Sink pass: y = min over in-neighbours (regular: final dist; the root if it
  // is a source: its message 0) of msg + w; dist = min(dist, y).
  for (uint32_t v = A.nreg + tid; v < A.nreg + A.nsink; v += nth)
  {
    uint32_t y = kInf;
    for (uint32_t i = A.in_ptr[v]; i < A.in_ptr[v + 1]; i++)
    {
      const uint32_t c = A.in_col[i];
      uint32_t cand;
      if (c < A.nreg) cand = A.dist[c] + A.in_w[i];
      else if (src && c == rp) cand = A.in_w[i];
      else continue;
      y = min(y, cand);
    }
    if (y < A.dist[v]) A.dist[v] = y;
  }
  if (!bar.sync()) return;
  unsigned long long r = 0;
  for (uint32_t i = tid; i < A.N; i += nth)
  {
    if (A.dist_out) A.dist_out[i] = A.dist[A.pos_of_id[i]];
    if (A.dist[i] != kInf) r += A.out_ptr[i + 1] - A.out_ptr[i];
  }
  r = block_sum_u64(r);
  if (threadIdx.x == 0 && r) atomicAdd(A.reached, r);
  if (!bar.sync()) return;
  if (tid == 0) *A.stats = SsspStats{it, examined, failed ? 1ull : 0ull, __ldcg(A.reached)};
}

static int sssp_scratch_build(la3g_graph* G, SsspScratch* ss)
{
  DevGraph& g = G->g;
  cudaStream_t s = G->stream;
  const uint32_t N = g.nslots;
  SsspArgs& A = ss->A;
  LA3G_TRY(galloc(G, &A.dist, N));
  LA3G_TRY(galloc(G, &A.msg, N));
  LA3G_TRY(galloc(G, &A.fmsg, N));
  LA3G_TRY(galloc(G, &ss->reg_end, N));
  LA3G_TRY(galloc(G, &A.small, N));
  LA3G_TRY(galloc(G, &A.big, N));
  LA3G_TRY(galloc(G, &A.big_task0, N));
  LA3G_TRY(galloc(G, &A.ctr, 3));
  LA3G_TRY(galloc(G, &A.fctr, 4));  // with `reached` and the barrier
  A.reached = A.fctr + 2;
  A.bar = (unsigned int*) (A.fctr + 3);
  LA3G_TRY(galloc(G, &A.fbits, (size_t) N / 32 + 2));
  LA3G_TRY(galloc(G, &A.pbits, (size_t) N / 32 + 2));
  LA3G_TRY(galloc(G, &ss->by_id, N));
  LA3G_CUDA(cudaHostAlloc(&ss->stats, sizeof(SsspStats), cudaHostAllocMapped));
  k_sssp_reg_end<<<grid_for(N, 256), 256, 0, s>>>(g.out_ptr, g.out_row, N, g.nreg, ss->reg_end);
  LA3G_LAUNCHED();
  LA3G_TRY(galloc(G, &ss->long_rows, std::max<uint32_t>(g.nreg, 1)));
  {
    // [0] long rows [1] regular in-edges [2] largest weight [3] smallest
    unsigned long long* c = (unsigned long long*) A.ctr;
    unsigned long long h[4];
    LA3G_CUDA(cudaMemsetAsync(c, 0, 3 * sizeof(unsigned long long), s));
    LA3G_CUDA(cudaMemsetAsync(c + 3, 0xFF, sizeof(unsigned long long), s));
    k_sssp_long_rows<<<grid_for(g.nreg, 256), 256, 0, s>>>(g.in_ptr, g.in_w, g.nreg, ss->long_rows, c, c + 1,
                                                           (unsigned int*) (c + 2), (unsigned int*) (c + 3));
    LA3G_LAUNCHED();
    LA3G_CUDA(cudaMemcpyAsync(h, c, sizeof h, cudaMemcpyDeviceToHost, s));
    LA3G_CUDA(cudaStreamSynchronize(s));
    ss->nlong = (uint32_t) h[0];
    ss->reg_in = h[1];
    ss->max_w = (uint32_t) h[2];
    ss->min_w = (uint32_t) h[3];
  }
  if (ss->nlong)
  {
    // cut the long rows into tasks of kPullChunk in-edges (host side: few rows)
    std::vector<uint32_t> rows(ss->nlong), ptr((size_t) g.nreg + 1);
    LA3G_CUDA(cudaMemcpy(rows.data(), ss->long_rows, ss->nlong * 4, cudaMemcpyDeviceToHost));
    LA3G_CUDA(cudaMemcpy(ptr.data(), g.in_ptr, ptr.size() * 4, cudaMemcpyDeviceToHost));
    std::vector<uint32_t> trow, tbeg, tend;
    for (uint32_t r : rows)
      for (uint64_t x = ptr[r]; x < ptr[r + 1]; x += kPullChunk)
      {
        trow.push_back(r);
        tbeg.push_back((uint32_t) x);
        tend.push_back((uint32_t) std::min<uint64_t>(x + kPullChunk, ptr[r + 1]));
      }
    const size_t nt = trow.size();
    uint32_t *row = nullptr, *be = nullptr;
    LA3G_TRY(galloc(G, &row, nt));
    LA3G_TRY(galloc(G, &be, 2 * nt));
    LA3G_CUDA(cudaMemcpy(row, trow.data(), nt * 4, cudaMemcpyHostToDevice));
    LA3G_CUDA(cudaMemcpy(be, tbeg.data(), nt * 4, cudaMemcpyHostToDevice));
    LA3G_CUDA(cudaMemcpy(be + nt, tend.data(), nt * 4, cudaMemcpyHostToDevice));
    A.task_row = row;
    A.task_begin = be;
    A.ntasks = (uint32_t) nt;
  }
  while ((uint64_t) g.nreg >> ss->rbits) ss->rbits++;
  while (ss->wbits < 32 && ss->max_w >> ss->wbits) ss->wbits++;
  // eight leading bits of the weight order a row well enough
  ss->wshift = std::max(0, ss->wbits - 8);
  ss->wbits -= ss->wshift;
  A.out_ptr = g.out_ptr;
  A.out_row = g.out_row;
  A.out_w = g.out_w;
  A.reg_end = ss->reg_end;
  A.in_ptr = g.in_ptr;
  A.in_col = g.in_col;
  A.in_w = g.in_w;
  A.pos_of_id = g.pos_of_id;
  A.N = N;
  A.nreg = g.nreg;
  A.nsink = g.nsink;
  A.src_base = g.src_base();
  A.iso_base = g.iso_base();
  A.reg_in = ss->reg_in;
  A.min_w = ss->min_w;
  A.max_w = ss->max_w;
  // with non-negative weights every distance is final after at most N + 1
  // iterations (Bellman-Ford), so a loop past N + 2 is a fault
  A.limit = (uint64_t) N + 2;
  A.wshift = ss->wshift;
  A.stats = ss->stats;
  LA3G_CUDA(cudaStreamSynchronize(s));
  return LA3G_OK;
}

static int sssp_scratch(la3g_graph* G, SsspScratch** out)
{
  LA3G_TRY(build_push_csr(G));
  return graph_scratch(G, kSlotSssp, sssp_scratch_free, out, [&](SsspScratch* ss) { return sssp_scratch_build(G, ss); });
}

// The ordered pull's arrays; rows ascend by position, so the regular rows'
// entries come first.  First the slots' sort, then the entries', in the same
// temporary memory.
template <class K>
static int sssp_order(la3g_graph* G, SsspScratch* ss)
{
  DevGraph& g = G->g;
  cudaStream_t s = G->stream;
  const size_t N = g.nslots, m = ss->reg_in;
  auto round = [](size_t b) { return (b + 255) & ~(size_t) 255; };
  const size_t n4 = round(N * 4), kb = round(m * sizeof(K)), vb = round(m * 8);
  size_t slot_lib = 0, entry_lib = 0;
  {
    uint32_t* z = nullptr;
    cub::DoubleBuffer<K> k(nullptr, nullptr);
    cub::DoubleBuffer<uint2> v(nullptr, nullptr);
    LA3G_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, slot_lib, z, z, z, z, (int64_t) N, 0, 32, s));
    if (m) LA3G_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, entry_lib, k, v, (int64_t) m, 0, ss->rbits + ss->wbits, s));
  }
  GallocScope scope(G);
  uint32_t* slot = nullptr;
  uint2* entry = nullptr;
  LA3G_TRY(galloc(G, &slot, N));
  LA3G_TRY(galloc(G, &entry, m + 1));
  DevBuf tmp;
  LA3G_TRY(tmp.alloc(std::max(4 * n4 + slot_lib, 2 * kb + vb + entry_lib)));
  char* p = tmp.as<char>();
  {
    uint32_t *key = (uint32_t*) p, *key2 = (uint32_t*) (p + n4), *iota = (uint32_t*) (p + 2 * n4);
    uint32_t* order = (uint32_t*) (p + 3 * n4);
    k_sssp_slot_keys<<<grid_for(N, 256), 256, 0, s>>>(g.out_ptr, (uint32_t) N, key, iota);
    LA3G_LAUNCHED();
    LA3G_CUDA(cub::DeviceRadixSort::SortPairs(p + 4 * n4, slot_lib, key, key2, iota, order, (int64_t) N, 0, 32, s));
    k_sssp_slots<<<grid_for(N, 256), 256, 0, s>>>(order, (uint32_t) N, slot);
    LA3G_LAUNCHED();
  }
  if (m)
  {
    cub::DoubleBuffer<K> k((K*) p, (K*) (p + kb));
    cub::DoubleBuffer<uint2> v(entry, (uint2*) (p + 2 * kb));
    k_sssp_entries<K><<<grid_for((uint64_t) g.nreg * 32, 256), 256, 0, s>>>(g.in_ptr, g.in_col, g.in_w, g.nreg, slot,
                                                                            ss->wbits, ss->wshift, k.Current(), v.Current());
    LA3G_LAUNCHED();
    LA3G_CUDA(cub::DeviceRadixSort::SortPairs(p + 2 * kb + vb, entry_lib, k, v, (int64_t) m, 0, ss->rbits + ss->wbits, s));
    if (v.Current() != entry) LA3G_CUDA(cudaMemcpyAsync(entry, v.Current(), m * 8, cudaMemcpyDeviceToDevice, s));
  }
  LA3G_CUDA(cudaStreamSynchronize(s));  // before the temporaries go
  scope.keep();
  ss->A.slot = slot;
  ss->A.entry = entry;
  ss->ordered = true;
  return LA3G_OK;
}

int sssp_run(la3g_graph* G, uint32_t root, uint32_t* dist_out, la3g_stats* st, bool order)
{
  if (!G) return set_error(LA3G_EINVAL, "null graph");
  DevGraph& g = G->g;
  if (!g.directed() || !g.weighted() || (g.flags & (LA3G_REVERSE | LA3G_ACYCLIC | LA3G_BIPARTITE)))
    return set_error(LA3G_EINVAL, "sssp needs a graph loaded with LA3G_DIRECTED | LA3G_WEIGHTED");
  CallTimer T(G, st);
  SsspScratch* ss = nullptr;
  LA3G_TRY(sssp_scratch(G, &ss));
  if (order && !ss->ordered && !ss->order_failed)
  {
    const int rc = ss->rbits + ss->wbits <= 32 ? sssp_order<uint32_t>(G, ss) : sssp_order<uint64_t>(G, ss);
    if (rc != LA3G_OK && rc != LA3G_ENOMEM) return rc;
    ss->order_failed = rc == LA3G_ENOMEM;  // the plain pulls give the same
  }
  cudaStream_t s = G->stream;
  const uint32_t N = g.nslots;
  const void* kernel = ss->ordered ? (const void*) k_sssp_run<true> : (const void*) k_sssp_run<false>;
  unsigned& grid = ss->grid[ss->ordered];
  SsspArgs A = ss->A;
  A.root = root;
  A.wait_polls = barrier_polls(G->wait_polls, g.nent);
  A.dist_out = dist_out ? ss->by_id : nullptr;
  ss->stats->status = kSsspRunning;
  if (!grid)  // few blocks for a small graph: a barrier takes longer the more there are
    LA3G_TRY(cooperative_blocks(kernel, kSsspThreads, std::max<uint64_t>(N, g.nent / 8), 3, &grid));
  T.device_begin();
  LA3G_CUDA(cudaMemsetAsync(A.bar, 0, sizeof *A.bar, s));
  {
    // distances and messages; the edges examined are added below
    ProfileScope p("sssp", s, 8.0 * N);
    void* args[] = {(void*) &A};
    LA3G_CUDA(cudaLaunchCooperativeKernel(kernel, grid, kSsspThreads, args, 0, s));
  }
  T.device_end();
  if (dist_out) LA3G_CUDA(cudaMemcpyAsync(dist_out, ss->by_id, (size_t) N * 4, cudaMemcpyDeviceToHost, s));
  LA3G_TRY(T.finish());
  const SsspStats r = *ss->stats;
  if (r.status == kSsspRunning) return set_error(LA3G_ETIMEOUT, "sssp: a grid barrier wait ran out");
  if (r.status) return set_error(LA3G_ETIMEOUT, "sssp did not converge");
  profile_add_bytes("sssp", 8.0 * (double) r.examined);
  if (st)
  {
    st->iterations = (uint32_t) r.iterations;
    st->edges_examined = r.examined;
    st->teps_edges = r.reached_deg;
    st->algo_bytes = r.examined * 8 + (uint64_t) N * 8;
  }
  return LA3G_OK;
}

}  // namespace la3g

using namespace la3g;

extern "C" int la3g_sssp(la3g_graph* G, uint32_t root, uint32_t* dist_out, la3g_stats* st)
{
  return sssp_run(G, root, dist_out, st, true);
}
