// Top-k over 64-bit keys (value in the high half, ~id in the low half, so
// that ties go to the smaller id), used by BM25, LM and the degree app, and
// the kernels the two information-retrieval apps share, BM25 (bm25.cu) and
// LM (lm.cu), over a bipartite corpus: docs 1..D then terms D+1..D+T,
// identity hash, so positions ascend with ids and a term's pull row lists
// its docs ascending.  The kernels are defined in bm25.cu.
#ifndef LA3G_IR_CUH
#define LA3G_IR_CUH

#include <algorithm>
#include <cstdint>
#include <cstring>

#include "la3g_internal.h"

namespace la3g {

constexpr int kTopKMax = 64;       // largest k of a top-k query
constexpr int kTopThreads = 128;   // threads of the top-k blocks (degree app)
constexpr int kTopBlocks = 2 * 152;  // partial top-k blocks (two per SM of a GB300)

// Block-level top-k of a key stream: each thread keeps its k best keys, the
// block then extracts the k largest by repeated block-wide max.
static __device__ void block_topk(unsigned long long* mine, int k, unsigned long long* out)
{
  __shared__ unsigned long long s_best[kTopThreads];
  __shared__ int s_who[kTopThreads];
  for (int r = 0; r < k; r++)
  {
    unsigned long long m = 0;
    int mi = -1;
    for (int i = 0; i < k; i++)
      if (mine[i] > m) { m = mine[i]; mi = i; }
    s_best[threadIdx.x] = m;
    s_who[threadIdx.x] = threadIdx.x;
    __syncthreads();
    for (int o = kTopThreads / 2; o > 0; o >>= 1)
    {
      if ((int) threadIdx.x < o && s_best[threadIdx.x + o] > s_best[threadIdx.x])
      {
        s_best[threadIdx.x] = s_best[threadIdx.x + o];
        s_who[threadIdx.x] = s_who[threadIdx.x + o];
      }
      __syncthreads();
    }
    unsigned long long top = s_best[0];
    int who = s_who[0];
    __syncthreads();
    if (threadIdx.x == 0) out[r] = top;
    if ((int) threadIdx.x == who && mi >= 0 && top != 0) mine[mi] = 0;
    __syncthreads();
  }
}

static __device__ __forceinline__ void keep_best(unsigned long long* mine, int k, unsigned long long key)
{
  int mi = 0;
  unsigned long long mv = mine[0];
  for (int i = 1; i < k; i++)
    if (mine[i] < mv) { mv = mine[i]; mi = i; }
  if (key > mv) mine[mi] = key;
}

// Sum of (float) tf over rows [row_lo, row_hi), ascending entry order, then
// length = sum (avg == 0) or BM25's K(d) (avg > 0).
__global__ void k_bm25_dl(const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ w, uint32_t row_lo,
                          uint32_t row_hi, float avg, float* length);
// Sum over positions of (uint64) length (values <= -1 count as 0).
__global__ void k_bm25_tokens(const float* __restrict__ length, uint32_t n, unsigned long long* out);
// StreamingArray push emulation of a query's term list: (position, value)
// pairs ascending by position in out[1..], count in out[0].
__global__ void k_bm25_pair(const uint32_t* __restrict__ q, uint32_t nq, uint32_t nslots, uint32_t nreg,
                            const uint32_t* __restrict__ pos_of_id, const float* __restrict__ length, uint32_t* out);
__global__ void k_f32_by_id(uint32_t N, const uint32_t* __restrict__ id_of_pos, const float* __restrict__ v, float* out);


// ---- one query, one kernel ---------------------------------------------------
//
// A doc's score is a float sum over the query's terms in ascending order, so
// the terms of one doc follow one another, but docs are independent: a block
// takes a chunk of consecutive positions, finds each term's postings in it
// (rows ascend: a 16-way search per term and end), adds them term by term into
// shared memory, one __syncthreads between terms, and extracts the chunk's top
// k; the last block to finish merges the blocks' lists.  Nothing per document
// touches global memory but the postings and the doc's own value.  A launch
// per term into global scores, an append to a touched list per doc and two
// top-k launches took 142 us a query (16 queries of 2 to 8 terms, 500k docs);
// this takes 42 us, 22 of them on the device.
constexpr int kIrThreads = 256;
constexpr uint32_t kIrChunk = 8192;     // most positions of a chunk (40 KB of shared memory)
constexpr uint32_t kIrMinChunk = 1024;  // fewest, unless the corpus is smaller
constexpr uint32_t kIrTerms = 64;       // terms handled at a time
constexpr int kIrPer = 4;               // postings of a thread in flight
constexpr uint32_t kIrCap = 256;        // keys listed by a top-k selection

struct IrResult  // pinned, written by the kernel
{
  unsigned long long ntouched, postings;
  unsigned long long best[kTopKMax];
};

struct IrScratch
{
  unsigned long long* ctr = nullptr;   // [0] touched [1] postings [2] blocks done; zero between queries
  unsigned long long* cand = nullptr;  // [blocks][k]
  IrResult* out = nullptr;
  uint32_t* qin = nullptr;             // longer queries: vertex ids, then k_bm25_pair's output
  uint32_t* qpos = nullptr;
  uint32_t qcap = 0;
};

// The query's term list: up to kIrTerms vertex ids by value, or the list
// k_bm25_pair made of a longer one.
struct IrQuery
{
  uint32_t n;
  const uint32_t* pairs;
  uint32_t vid[kIrTerms];
};

// Order of the answers: score desc, id asc.  The keys carry positions: the
// regular positions of a corpus (identity hash) ascend with their ids.
static __device__ __forceinline__ unsigned long long ir_key(float s, uint32_t pos)
{
  // order-preserving map of the score (with -0 == +0), then smaller id first
  uint32_t u = __float_as_uint(s);
  if ((u & 0x7FFFFFFFu) == 0) u = 0;
  u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
  return ((unsigned long long) u << 32) | (0xFFFFFFFFu - pos);
}

// First index of the ascending a[b, e) with a value of at least v, by 16
// lanes (half a warp) together.
static __device__ __forceinline__ uint32_t ir_search(const uint32_t* __restrict__ a, uint32_t b, uint32_t e, uint32_t v)
{
  const uint32_t lane = threadIdx.x & 15, half = threadIdx.x & 16;
  const unsigned mask = 0xFFFFu << half;
  while (e - b > 16)
  {
    const uint32_t n = e - b;
    const uint32_t p = b + (uint32_t) ((uint64_t) n * (lane + 1) / 17);
    const uint32_t less = __popc(__ballot_sync(mask, a[p] < v) >> half & 0xFFFFu);  // ascending: the first `less` probes
    const uint32_t lo = less ? b + (uint32_t) ((uint64_t) n * less / 17) + 1 : b;
    e = less < 16 ? b + (uint32_t) ((uint64_t) n * (less + 1) / 17) : e;
    b = lo;
  }
  return b + __popc(__ballot_sync(mask, b + lane < e && a[b + lane] < v) >> half & 0xFFFFu);
}

// The k largest of key(0 .. n - 1) into out[0, k), in order and filled up with
// zeros, by the whole block; keys differ, but for zeros, which do not count.
// `best` is the thread's largest key and list(T, push) gives push the thread's
// keys of at least T.  A threshold that at least k threads' best reach is
// looked for downwards from the largest key, then by bisection, one
// __syncthreads_count a step; at least k keys reach it, and seldom many more,
// so those are listed and each takes the place that the number of larger ones
// gives it.  If the list overflows, a bisection counts all keys.
struct IrTop
{
  unsigned long long list[kIrCap];
  uint32_t n, max;
};

template <class Key, class List>
static __device__ __forceinline__ void ir_topk(uint32_t n, Key key, unsigned long long best, List list, int k, IrTop& S,
                                               unsigned long long* out)
{
  const uint32_t tid = threadIdx.x, mine = (uint32_t) (best >> 32);
  if (tid == 0) S.n = S.max = 0;
  for (int r = tid; r < k; r += kIrThreads) out[r] = 0;
  const int have = __syncthreads_count(best != 0), enough = k + 22;
  uint32_t t = 0;
  if (have > enough)
  {
    const uint32_t wmax = __reduce_max_sync(0xffffffffu, mine);
    if ((tid & 31) == 0) atomicMax(&S.max, wmax);
    __syncthreads();
    // [t, hi): more than `enough` threads reach t, fewer than k reach hi; the
    // first steps down are an eighth of a binade of the score, then twice as far
    uint32_t hi = S.max + 1, down = 1u << 20;
    while (hi - t > 1)
    {
      const uint32_t mid = down && hi - t > down ? hi - down : t + (hi - t) / 2;
      const int c = __syncthreads_count(mine >= mid);
      if (c < k) hi = mid;
      else t = mid;
      if (c >= k && c <= enough) break;
      down = c < k ? down << 1 : 0;
    }
  }
  const unsigned long long T = max((unsigned long long) t << 32, 1ull);
  if (best >= T)
    list(T, [&](unsigned long long x) {
      const uint32_t at = atomicAdd(&S.n, 1u);
      if (at < kIrCap) S.list[at] = x;
    });
  __syncthreads();
  uint32_t m = S.n;
  if (m > kIrCap)
  {
    // all keys counted: `lo` becomes the largest value that k keys reach
    unsigned long long lo = T, hi = ~0ull;
    while (hi - lo > 1)
    {
      const unsigned long long mid = lo + (hi - lo) / 2;
      __syncthreads();
      if (tid == 0) S.n = 0;
      __syncthreads();
      uint32_t c = 0;
      for (uint32_t i = tid; i < n; i += kIrThreads) c += key(i) >= mid;
      if (c) atomicAdd(&S.n, c);
      __syncthreads();
      if (S.n < (uint32_t) k) hi = mid;
      else lo = mid;
    }
    __syncthreads();
    if (tid == 0) S.n = 0;
    __syncthreads();
    for (uint32_t i = tid; i < n; i += kIrThreads)
    {
      const unsigned long long x = key(i);
      if (x >= lo) S.list[atomicAdd(&S.n, 1u)] = x;  // exactly k of them: keys differ
    }
    __syncthreads();
    m = S.n;
  }
  for (uint32_t i = tid; i < m; i += kIrThreads)
  {
    const unsigned long long x = S.list[i];
    uint32_t rank = 0;
#pragma unroll 8
    for (uint32_t j = 0; j < m; j++) rank += S.list[j] > x;
    if (rank < (uint32_t) k) out[rank] = x;
  }
  __syncthreads();
}

// Scorer: `own` is a position's own value, `term` is one posting's contribution, `value` a term's pushed value
// prepared for it, `done` the final score of a touched position.
template <class Scorer>
__global__ void __launch_bounds__(kIrThreads)
k_ir_query(IrQuery Q, Scorer S, const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ col,
           const uint32_t* __restrict__ w, uint32_t nslots, uint32_t nreg, uint32_t chunk,
           const uint32_t* __restrict__ pos_of_id, const uint32_t* __restrict__ id_of_pos,
           const float* __restrict__ length, uint32_t leftover_from, int k, unsigned long long* ctr,
           unsigned long long* cand, IrResult* out, float* all, uint8_t* act)
{
  extern __shared__ __align__(16) unsigned char ir_smem[];
  float* score = (float*) ir_smem;                  // [chunk]
  uint8_t* touched = (uint8_t*) (score + chunk);    // [chunk]
  __shared__ IrTop s_top;
  __shared__ unsigned long long s_best[kTopKMax], s_new[kTopKMax];
  __shared__ uint32_t s_t[kIrTerms], s_lo[kIrTerms], s_hi[kIrTerms], s_in[kIrTerms], s_end[kIrTerms], s_cnt, s_touched, s_last;
  __shared__ float s_v[kIrTerms];
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) s_cnt = s_touched = 0;
  for (int r = tid; r < k; r += kIrThreads) s_best[r] = 0;
  __syncthreads();
  uint32_t cnt;
  if (Q.pairs) cnt = Q.pairs[0];
  else
  {
    // StreamingArray push emulation (k_bm25_pair): the j-th smallest of the
    // distinct regular positions takes the value of the j-th distinct push
    uint32_t p = 0xFFFFFFFFu;
    if (tid < Q.n && Q.vid[tid] < nslots) p = pos_of_id[Q.vid[tid]];
    if (p >= nreg) p = 0xFFFFFFFFu;
    if (tid < kIrTerms) s_in[tid] = p;
    __syncthreads();
    bool first = tid < Q.n && p != 0xFFFFFFFFu;
    for (uint32_t j = 0; first && j < tid; j++) first = s_in[j] != p;
    __syncthreads();
    if (tid < kIrTerms && !first) s_in[tid] = 0xFFFFFFFFu;
    __syncthreads();
    if (first)
    {
      uint32_t slot = 0, rank = 0;
      for (uint32_t j = 0; j < Q.n; j++)
      {
        slot += j < tid && s_in[j] != 0xFFFFFFFFu;
        rank += s_in[j] < p;
      }
      s_t[rank] = p;
      s_v[slot] = S.value(length[p]);
      atomicAdd(&s_cnt, 1u);
    }
    __syncthreads();
    cnt = s_cnt;
  }
  unsigned long long postings = 0;
  for (uint32_t c = blockIdx.x; (uint64_t) c * chunk < nreg; c += gridDim.x)
  {
    const uint32_t lo = c * chunk, n = min(chunk, nreg - lo);
    for (uint32_t i = tid; i < n; i += kIrThreads)
    {
      score[i] = 0.0f;
      touched[i] = 0;
    }
    for (uint32_t t0 = 0; t0 < cnt; t0 += kIrTerms)
    {
      const uint32_t nt = min(kIrTerms, cnt - t0);
      if (Q.pairs)
      {
        __syncthreads();
        if (tid < nt)
        {
          s_t[tid] = Q.pairs[1 + t0 + tid];
          s_v[tid] = S.value(__uint_as_float(Q.pairs[1 + Q.n + t0 + tid]));
        }
        __syncthreads();
      }
      for (uint32_t j = tid / 16; j < 2 * nt; j += kIrThreads / 16)
      {
        const uint32_t t = s_t[j >> 1];
        const uint32_t at = ir_search(col, ptr[t], ptr[t + 1], (j & 1) ? lo + n : lo);
        if ((tid & 15) == 0) ((j & 1) ? s_hi : s_lo)[j >> 1] = at;
      }
      __syncthreads();
      // the terms' postings one after another; a round's are read and their
      // contributions formed all at once, then added term by term
      if (warp == 0)
      {
        uint32_t sum = 0;
        for (uint32_t t = lane; t < kIrTerms; t += 32)
        {
          uint32_t x = t < nt ? s_hi[t] - s_lo[t] : 0;
          for (int o = 1; o < 32; o <<= 1)
          {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if ((int) lane >= o) x += y;
          }
          x += sum;
          s_end[t] = x;
          sum = __shfl_sync(0xffffffffu, x, 31);
        }
      }
      __syncthreads();
      const uint32_t total = s_end[nt - 1];
      if (tid == 0) postings += total;
      uint32_t t = 0;  // the term of my next posting
      for (uint32_t f0 = 0; f0 < total; f0 += kIrPer * kIrThreads)
      {
        uint32_t at[kIrPer], d[kIrPer], tf[kIrPer];
        float v[kIrPer];
        // no branches between the loads, so that they are all in flight: a
        // thread without a posting reads the first one
#pragma unroll
        for (int u = 0; u < kIrPer; u++)
        {
          const uint32_t f = f0 + u * kIrThreads + tid;
          while (f < total && f >= s_end[t]) t++;
          at[u] = f < total ? t : 0xFFFFFFFFu;
          d[u] = f < total ? s_hi[t] - (s_end[t] - f) : s_lo[0];
        }
#pragma unroll
        for (int u = 0; u < kIrPer; u++)
        {
          tf[u] = w[d[u]];
          d[u] = col[d[u]];
        }
#pragma unroll
        for (int u = 0; u < kIrPer; u++) v[u] = S.own(d[u]);
#pragma unroll
        for (int u = 0; u < kIrPer; u++) v[u] = S.term(v[u], (float) tf[u], s_v[at[u] != 0xFFFFFFFFu ? at[u] : 0]);
        // this round's terms: from that of its first posting to that of its last
        uint32_t ta = 0, tb;
        while (f0 >= s_end[ta]) ta++;
        tb = ta;
        while (min(total, f0 + kIrPer * kIrThreads) > s_end[tb]) tb++;
        for (uint32_t k2 = ta; k2 <= tb; k2++)
        {
#pragma unroll
          for (int u = 0; u < kIrPer; u++)
            if (at[u] == k2)
            {
              score[d[u] - lo] = __fadd_rn(score[d[u] - lo], v[u]);
              touched[d[u] - lo] = 1;
            }
          __syncthreads();
        }
      }
    }
    if (!cnt) __syncthreads();
    // final scores, the touched count, the dumps
    uint32_t mine = 0;
    for (uint32_t i = tid; i < n; i += kIrThreads)
    {
      const bool on = touched[i];
      if (on) score[i] = S.done(lo + i, score[i]);
      else if (lo + i >= leftover_from) touched[i] = 1;  // joins with score 0
      if (!touched[i]) continue;
      mine++;
      if (all || act)
      {
        const uint32_t id = id_of_pos[lo + i];
        if (all) all[id] = score[i];
        if (act) act[id] = 1;
      }
    }
    mine = __reduce_add_sync(0xffffffffu, mine);
    if (lane == 0 && mine) atomicAdd(&s_touched, mine);
    if (!k) continue;  // a thread's own entries only: nothing to wait for
    // the chunk's top k, with the block's so far
    auto key = [&](uint32_t i) {
      return i >= n ? s_best[i - n] : touched[i] ? ir_key(score[i], lo + i) : 0ull;
    };
    unsigned long long best = 0;
#pragma unroll 4
    for (uint32_t i = tid; i < n + k; i += kIrThreads) best = max(best, key(i));
    ir_topk(
        n + k, key, best,
        [&](unsigned long long T, auto push) {
          for (uint32_t i = tid; i < n + k; i += kIrThreads)
            if (key(i) >= T) push(key(i));
        },
        k, s_top, s_new);
    for (int r = tid; r < k; r += kIrThreads) s_best[r] = s_new[r];
    __syncthreads();
  }
  __syncthreads();
  for (int r = tid; r < k; r += kIrThreads) cand[(size_t) blockIdx.x * k + r] = s_best[r];
  __syncthreads();
  if (tid == 0)
  {
    if (s_touched) atomicAdd(&ctr[0], (unsigned long long) s_touched);
    if (postings) atomicAdd(&ctr[1], postings);
    __threadfence();  // the block's list and counts before its ticket
    s_last = atomicAdd(&ctr[2], 1ull) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  // the last block: every list is written
  __threadfence();
  if (k)
  {
    // a thread takes the (descending) lists tid, tid + kIrThreads, ...: their
    // heads at once, the rest of the few lists that reach the threshold
    constexpr int kLists = 4;
    unsigned long long head[kLists], best = 0;
#pragma unroll
    for (int u = 0; u < kLists; u++)
    {
      const uint32_t b = tid + u * kIrThreads;
      head[u] = b < gridDim.x ? __ldcg(&cand[(size_t) b * k]) : 0;
    }
#pragma unroll
    for (int u = 0; u < kLists; u++) best = max(best, head[u]);
    ir_topk(
        gridDim.x * k, [&](uint32_t i) { return __ldcg(&cand[i]); }, best,
        [&](unsigned long long T, auto push) {
#pragma unroll
          for (int u = 0; u < kLists; u++)
          {
            unsigned long long x = head[u];
            for (int r = 1; x >= T; r++)
            {
              push(x);
              x = r < k ? __ldcg(&cand[(size_t) (tid + u * kIrThreads) * k + r]) : 0;
            }
          }
        },
        k, s_top, s_new);
    for (int r = tid; r < k; r += kIrThreads)
    {
      const unsigned long long top = s_new[r];  // ids for positions
      out->best[r] = top ? top - id_of_pos[~(uint32_t) top] + ~(uint32_t) top : 0;
    }
  }
  if (tid == 0)
  {
    out->ntouched = __ldcg(&ctr[0]);
    out->postings = __ldcg(&ctr[1]);
    ctr[0] = ctr[1] = ctr[2] = 0;
  }
}

// Most blocks of a query: four per SM; the last block's threads walk four lists each.
static uint32_t ir_blocks() { return std::min<uint32_t>(num_sms() * 4, 4 * kIrThreads); }

static int ir_scratch(la3g_graph* G, IrScratch* b)
{
  LA3G_TRY(galloc(G, &b->ctr, 3));
  LA3G_TRY(galloc(G, &b->cand, (size_t) ir_blocks() * kTopKMax));
  LA3G_CUDA(cudaHostAlloc(&b->out, sizeof(IrResult), cudaHostAllocMapped));
  LA3G_CUDA(cudaMemsetAsync(b->ctr, 0, 3 * sizeof(unsigned long long), G->stream));
  return LA3G_OK;
}

// One query: la3g_bm25_query / la3g_lm_query after their checks.  `length`:
// what the terms push; positions from leftover_from on join the pool with
// score 0 if the query does not reach them.
template <class Scorer>
static int ir_query(la3g_graph* G, IrScratch* b, const Scorer& S, const float* length, uint32_t leftover_from,
                    const char* scope, const uint32_t* term_vids, uint32_t nterms, uint32_t k, uint32_t* ids_out,
                    float* scores_out, uint32_t* nout, float* all_scores_out, uint8_t* active_out, la3g_stats* st)
{
  DevGraph& g = G->g;
  cudaStream_t s = G->stream;
  const uint32_t N = g.nslots;
  CallTimer T(G, st);
  IrQuery Q;
  Q.n = nterms;
  Q.pairs = nullptr;
  if (nterms > kIrTerms)
  {
    if (nterms > b->qcap)
    {
      GallocScope scope(G);
      uint32_t *qin = nullptr, *qpos = nullptr;
      LA3G_TRY(galloc(G, &qin, nterms));
      LA3G_TRY(galloc(G, &qpos, 1 + 2 * (size_t) nterms));
      scope.keep();
      b->qin = qin;
      b->qpos = qpos;
      b->qcap = nterms;
    }
    Q.pairs = b->qpos;
  }
  else
    for (uint32_t i = 0; i < nterms; i++) Q.vid[i] = term_vids[i];
  DevBuf all, act;
  if (all_scores_out) LA3G_TRY(all.alloc((size_t) N * 4));
  if (active_out) LA3G_TRY(act.alloc(N));
  T.device_begin();
  if (Q.pairs)
  {
    LA3G_CUDA(cudaMemcpyAsync(b->qin, term_vids, (size_t) nterms * 4, cudaMemcpyHostToDevice, s));
    k_bm25_pair<<<1, 1, 0, s>>>(b->qin, nterms, N, g.nreg, g.pos_of_id, length, b->qpos);
    LA3G_LAUNCHED();
    tls_launches++;
  }
  if (all_scores_out) LA3G_CUDA(cudaMemsetAsync(all.p, 0, (size_t) N * 4, s));
  if (active_out) LA3G_CUDA(cudaMemsetAsync(act.p, 0, N, s));
  const uint32_t blocks = std::min<uint32_t>(std::max<uint32_t>((g.nreg + kIrMinChunk - 1) / kIrMinChunk, 1), ir_blocks());
  const uint32_t chunk = std::max<uint32_t>(std::min<uint32_t>(((g.nreg + blocks - 1) / blocks + 31) & ~31u, kIrChunk), 32);
  {
    ProfileScope p(scope, s, 0.0);
    k_ir_query<Scorer><<<blocks, kIrThreads, chunk * 5, s>>>(Q, S, g.in_ptr, g.in_col, g.in_w, N, g.nreg, chunk, g.pos_of_id,
                                                             g.id_of_pos, length, leftover_from, (int) k, b->ctr,
                                                             b->cand, b->out, all.as<float>(), act.as<uint8_t>());
    LA3G_LAUNCHED();
  }
  T.device_end();
  if (all_scores_out) LA3G_CUDA(cudaMemcpyAsync(all_scores_out, all.p, (size_t) N * 4, cudaMemcpyDeviceToHost, s));
  if (active_out) LA3G_CUDA(cudaMemcpyAsync(active_out, act.p, N, cudaMemcpyDeviceToHost, s));
  LA3G_TRY(T.finish());
  const unsigned long long ntouched = b->out->ntouched, postings = b->out->postings;
  const uint32_t n = (uint32_t) std::min<unsigned long long>(ntouched, (unsigned long long) k);
  for (uint32_t i = 0; i < n; i++)
  {
    const unsigned long long best = b->out->best[i];
    uint32_t u = (uint32_t) (best >> 32);
    u = (u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u;
    float sc;
    std::memcpy(&sc, &u, 4);
    if (ids_out) ids_out[i] = 0xFFFFFFFFu - (uint32_t) best;
    if (scores_out) scores_out[i] = sc;
  }
  if (nout) *nout = n;
  // algorithmic bytes: doc id + tf per posting walked, the doc's value read
  // and its score formed per touched doc
  const double bytes = 8.0 * (double) postings + 12.0 * (double) ntouched;
  profile_add_bytes(scope, bytes);
  if (st)
  {
    st->iterations = 1;
    st->teps_edges = ntouched;
    st->edges_examined = postings;
    st->algo_bytes = (uint64_t) bytes;
  }
  return LA3G_OK;
}

}  // namespace la3g

#endif
