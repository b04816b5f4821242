// BM25: the reference bm25 app (src/apps/information_retrieval/bm25.cpp:8-114,
// bm25.h:11-92, helpers.hpp:76-123) on the device.
//
// The graph is bipartite and undirected (docs 1..D, terms D+1..D+T, identity
// hash), so every vertex with postings is regular and positions ascend with
// ids: docs first, then terms.  A term's row of the pull CSR lists its docs
// ascending, a doc's row lists its terms ascending — the order in which the
// reference's single-iteration SpMV visits them.
//
// prepare (bm25.cpp:16-47):
//   IDF:  y(t) = sum of 1.0f over t's docs (exactly min(df, 2^24) in float);
//         idf = (float) log10((double)((float) D - y) + 0.5) / ((double) y + 0.5));
//   DL 1: len(d) = sum over d's terms, ascending, of (float) tf (float adds);
//   tokens = sum over every vertex of (uint64) its float length (terms
//         contribute their truncated idf; values <= -1 count as 0);
//   avg = (float) tokens / (float) D;
//   DL 2: K(d) = 1.2f * ((1 - 0.75f) + 0.75f * (len / avg)).
// query (bm25.cpp:57-108): the listed term vertices push their idf through
//   a StreamingArray (values in push order, indices ascending — a list that
//   is not ascending pairs them the way the reference does, reproduced by
//   k_bm25_pair); then, term by term in ascending order, every doc of the
//   term gets score += (tf * 2.2f) / (tf + K(d)) * idf in float, starting
//   from 0.0f; the top k of the touched docs are returned in the order
//   score desc, id asc.
// All float operations are explicit _rn intrinsics (no contraction).
#include <algorithm>
#include <cstring>
#include <vector>

#include "la3g_internal.h"
#include "ir.cuh"

namespace la3g {

static constexpr float kK1 = 1.2f;
static constexpr float kB = 0.75f;

struct Bm25Scratch
{
  IrScratch ir;
  float* length = nullptr;      // [nslots] DtState.length by position
  unsigned long long* tok = nullptr;  // token count
  uint32_t term_row0 = 0;       // first regular position of a term (docs come first)
  uint64_t tokens = 0;
  float avg = 0.0f;
  bool prepared = false;
};

static void bm25_scratch_free(void* p)
{
  Bm25Scratch* b = (Bm25Scratch*) p;
  if (b->ir.out) cudaFreeHost(b->ir.out);
  delete b;
}

// IDF on term rows [row_lo, row_hi).
__global__ void k_bm25_idf(const uint32_t* __restrict__ ptr, uint32_t row_lo, uint32_t row_hi, uint32_t ndocs,
                           float* length)
{
  for (uint32_t r = row_lo + blockIdx.x * blockDim.x + threadIdx.x; r < row_hi; r += gridDim.x * blockDim.x)
  {
    uint32_t df = ptr[r + 1] - ptr[r];
    float y = df > (1u << 24) ? 16777216.0f : (float) df;  // sequential 1.0f adds saturate at 2^24
    float t = __fsub_rn((float) ndocs, y);
    double num = __dadd_rn((double) t, 0.5);
    double den = __dadd_rn((double) y, 0.5);
    length[r] = (float) log10(__ddiv_rn(num, den));
  }
}

// DL on doc rows [row_lo, row_hi): sum of tf in float, ascending term order.
__global__ void k_bm25_dl(const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ w, uint32_t row_lo,
                          uint32_t row_hi, float avg, float* length)
{
  for (uint32_t r = row_lo + blockIdx.x * blockDim.x + threadIdx.x; r < row_hi; r += gridDim.x * blockDim.x)
  {
    float y = 0.0f;
    for (uint32_t e = ptr[r]; e < ptr[r + 1]; e++) y = __fadd_rn(y, (float) w[e]);
    y = __fadd_rn(0.0f, y);  // combine(partial, A())
    if (avg == 0.0f) length[r] = y;
    else length[r] = __fmul_rn(kK1, __fadd_rn(__fsub_rn(1.0f, kB), __fmul_rn(kB, __fdiv_rn(y, avg))));
  }
}

__global__ void k_bm25_tokens(const float* __restrict__ length, uint32_t n, unsigned long long* out)
{
  unsigned long long s = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
  {
    float f = length[i];
    s += f > 0.0f ? (unsigned long long) f : 0ull;
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0 && s) atomicAdd(out, s);
}

// StreamingArray push emulation (streaming_array.h:92-96) for one query:
// push(i, v) stores v at slot count and sets bit i; the j-th smallest set
// index is then read with the value of slot j.  Output: (position, idf)
// pairs ascending by position, count in qpos[0].
__global__ void k_bm25_pair(const uint32_t* __restrict__ q, uint32_t nq, uint32_t nslots, uint32_t nreg,
                            const uint32_t* __restrict__ pos_of_id, const float* __restrict__ length, uint32_t* out)
{
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  uint32_t* idx = out + 1;        // set indices (insertion order)
  uint32_t* val = out + 1 + nq;   // slot values
  uint32_t cnt = 0;
  for (uint32_t i = 0; i < nq; i++)
  {
    uint32_t v = q[i];
    if (v >= nslots) continue;        // not a local vertex (vertex_program.hpp:199)
    uint32_t p = pos_of_id[v];
    if (p >= nreg) continue;          // isolated: init only, no scatter
    val[cnt] = __float_as_uint(length[p]);
    bool seen = false;
    for (uint32_t j = 0; j < cnt; j++) seen |= idx[j] == p;
    if (!seen) idx[cnt++] = p;
  }
  // sort the indices ascending (insertion sort; queries are short)
  for (uint32_t a = 1; a < cnt; a++)
  {
    uint32_t x = idx[a];
    int b = (int) a - 1;
    while (b >= 0 && idx[b] > x) { idx[b + 1] = idx[b]; b--; }
    idx[b + 1] = x;
  }
  out[0] = cnt;
}

// One posting adds (tf * 2.2) / (tf + K(d)) * idf.  gather reads the row's
// mirror state, taken when the TFIDF program was first initialised: docs hold
// K(d); terms (not active then) hold zero.  A term row is reached only by a
// query that names a document vertex.
struct Bm25Scorer
{
  const float* __restrict__ length;
  uint32_t term_row0;
  __device__ __forceinline__ float value(float idf) const { return idf; }
  __device__ __forceinline__ float own(uint32_t d) const { return d < term_row0 ? length[d] : 0.0f; }
  __device__ __forceinline__ float term(float kd, float wf, float idf) const
  {
    return __fmul_rn(__fdiv_rn(__fmul_rn(wf, __fadd_rn(kK1, 1.0f)), __fadd_rn(wf, kd)), idf);
  }
  __device__ __forceinline__ float done(uint32_t, float y) const { return y; }
};

__global__ void k_f32_by_id(uint32_t N, const uint32_t* __restrict__ id_of_pos, const float* __restrict__ v, float* out)
{
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < N; p += gridDim.x * blockDim.x) out[id_of_pos[p]] = v[p];
}

static int bm25_scratch_build(la3g_graph* G, Bm25Scratch* b)
{
  const uint32_t N = G->g.nslots;
  LA3G_TRY(galloc(G, &b->length, N));
  LA3G_TRY(galloc(G, &b->tok, 1));
  LA3G_TRY(ir_scratch(G, &b->ir));
  return LA3G_OK;
}

static int bm25_scratch(la3g_graph* G, Bm25Scratch** out)
{
  return graph_scratch(G, kSlotBm25, bm25_scratch_free, out, [&](Bm25Scratch* b) { return bm25_scratch_build(G, b); });
}

// First term row: positions ascend with ids, docs (ids <= D) come first.
int bipartite_first_term_row(la3g_graph* G, uint32_t* out)
{
  DevGraph& g = G->g;
  // binary search over id_of_pos[0, nreg) for the first id > nleft
  uint32_t lo = 0, hi = g.nreg;
  while (lo < hi)
  {
    uint32_t mid = (lo + hi) / 2, id = 0;
    LA3G_CUDA(cudaMemcpy(&id, g.id_of_pos + mid, 4, cudaMemcpyDeviceToHost));
    if (id <= g.nleft) lo = mid + 1;
    else hi = mid;
  }
  *out = lo;
  return LA3G_OK;
}

}  // namespace la3g

using namespace la3g;

extern "C" int la3g_bm25_prepare(la3g_graph* G, uint64_t* ntokens_out, float* avg_out, float* length_out)
{
  if (!G) return set_error(LA3G_EINVAL, "null graph");
  DevGraph& g = G->g;
  if (!(g.flags & LA3G_BIPARTITE) || g.directed() || !g.weighted())
    return set_error(LA3G_EINVAL, "bm25 needs a graph loaded with LA3G_BIPARTITE | LA3G_WEIGHTED (undirected)");
  Bm25Scratch* b = nullptr;
  LA3G_TRY(bm25_scratch(G, &b));
  cudaStream_t s = G->stream;
  const uint32_t N = g.nslots;
  LA3G_CUDA(cudaStreamSynchronize(s));
  uint32_t tb = 0;
  LA3G_TRY(bipartite_first_term_row(G, &tb));
  b->term_row0 = tb;
  LA3G_CUDA(cudaMemsetAsync(b->length, 0, (size_t) N * 4, s));
  LA3G_CUDA(cudaMemsetAsync(b->tok, 0, 8, s));
  {
    ProfileScope p("bm25_idf", s, 4.0 * (g.nreg - tb + 1) + 4.0 * (g.nreg - tb));
    k_bm25_idf<<<grid_for(g.nreg - tb, 256), 256, 0, s>>>(g.in_ptr, tb, g.nreg, g.nleft, b->length);
    LA3G_LAUNCHED();
  }
  {
    ProfileScope p("bm25_dl", s, 8.0 * g.nent / 2);
    k_bm25_dl<<<grid_for(tb, 256), 256, 0, s>>>(g.in_ptr, g.in_w, 0, tb, 0.0f, b->length);
    LA3G_LAUNCHED();
  }
  k_bm25_tokens<<<grid_for(N, 256), 256, 0, s>>>(b->length, N, b->tok);
  LA3G_LAUNCHED();
  unsigned long long tok = 0;
  LA3G_CUDA(cudaMemcpyAsync(&tok, b->tok, 8, cudaMemcpyDeviceToHost, s));
  LA3G_CUDA(cudaStreamSynchronize(s));
  // avg = collection_ntokens / (float) ndocs (bm25.cpp:38): uint64 -> float, float divide
  const float avg = (float) tok / (float) g.nleft;
  {
    ProfileScope p("bm25_dl", s, 8.0 * g.nent / 2);
    k_bm25_dl<<<grid_for(tb, 256), 256, 0, s>>>(g.in_ptr, g.in_w, 0, tb, avg, b->length);
    LA3G_LAUNCHED();
  }
  b->tokens = tok;
  b->avg = avg;
  b->prepared = true;
  if (ntokens_out) *ntokens_out = tok;
  if (avg_out) *avg_out = avg;
  if (length_out)
  {
    DevBuf tmp;
    LA3G_TRY(tmp.alloc((size_t) N * 4));
    k_f32_by_id<<<grid_for(N, 256), 256, 0, s>>>(N, g.id_of_pos, b->length, tmp.as<float>());
    LA3G_LAUNCHED();
    LA3G_CUDA(cudaMemcpyAsync(length_out, tmp.p, (size_t) N * 4, cudaMemcpyDeviceToHost, s));
  }
  LA3G_CUDA(cudaStreamSynchronize(s));
  return LA3G_OK;
}

extern "C" int la3g_bm25_query(la3g_graph* G, const uint32_t* term_vids, uint32_t nterms, uint32_t k,
                               uint32_t* ids_out, float* scores_out, uint32_t* nout, float* all_scores_out,
                               uint8_t* active_out, la3g_stats* st)
{
  if (!G) return set_error(LA3G_EINVAL, "null graph");
  if (nterms && !term_vids) return set_error(LA3G_EINVAL, "term_vids is null");
  if (k > kTopKMax) return set_error(LA3G_EINVAL, "k = %u exceeds the maximum of %d", k, kTopKMax);
  Bm25Scratch* b = (Bm25Scratch*) G->slot[kSlotBm25];
  if (!b || !b->prepared) return set_error(LA3G_EINVAL, "call la3g_bm25_prepare first");
  return ir_query(G, &b->ir, Bm25Scorer{b->length, b->term_row0}, b->length, 0xFFFFFFFFu, "bm25_term", term_vids, nterms, k,
                  ids_out, scores_out, nout, all_scores_out, active_out, st);
}
