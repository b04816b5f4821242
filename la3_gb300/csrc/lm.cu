// LM: the reference lm app (src/apps/information_retrieval/lm.cpp:8-144,
// lm.h:16-75) on the device: query likelihood with Dirichlet smoothing
// (mu = 2000) over the same bipartite corpus as BM25.
//
// prepare (lm.cpp:16-46):
//   DL:  length(d) = sum over d's terms, ascending, of (float) tf (float adds);
//   tokens = sum over every vertex of (uint64) its float length (terms hold 0);
//   TL:  length(t) = (sum over t's docs, ascending, of (float) tf) / (float)
//        tokens — the sums of frequent terms pass 2^24, where float addition
//        rounds, so each term row is summed in the reference's order (a warp
//        loads 32 entries at a time, lanes' values are added one after
//        another);
//   the per-vertex factor log10f(mu / (length + mu)) of the score
//        (lm.h:74): that log10 takes a float, so the reference calls the float
//        overload of the platform's libm, which is not correctly rounded; the
//        factor depends only on the vertex's length and is evaluated once per
//        vertex here, with the same libm function, and kept on the device.
// query (lm.cpp:57-87): the listed term vertices push their length through a
//   StreamingArray (k_bm25_pair); term by term, ascending, every doc of the
//   term adds (float) log10(1.0 + (double) (tf / (mu * length(t)))) — a
//   double log10, rounded to float — to its score, from 0.0f; the touched
//   vertices then take score = y + (float) nterms * factor.  The top k of the
//   active vertices are returned (score desc, id asc).  The TFIDF program
//   reads no state in gather, so the reference takes no mirrors at its first
//   initialize and the activity the TL pass left (every term row) is still
//   set in the first query after prepare: those terms join that query's pool
//   with score 0, as in the reference.
// All float operations are explicit _rn intrinsics (no contraction).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "la3g_internal.h"
#include "ir.cuh"

namespace la3g {

static constexpr float kMu = 2000.0f;

struct LmScratch
{
  IrScratch ir;
  float* length = nullptr;      // [nslots] DtState.length by position
  float* factor = nullptr;      // [nslots] log10f(mu / (length + mu)) by position
  unsigned long long* tok = nullptr;  // token count
  uint32_t term_row0 = 0;
  uint64_t tokens = 0;
  bool prepared = false;
  bool leftover = false;        // the TL pass's activity is still set (first query)
};

static void lm_scratch_free(void* p)
{
  LmScratch* b = (LmScratch*) p;
  if (b->ir.out) cudaFreeHost(b->ir.out);
  delete b;
}

// TL on term rows [row_lo, row_hi): a warp per row, lanes load 32 entries at
// a time and the sum runs through them in entry (ascending doc) order.
__global__ void k_lm_tl(const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ w, uint32_t row_lo,
                        uint32_t row_hi, float ntok, float* length)
{
  const int lane = threadIdx.x & 31;
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t r = row_lo + warp; r < row_hi; r += nwarps)
  {
    const uint32_t b = ptr[r], e = ptr[r + 1];
    float y = 0.0f;
    for (uint32_t c0 = b; c0 < e; c0 += 32)
    {
      const uint32_t n = min(32u, e - c0);
      const float v = (uint32_t) lane < n ? (float) w[c0 + lane] : 0.0f;
      for (uint32_t j = 0; j < n; j++) y = __fadd_rn(y, __shfl_sync(0xffffffffu, v, j));
    }
    y = __fadd_rn(0.0f, y);  // combine(partial, A())
    if (lane == 0) length[r] = __fdiv_rn(y, ntok);
  }
}

// One posting adds log10(1 + tf / (mu * msg)); a touched vertex then takes
// score = y + (float) nterms * factor.
struct LmScorer
{
  const float* __restrict__ factor;
  float nterms;
  __device__ __forceinline__ float value(float msg) const { return __fmul_rn(kMu, msg); }
  __device__ __forceinline__ float own(uint32_t) const { return 0.0f; }
  __device__ __forceinline__ float term(float, float wf, float den) const
  {
    return (float) log10(__dadd_rn(1.0, (double) __fdiv_rn(wf, den)));
  }
  __device__ __forceinline__ float done(uint32_t d, float y) const
  {
    return __fadd_rn(y, __fmul_rn(nterms, factor[d]));
  }
};

static int lm_scratch_build(la3g_graph* G, LmScratch* b)
{
  const uint32_t N = G->g.nslots;
  LA3G_TRY(galloc(G, &b->length, N));
  LA3G_TRY(galloc(G, &b->factor, N));
  LA3G_TRY(galloc(G, &b->tok, 1));
  LA3G_TRY(ir_scratch(G, &b->ir));
  return LA3G_OK;
}

static int lm_scratch(la3g_graph* G, LmScratch** out)
{
  return graph_scratch(G, kSlotLm, lm_scratch_free, out, [&](LmScratch* b) { return lm_scratch_build(G, b); });
}

}  // namespace la3g

using namespace la3g;

extern "C" int la3g_lm_prepare(la3g_graph* G, uint64_t* ntokens_out, float* length_out)
{
  if (!G) return set_error(LA3G_EINVAL, "null graph");
  DevGraph& g = G->g;
  if (!(g.flags & LA3G_BIPARTITE) || g.directed() || !g.weighted())
    return set_error(LA3G_EINVAL, "lm needs a graph loaded with LA3G_BIPARTITE | LA3G_WEIGHTED (undirected)");
  LmScratch* b = nullptr;
  LA3G_TRY(lm_scratch(G, &b));
  cudaStream_t s = G->stream;
  const uint32_t N = g.nslots;
  LA3G_CUDA(cudaStreamSynchronize(s));
  uint32_t tb = 0;
  LA3G_TRY(bipartite_first_term_row(G, &tb));
  b->term_row0 = tb;
  LA3G_CUDA(cudaMemsetAsync(b->length, 0, (size_t) N * 4, s));
  LA3G_CUDA(cudaMemsetAsync(b->tok, 0, 8, s));
  {
    ProfileScope p("lm_dl", s, 8.0 * g.nent / 2);
    k_bm25_dl<<<grid_for(tb, 256), 256, 0, s>>>(g.in_ptr, g.in_w, 0, tb, 0.0f, b->length);
    LA3G_LAUNCHED();
  }
  k_bm25_tokens<<<grid_for(N, 256), 256, 0, s>>>(b->length, N, b->tok);
  LA3G_LAUNCHED();
  unsigned long long tok = 0;
  LA3G_CUDA(cudaMemcpyAsync(&tok, b->tok, 8, cudaMemcpyDeviceToHost, s));
  LA3G_CUDA(cudaStreamSynchronize(s));
  if (g.nreg > tb)
  {
    ProfileScope p("lm_tl", s, 8.0 * g.nent / 2);
    // length = y / collection_ntokens (lm.h:55): the uint64 count as float
    k_lm_tl<<<grid_for((uint64_t) (g.nreg - tb) * 32, 256), 256, 0, s>>>(g.in_ptr, g.in_w, tb, g.nreg, (float) tok,
                                                                         b->length);
    LA3G_LAUNCHED();
  }
  // the score's per-vertex factor with the platform's log10f (see the top)
  std::vector<float> len(g.nreg), fac(g.nreg);
  if (g.nreg)
  {
    LA3G_CUDA(cudaMemcpyAsync(len.data(), b->length, (size_t) g.nreg * 4, cudaMemcpyDeviceToHost, s));
    LA3G_CUDA(cudaStreamSynchronize(s));
    for (uint32_t i = 0; i < g.nreg; i++) fac[i] = log10f(kMu / (len[i] + kMu));
    LA3G_CUDA(cudaMemcpyAsync(b->factor, fac.data(), (size_t) g.nreg * 4, cudaMemcpyHostToDevice, s));
  }
  b->tokens = tok;
  b->prepared = true;
  b->leftover = true;
  if (ntokens_out) *ntokens_out = tok;
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

extern "C" int la3g_lm_query(la3g_graph* G, const uint32_t* term_vids, uint32_t nterms, uint32_t k, uint32_t* ids_out,
                             float* scores_out, uint32_t* nout, float* all_scores_out, uint8_t* active_out,
                             la3g_stats* st)
{
  if (!G) return set_error(LA3G_EINVAL, "null graph");
  if (nterms && !term_vids) return set_error(LA3G_EINVAL, "term_vids is null");
  if (k > kTopKMax) return set_error(LA3G_EINVAL, "k = %u exceeds the maximum of %d", k, kTopKMax);
  LmScratch* b = (LmScratch*) G->slot[kSlotLm];
  if (!b || !b->prepared) return set_error(LA3G_EINVAL, "call la3g_lm_prepare first");
  // the leftover activity of the TL pass lasts for one query
  // (tfidf.reset_activity() after it, lm.cpp:86)
  const uint32_t leftover_from = b->leftover ? b->term_row0 : 0xFFFFFFFFu;
  // query_nterms = queries[q].size() (lm.cpp:66), as float in the apply
  LA3G_TRY(ir_query(G, &b->ir, LmScorer{b->factor, (float) nterms}, b->length, leftover_from, "lm_term", term_vids, nterms,
                    k, ids_out, scores_out, nout, all_scores_out, active_out, st));
  b->leftover = false;
  return LA3G_OK;
}
