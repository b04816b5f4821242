// Device ingest: LA3 records -> the device matrix in internal order.
//
// Follows Graph::load_binary (src/matrix/graph.hpp:37-214) record by record,
// the per-tile dedup that keeps the first inserted triple
// (src/matrix/csc_matrix2d.hpp:62-72), the regular/sink/source/isolated
// classification (src/matrix/processed_matrix2d.hpp:203-228) and the locator
// order (src/utils/locator.h:84-155).  The reference builds one CSC per tile
// on the host with hash sets; here the records are transformed on the
// device, sorted (stable radix sort keeps insertion order among duplicates),
// deduplicated, ranked per class, and laid out as CSR arrays.
#include <sys/stat.h>

#include <algorithm>
#include <cstring>
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <cub/device/device_select.cuh>

#include "la3g_internal.h"

namespace la3g {

struct IngestParams
{
  uint64_t N;            // nslots
  uint32_t nleft;        // bipartite column shift
  bool bipartite, directed, reverse, acyclic;
  Hasher h;
};

// One record's entry by graph.hpp:160-191: false for a self-loop; hr / hc are
// the hashed row and column (the caller checks their range).
__device__ __forceinline__ bool ingest_record(const IngestParams& P, uint32_t row, uint32_t col, uint32_t& hr, uint32_t& hc)
{
  if (P.bipartite) col += P.nleft;
  if (row == col) return false;
  if (P.directed && !P.reverse) { uint32_t t = row; row = col; col = t; }
  if (P.acyclic && ((!P.reverse && col > row) || (P.reverse && col < row))) { uint32_t t = row; row = col; col = t; }
  hr = P.h.hash(row);
  hc = P.h.hash(col);
  return true;
}

// Which hashed ids have a non-empty row / column (duplicates do not matter
// for that, so the classes and positions are known before the entries are
// sorted, and one sort by position serves for dropping the duplicates too).
// Undirected records stand for both directions.  A flag is read before it is
// written: most are set already, and the read stays in L1.
__global__ void k_mark(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b, uint32_t stride, uint64_t nrec,
                       IngestParams P, uint8_t* rowne, uint8_t* colne, unsigned long long* bad)
{
  for (uint64_t i = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x; i < nrec;
       i += (uint64_t) gridDim.x * blockDim.x)
  {
    uint32_t hr, hc;
    if (!ingest_record(P, a[i * stride], b[i * stride], hr, hc)) continue;
    if (hr >= P.N || hc >= P.N)
    {
      atomicMin(bad, (unsigned long long) i);
      continue;
    }
    if (!rowne[hr]) rowne[hr] = 1;
    if (!colne[hc]) colne[hc] = 1;
    if (!P.directed)
    {
      if (!rowne[hc]) rowne[hc] = 1;
      if (!colne[hr]) colne[hr] = 1;
    }
  }
}

struct ClassCounts
{
  uint32_t reg, sink, src;
};

struct ClassSum
{
  __host__ __device__ ClassCounts operator()(const ClassCounts& x, const ClassCounts& y) const
  {
    return {x.reg + y.reg, x.sink + y.sink, x.src + y.src};
  }
};

// Item N stays 0: its exclusive sum is the total.
__global__ void k_class_flags(uint32_t N, const uint8_t* rowne, const uint8_t* colne, ClassCounts* f)
{
  for (uint64_t h = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; h <= N; h += (uint64_t) gridDim.x * blockDim.x)
  {
    const uint32_t r = h < N ? rowne[h] : 0, c = h < N ? colne[h] : 0;
    f[h] = {r & c, r & (c ^ 1u), (r ^ 1u) & c};
  }
}

// Exclusive per-class ranks -> positions (regular, sink, source, rest).
__global__ void k_positions(uint32_t N, const uint8_t* rowne, const uint8_t* colne, const ClassCounts* sum, uint32_t nreg,
                            uint32_t nsink, uint32_t nsrc, Hasher hs, uint32_t* hash_of_pos, uint32_t* pos_of_hash,
                            uint32_t* id_of_pos, uint32_t* pos_of_id)
{
  for (uint32_t h = blockIdx.x * blockDim.x + threadIdx.x; h < N; h += gridDim.x * blockDim.x)
  {
    uint8_t r = rowne[h], c = colne[h];
    const ClassCounts k = sum[h];
    uint32_t p;
    if (r & c) p = k.reg;
    else if (r) p = nreg + k.sink;
    else if (c) p = nreg + nsink + k.src;
    else p = nreg + nsink + nsrc + (h - k.reg - k.sink - k.src);
    hash_of_pos[p] = h;
    pos_of_hash[h] = p;
    uint32_t id = hs.unhash(h);
    id_of_pos[p] = id;
    pos_of_id[id] = p;
  }
}

// Sort key of an entry: row position, then the column in the order the
// reference's SpMV visits it (source columns before regular ones,
// process_ready_messages, vertex_program_execute.hpp:479-482), cbits wide.
// Dropped records get row nrows and sort last.  The sort is stable and its
// payload is the weight, so the first of equal keys is the entry the reference
// keeps.  Undirected records emit the edge and its mirror at slots 2i, 2i + 1
// (insertion order of the reference).
__global__ void k_keys(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b, const uint32_t* __restrict__ w,
                       uint32_t stride, uint64_t nrec, IngestParams P, const uint32_t* __restrict__ pos_of_hash,
                       uint32_t nrows, uint32_t nsrc, int cbits, uint64_t* __restrict__ keys, uint32_t* __restrict__ vals)
{
  for (uint64_t i = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x; i < nrec;
       i += (uint64_t) gridDim.x * blockDim.x)
  {
    uint32_t hr, hc;
    const bool keep = ingest_record(P, a[i * stride], b[i * stride], hr, hc);
    const uint32_t wt = w ? w[i * stride] : 0;
    // source columns are the positions from nrows on
    uint32_t rp = nrows, cp = 0, rk = 0, ck = 0;
    if (keep)
    {
      rp = pos_of_hash[hr];
      cp = pos_of_hash[hc];
      rk = rp >= nrows ? rp - nrows : rp + nsrc;
      ck = cp >= nrows ? cp - nrows : cp + nsrc;
    }
    const uint64_t k0 = ((uint64_t) rp << cbits) | ck, k1 = ((uint64_t) (keep ? cp : nrows) << cbits) | rk;
    if (P.directed)
    {
      keys[i] = k0;
      if (w) vals[i] = wt;
    }
    else
    {
      keys[2 * i] = k0;
      keys[2 * i + 1] = k1;
      if (w) vals[2 * i] = vals[2 * i + 1] = wt;
    }
  }
}

// The number of kept entries: the different keys but the dropped records'.
__global__ void k_kept(const uint64_t* __restrict__ keys, const unsigned long long* __restrict__ nsel, uint32_t nrows,
                       int cbits, unsigned long long* out)
{
  const unsigned long long n = *nsel;
  *out = n && (keys[n - 1] >> cbits) == nrows ? n - 1 : n;
}

// The pull CSR from the different sorted keys.  Every row below nrows has an
// entry, so the first entry of each row writes its offset; the rest of the
// offsets are the entry count.
__global__ void k_pull_fill(const uint64_t* __restrict__ keys, const uint32_t* __restrict__ vals, uint64_t m, uint32_t N,
                            uint32_t nrows, uint32_t nsrc, int cbits, uint32_t* __restrict__ ptr,
                            uint32_t* __restrict__ col, uint32_t* __restrict__ w)
{
  const uint64_t tid = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x, nth = (uint64_t) gridDim.x * blockDim.x;
  for (uint64_t i = tid; i < m; i += nth)
  {
    const uint64_t k = keys[i];
    const uint32_t r = (uint32_t) (k >> cbits), ck = (uint32_t) (k & ((1ull << cbits) - 1));
    col[i] = ck < nsrc ? nrows + ck : ck - nsrc;
    if (w) w[i] = vals[i];
    if (i == 0 || (uint32_t) (keys[i - 1] >> cbits) != r) ptr[r] = (uint32_t) i;
  }
  for (uint64_t q = nrows + tid; q <= N; q += nth) ptr[q] = (uint32_t) m;
}

static int bits_for(uint64_t v)
{
  int b = 0;
  while (b < 64 && (v >> b) != 0) b++;
  return b < 1 ? 1 : b;
}

// Bytes rounded up so that the next array of an arena is aligned.
static size_t arena_size(size_t bytes) { return (bytes + 255) & ~(size_t) 255; }

static constexpr size_t kRecSlack = 512;  // lets two sort arrays, rounded up, take the records' place

struct Arena
{
  char* p;
  template <class T>
  T* take(size_t count)
  {
    T* r = (T*) p;
    p += arena_size(count * sizeof(T));
    return r;
  }
};

// Builds the device graph from records already on the device in `rec`.  `a`,
// `b`, `w` point at the src / dst / weight words inside it with the given
// stride (3 or 2 for on-disk records, 1 for separate arrays).  Once the sort
// keys are made the records are done with, and their memory is the sort's
// second buffer where it is large enough (directed loads); everything else
// temporary is one allocation (each costs about 70 us with its release).
// A weighted directed R-MAT 2^20 (17.3M records in host memory): 8.7 ms with
// two sorts, a row-offset pass whose last thread wrote all the empty rows'
// offsets alone (1.8 ms) and 27 temporary buffers; 3.8 ms.
static int build_graph(la3g_graph* G, DevBuf& rec, const uint32_t* a, const uint32_t* b, const uint32_t* w,
                       uint32_t stride, uint64_t nrec)
{
  DevGraph& g = G->g;
  cudaStream_t s = G->stream;
  const uint64_t N = g.nslots;
  if (N > (1ull << 31)) return set_error(LA3G_EINVAL, "too many vertices (%llu)", (unsigned long long) N);
  if (nrec >= (1ull << 32) - 1) return set_error(LA3G_EINVAL, "too many records");
  const bool directed = g.flags & LA3G_DIRECTED;
  const uint64_t m0 = directed ? nrec : 2 * nrec;
  if (!g.weighted()) w = nullptr;
  IngestParams P;
  P.N = N;
  P.nleft = g.nleft;
  P.bipartite = g.flags & LA3G_BIPARTITE;
  P.directed = directed;
  P.reverse = g.flags & LA3G_REVERSE;
  P.acyclic = g.flags & LA3G_ACYCLIC;
  P.h = g.hasher;

  // temporaries: the library calls' storage is asked for at the widest keys
  size_t tb_scan = 0, tb_sort = 0, tb_uniq = 0;
  {
    ClassCounts* c = nullptr;
    LA3G_CUDA(cub::DeviceScan::ExclusiveScan(nullptr, tb_scan, c, c, ClassSum(), ClassCounts{0, 0, 0}, (int64_t) N + 1, s));
    cub::DoubleBuffer<uint64_t> k(nullptr, nullptr);
    cub::DoubleBuffer<uint32_t> v(nullptr, nullptr);
    const uint64_t* ki = nullptr;
    const uint32_t* vi = nullptr;
    uint64_t* ko = nullptr;
    uint32_t* vo = nullptr;
    unsigned long long* n = nullptr;
    if (m0 && w)
    {
      LA3G_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb_sort, k, v, (int64_t) m0, 0, 64, s));
      LA3G_CUDA(cub::DeviceSelect::UniqueByKey(nullptr, tb_uniq, ki, vi, ko, vo, n, (int64_t) m0, s));
    }
    else if (m0)
    {
      LA3G_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, tb_sort, k, (int64_t) m0, 0, 64, s));
      LA3G_CUDA(cub::DeviceSelect::Unique(nullptr, tb_uniq, ki, ko, n, (int64_t) m0, s));
    }
  }
  const size_t tb = std::max(tb_scan, std::max(tb_sort, tb_uniq));
  const size_t sort_bytes = arena_size(m0 * 8) + (w ? arena_size(m0 * 4) : 0);
  const bool in_rec = rec.bytes >= sort_bytes;
  DevBuf temp;
  LA3G_TRY(temp.alloc(sort_bytes * (in_rec ? 1 : 2) + 2 * arena_size(N) + 2 * arena_size((N + 1) * sizeof(ClassCounts)) +
                      arena_size(N * 4) + arena_size(32) + arena_size(tb)));
  Arena A{temp.as<char>()};
  uint64_t *k1 = A.take<uint64_t>(m0), *k2;
  uint32_t *v1 = w ? A.take<uint32_t>(m0) : nullptr, *v2;
  {
    Arena B = in_rec ? Arena{rec.as<char>()} : A;
    k2 = B.take<uint64_t>(m0);
    v2 = w ? B.take<uint32_t>(m0) : nullptr;
    if (!in_rec) A = B;
  }
  uint8_t *rowne = A.take<uint8_t>(N), *colne = A.take<uint8_t>(N);
  ClassCounts *cls = A.take<ClassCounts>(N + 1), *sum = A.take<ClassCounts>(N + 1);
  uint32_t* pos_of_hash = A.take<uint32_t>(N);
  unsigned long long* ctr = A.take<unsigned long long>(4);  // [0] first bad record [1] different keys [2] kept
  void* lib = A.take<char>(tb);

  // Classes and positions.
  LA3G_CUDA(cudaMemsetAsync(ctr, 0xFF, 8, s));
  LA3G_CUDA(cudaMemsetAsync(rowne, 0, arena_size(N) + N, s));  // rowne and colne
  if (nrec)
  {
    k_mark<<<grid_for(nrec, 256), 256, 0, s>>>(a, b, stride, nrec, P, rowne, colne, ctr);
    LA3G_LAUNCHED();
  }
  k_class_flags<<<grid_for(N + 1, 256), 256, 0, s>>>((uint32_t) N, rowne, colne, cls);
  LA3G_LAUNCHED();
  size_t tbu = tb;
  LA3G_CUDA(cub::DeviceScan::ExclusiveScan(lib, tbu, cls, sum, ClassSum(), ClassCounts{0, 0, 0}, (int64_t) N + 1, s));
  unsigned long long badi = ~0ull;
  ClassCounts tot{0, 0, 0};
  LA3G_CUDA(cudaMemcpyAsync(&badi, ctr, 8, cudaMemcpyDeviceToHost, s));
  LA3G_CUDA(cudaMemcpyAsync(&tot, sum + N, sizeof tot, cudaMemcpyDeviceToHost, s));
  LA3G_CUDA(cudaStreamSynchronize(s));
  if (badi != ~0ull)
    return set_error(LA3G_EINVAL, "record %llu: vertex id out of range for %llu slots", badi, (unsigned long long) N);
  g.nreg = tot.reg;
  g.nsink = tot.sink;
  g.nsrc = tot.src;
  const uint32_t nrows = g.nrows();
  {
    void* p = nullptr;
    LA3G_TRY(galloc_bytes(G, &p, 3 * arena_size(N * 4)));
    Arena B{(char*) p};
    g.hash_of_pos = B.take<uint32_t>(N);
    g.id_of_pos = B.take<uint32_t>(N);
    g.pos_of_id = B.take<uint32_t>(N);
  }
  k_positions<<<grid_for(N, 256), 256, 0, s>>>((uint32_t) N, rowne, colne, sum, g.nreg, g.nsink, g.nsrc, g.hasher,
                                               g.hash_of_pos, pos_of_hash, g.id_of_pos, g.pos_of_id);
  LA3G_LAUNCHED();

  // Stable sort by (row, column); the first of each run of equal keys wins.
  uint64_t mu = 0;
  const int cbits = bits_for((uint64_t) g.nreg + g.nsrc), end_bit = cbits + bits_for(nrows);
  const uint64_t* ukeys = nullptr;
  const uint32_t* uvals = nullptr;
  if (m0)
  {
    k_keys<<<grid_for(nrec, 256), 256, 0, s>>>(a, b, w, stride, nrec, P, pos_of_hash, nrows, g.nsrc, cbits, k1, v1);
    LA3G_LAUNCHED();
    cub::DoubleBuffer<uint64_t> k(k1, k2);
    cub::DoubleBuffer<uint32_t> v(v1, v2);
    tbu = tb;
    if (w) LA3G_CUDA(cub::DeviceRadixSort::SortPairs(lib, tbu, k, v, (int64_t) m0, 0, end_bit, s));
    else LA3G_CUDA(cub::DeviceRadixSort::SortKeys(lib, tbu, k, (int64_t) m0, 0, end_bit, s));
    tbu = tb;
    if (w)
      LA3G_CUDA(cub::DeviceSelect::UniqueByKey(lib, tbu, (const uint64_t*) k.Current(), (const uint32_t*) v.Current(),
                                               k.Alternate(), v.Alternate(), ctr + 1, (int64_t) m0, s));
    else
      LA3G_CUDA(cub::DeviceSelect::Unique(lib, tbu, (const uint64_t*) k.Current(), k.Alternate(), ctr + 1, (int64_t) m0, s));
    ukeys = k.Alternate();
    uvals = w ? v.Alternate() : nullptr;
    k_kept<<<1, 1, 0, s>>>(ukeys, ctr + 1, nrows, cbits, ctr + 2);
    LA3G_LAUNCHED();
    unsigned long long kept = 0;
    LA3G_CUDA(cudaMemcpyAsync(&kept, ctr + 2, 8, cudaMemcpyDeviceToHost, s));
    LA3G_CUDA(cudaStreamSynchronize(s));
    mu = kept;
  }
  if (mu >= (1ull << 32) - 1) return set_error(LA3G_EINVAL, "too many stored entries (%llu)", (unsigned long long) mu);
  g.nent = mu;

  // Pull CSR.
  {
    void* p = nullptr;
    LA3G_TRY(galloc_bytes(G, &p, arena_size((N + 1) * 4) + arena_size((mu + 1) * 4) * (w ? 2 : 1)));
    Arena B{(char*) p};
    g.in_ptr = B.take<uint32_t>(N + 1);
    g.in_col = B.take<uint32_t>(mu + 1);
    if (w) g.in_w = B.take<uint32_t>(mu + 1);
  }
  k_pull_fill<<<grid_for(std::max<uint64_t>(mu, N + 1), 256), 256, 0, s>>>(ukeys, uvals, mu, (uint32_t) N, nrows, g.nsrc,
                                                                           cbits, g.in_ptr, g.in_col, g.in_w);
  LA3G_LAUNCHED();
  if (!directed)
  {
    g.out_ptr = g.in_ptr;
    g.out_row = g.in_col;
    g.out_w = g.in_w;
  }
  LA3G_CUDA(cudaStreamSynchronize(s));
  return LA3G_OK;
}

// Push CSR for directed graphs: the pull entries, which are in row order,
// sorted stably by column alone, the row (and weight) as payload.
template <class V>
__global__ void __launch_bounds__(256)
k_push_entries(const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ col, const uint32_t* __restrict__ w,
               uint32_t nrows, uint32_t* __restrict__ key, V* __restrict__ val)
{
  const uint32_t lane = threadIdx.x & 31, nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < nrows; r += nw)
    for (uint32_t e = ptr[r] + lane; e < ptr[r + 1]; e += 32)
    {
      key[e] = col[e];
      V v = (V) r;
      if (sizeof(V) == 8) v |= (V) ((uint64_t) w[e] << 32);
      val[e] = v;
    }
}

// Every regular and source column has an entry: the first of each writes its
// offset; k_push_gaps fills in those of the sinks and of the rest.
template <class V>
__global__ void k_push_fill(const uint32_t* __restrict__ key, const V* __restrict__ val, uint64_t m, uint32_t* __restrict__ ptr,
                            uint32_t* __restrict__ row, uint32_t* __restrict__ w)
{
  for (uint64_t i = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (uint64_t) gridDim.x * blockDim.x)
  {
    row[i] = (uint32_t) val[i];
    if (sizeof(V) == 8) w[i] = (uint32_t) ((uint64_t) val[i] >> 32);
    if (i == 0 || key[i - 1] != key[i]) ptr[key[i]] = (uint32_t) i;
  }
}

__global__ void k_push_gaps(uint32_t N, uint32_t nreg, uint32_t src_base, uint32_t iso_base, uint64_t m, uint32_t* ptr)
{
  const uint32_t sinks = src_base < iso_base ? ptr[src_base] : (uint32_t) m;
  for (uint64_t q = nreg + blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; q <= N; q += (uint64_t) gridDim.x * blockDim.x)
    if (q < src_base) ptr[q] = sinks;
    else if (q >= iso_base) ptr[q] = (uint32_t) m;
}

template <class V>
static int push_csr(la3g_graph* G)
{
  DevGraph& g = G->g;
  cudaStream_t s = G->stream;
  const uint64_t N = g.nslots, m = g.nent;
  if (m)
  {
    cub::DoubleBuffer<uint32_t> k(nullptr, nullptr);
    cub::DoubleBuffer<V> v(nullptr, nullptr);
    size_t tb = 0;
    LA3G_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, k, v, (int64_t) m, 0, 32, s));
    DevBuf temp;
    LA3G_TRY(temp.alloc(2 * arena_size(m * 4) + 2 * arena_size(m * sizeof(V)) + arena_size(tb)));
    Arena A{temp.as<char>()};
    k = cub::DoubleBuffer<uint32_t>(A.take<uint32_t>(m), A.take<uint32_t>(m));
    v = cub::DoubleBuffer<V>(A.take<V>(m), A.take<V>(m));
    void* lib = A.take<char>(tb);
    k_push_entries<V><<<grid_for((uint64_t) g.nrows() * 32, 256), 256, 0, s>>>(g.in_ptr, g.in_col, g.in_w, g.nrows(),
                                                                               k.Current(), v.Current());
    LA3G_LAUNCHED();
    LA3G_CUDA(cub::DeviceRadixSort::SortPairs(lib, tb, k, v, (int64_t) m, 0, bits_for(N), s));
    k_push_fill<V><<<grid_for(m, 256), 256, 0, s>>>(k.Current(), v.Current(), m, g.out_ptr, g.out_row, g.out_w);
    LA3G_LAUNCHED();
    k_push_gaps<<<grid_for(N + 1, 256), 256, 0, s>>>((uint32_t) N, g.nreg, g.src_base(), g.iso_base(), m, g.out_ptr);
    LA3G_LAUNCHED();
    LA3G_CUDA(cudaStreamSynchronize(s));  // before the temporaries go
  }
  else
  {
    LA3G_CUDA(cudaMemsetAsync(g.out_ptr, 0, (N + 1) * 4, s));
    LA3G_CUDA(cudaStreamSynchronize(s));
  }
  return LA3G_OK;
}

int build_push_csr(la3g_graph* G)
{
  DevGraph& g = G->g;
  if (g.out_ptr) return LA3G_OK;
  const uint64_t N = g.nslots, m = g.nent;
  GallocScope scope(G);
  uint32_t *ptr = nullptr, *row = nullptr, *w = nullptr;
  LA3G_TRY(galloc(G, &ptr, N + 1));
  LA3G_TRY(galloc(G, &row, m + 1));
  if (g.weighted()) LA3G_TRY(galloc(G, &w, m + 1));
  g.out_ptr = ptr;
  g.out_row = row;
  g.out_w = w;
  const int rc = g.weighted() ? push_csr<uint64_t>(G) : push_csr<uint32_t>(G);
  if (rc)
  {
    g.out_ptr = g.out_row = g.out_w = nullptr;  // not built: the next call tries again
    return rc;
  }
  return scope.keep();
}

static int new_graph(uint32_t n, uint32_t nright, uint32_t flags, la3g_graph** out, la3g_graph** G)
{
  *out = nullptr;
  la3g_graph* g = new (std::nothrow) la3g_graph();
  if (!g) return set_error(LA3G_ENOMEM, "out of host memory");
  if (cudaStreamCreateWithFlags(&g->own_stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreate(&g->ev0) != cudaSuccess || cudaEventCreate(&g->ev1) != cudaSuccess)
  {
    cudaError_t e = cudaGetLastError();
    la3g_graph_free(g);
    return set_error(LA3G_ECUDA, "cannot create a CUDA stream: %s", cudaGetErrorString(e));
  }
  g->stream = g->own_stream;
  DevGraph& d = g->g;
  const bool bip = flags & LA3G_BIPARTITE;
  d.flags = flags;
  d.nleft = n;
  d.nvertices = bip ? n + nright : n;
  d.nslots = d.nvertices + 1;  // tile_height = nrows / nrowgrps + 1 (matrix2d.hpp:8)
  d.hasher.null_hash = bip;
  if (!bip)
  {
    d.hasher.height = (uint64_t) d.nvertices / 128u;
    d.hasher.max_range = d.hasher.height * 128u;
  }
  *G = g;
  return LA3G_OK;
}

static bool check_flags(uint32_t flags)
{
  if (flags & ~0x1Fu) return false;
  if ((flags & LA3G_BIPARTITE) && (flags & LA3G_ACYCLIC)) return false;
  if (!(flags & LA3G_DIRECTED) && (flags & (LA3G_REVERSE | LA3G_ACYCLIC))) return false;
  return true;
}

}  // namespace la3g

using namespace la3g;

extern "C" void la3g_graph_free(la3g_graph* g)
{
  if (!g) return;
  if (g->stream) cudaStreamSynchronize(g->stream);
  if (g->own_stream && g->own_stream != g->stream) cudaStreamSynchronize(g->own_stream);
  for (int i = 0; i < kSlotCount; i++)
    if (g->slot[i] && g->slot_free[i]) g->slot_free[i](g->slot[i]);
  for (const auto& a : g->allocations) cudaFree(a.first);
  if (g->ev0) cudaEventDestroy(g->ev0);
  if (g->ev1) cudaEventDestroy(g->ev1);
  if (g->own_stream) cudaStreamDestroy(g->own_stream);
  delete g;
}

extern "C" int la3g_graph_set_stream(la3g_graph* g, void* cuda_stream)
{
  if (!g) return set_error(LA3G_EINVAL, "null graph");
  LA3G_CUDA(cudaStreamSynchronize(g->stream));
  g->stream = cuda_stream ? (cudaStream_t) cuda_stream : g->own_stream;
  return LA3G_OK;
}

extern "C" int la3g_set_wait_limit(la3g_graph* g, long long polls)
{
  if (!g) return set_error(LA3G_EINVAL, "null graph");
  g->wait_polls = polls;
  return LA3G_OK;
}

extern "C" int la3g_graph_from_records(const void* records, uint64_t nrec, uint32_t n, uint32_t nright,
                                       uint32_t flags, la3g_graph** out)
{
  if (!out) return set_error(LA3G_EINVAL, "out is null");
  *out = nullptr;
  if (!check_flags(flags)) return set_error(LA3G_EINVAL, "invalid flag combination 0x%x", flags);
  if (n == 0) return set_error(LA3G_EINVAL, "n must be > 0 for in-memory records");
  if (nrec && !records) return set_error(LA3G_EINVAL, "records is null");
  la3g_graph* G = nullptr;
  LA3G_TRY(new_graph(n, nright, flags, out, &G));
  const uint32_t wpr = (flags & LA3G_WEIGHTED) ? 3 : 2;
  DevBuf rec;
  int rc = rec.alloc(nrec * wpr * 4 + kRecSlack);
  if (!rc && nrec)
  {
    cudaError_t e = cudaMemcpyAsync(rec.p, records, nrec * wpr * 4, cudaMemcpyHostToDevice, G->stream);
    if (e != cudaSuccess) rc = set_error(LA3G_ECUDA, "record upload failed: %s", cudaGetErrorString(e));
  }
  G->g.nrecords = nrec;
  if (!rc) rc = build_graph(G, rec, rec.as<uint32_t>(), rec.as<uint32_t>() + 1, rec.as<uint32_t>() + 2, wpr, nrec);
  if (rc) { la3g_graph_free(G); return rc; }
  *out = G;
  return LA3G_OK;
}

extern "C" int la3g_graph_from_edges(const la3g_edges* e, uint32_t n, uint32_t nright, uint32_t flags,
                                     la3g_graph** out)
{
  if (!out || !e) return set_error(LA3G_EINVAL, "null argument");
  *out = nullptr;
  if (!check_flags(flags)) return set_error(LA3G_EINVAL, "invalid flag combination 0x%x", flags);
  if ((flags & LA3G_WEIGHTED) && !e->w) return set_error(LA3G_EINVAL, "weighted load of an unweighted edge list");
  if (n == 0) { n = e->n; nright = e->nright; }
  la3g_graph* G = nullptr;
  LA3G_TRY(new_graph(n, nright, flags, out, &G));
  const uint64_t m = e->m;
  const size_t part = arena_size(m * 4);
  DevBuf rec;
  int rc = rec.alloc(part * 3);
  Arena A{rec.as<char>()};
  uint32_t *a = A.take<uint32_t>(m), *b = A.take<uint32_t>(m), *w = A.take<uint32_t>(m);
  if (!rc && m)
  {
    cudaError_t c = cudaMemcpyAsync(a, e->src, m * 4, cudaMemcpyHostToDevice, G->stream);
    if (c == cudaSuccess) c = cudaMemcpyAsync(b, e->dst, m * 4, cudaMemcpyHostToDevice, G->stream);
    if (c == cudaSuccess && (flags & LA3G_WEIGHTED)) c = cudaMemcpyAsync(w, e->w, m * 4, cudaMemcpyHostToDevice, G->stream);
    if (c != cudaSuccess) rc = set_error(LA3G_ECUDA, "edge upload failed: %s", cudaGetErrorString(c));
  }
  G->g.nrecords = m;
  if (!rc) rc = build_graph(G, rec, a, b, w, 1, m);
  if (rc) { la3g_graph_free(G); return rc; }
  *out = G;
  return LA3G_OK;
}

extern "C" int la3g_graph_load(const char* path, uint32_t n, uint32_t nright, uint32_t flags, la3g_graph** out)
{
  if (!out || !path) return set_error(LA3G_EINVAL, "null argument");
  *out = nullptr;
  if (!check_flags(flags)) return set_error(LA3G_EINVAL, "invalid flag combination 0x%x", flags);
  FILE* f = std::fopen(path, "rb");
  if (!f) return set_error(LA3G_EIO, "cannot open %s", path);
  struct stat st;
  if (fstat(fileno(f), &st) != 0) { std::fclose(f); return set_error(LA3G_EIO, "cannot stat %s", path); }
  uint64_t size = (uint64_t) st.st_size, offset = 0;
  const uint32_t wpr = (flags & LA3G_WEIGHTED) ? 3 : 2;
  if (n == 0)
  {
    // 16-byte header {u32 n-1, u32 m-1, u64 nnz} (graph.hpp:207-235).  The
    // vertex count is taken from it for every graph kind.
    uint32_t h[4];
    if (std::fread(h, 16, 1, f) != 1) { std::fclose(f); return set_error(LA3G_EFORMAT, "%s: short header", path); }
    n = h[0] + 1;
    if (flags & LA3G_BIPARTITE) nright = h[1] + 1;
    offset = 16;
  }
  if ((size - offset) % (wpr * 4) != 0)
  {
    std::fclose(f);
    return set_error(LA3G_EFORMAT, "%s: %llu bytes is not a whole number of %u-byte records", path,
                     (unsigned long long) (size - offset), wpr * 4);
  }
  const uint64_t nrec = (size - offset) / (wpr * 4);
  la3g_graph* G = nullptr;
  int rc = new_graph(n, nright, flags, out, &G);
  if (rc) { std::fclose(f); return rc; }
  DevBuf rec;
  rc = rec.alloc(nrec * wpr * 4 + kRecSlack);
  // Stream the file through a pinned staging buffer.
  const size_t chunk = 64u << 20;
  void* stage = nullptr;
  if (!rc && cudaHostAlloc(&stage, chunk, cudaHostAllocDefault) != cudaSuccess)
  {
    cudaGetLastError();
    stage = nullptr;
    rc = set_error(LA3G_ENOMEM, "cannot allocate pinned staging memory");
  }
  uint64_t done = 0, total = nrec * wpr * 4;
  while (!rc && done < total)
  {
    size_t want = (size_t) std::min<uint64_t>(chunk, total - done);
    if (std::fread(stage, 1, want, f) != want) { rc = set_error(LA3G_EIO, "%s: short read", path); break; }
    cudaError_t e = cudaMemcpy((char*) rec.p + done, stage, want, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) rc = set_error(LA3G_ECUDA, "upload failed: %s", cudaGetErrorString(e));
    done += want;
  }
  if (stage) cudaFreeHost(stage);
  std::fclose(f);
  if (!rc)
  {
    G->g.nrecords = nrec;
    rc = build_graph(G, rec, rec.as<uint32_t>(), rec.as<uint32_t>() + 1, rec.as<uint32_t>() + 2, wpr, nrec);
  }
  if (rc) { la3g_graph_free(G); return rc; }
  *out = G;
  return LA3G_OK;
}

extern "C" int la3g_graph_info_get(const la3g_graph* G, la3g_graph_info* out)
{
  if (!G || !out) return set_error(LA3G_EINVAL, "null argument");
  const DevGraph& g = G->g;
  std::memset(out, 0, sizeof *out);
  out->nslots = g.nslots;
  out->nvertices = g.nvertices;
  out->nleft = g.nleft;
  out->flags = g.flags;
  out->nrecords = g.nrecords;
  out->nentries = g.nent;
  out->nregular = g.nreg;
  out->nsink = g.nsink;
  out->nsource = g.nsrc;
  out->nisolated = g.nslots - g.nreg - g.nsink - g.nsrc;
  out->device_bytes = G->device_bytes;
  return LA3G_OK;
}

extern "C" int la3g_graph_positions(const la3g_graph* G, uint32_t* pos_of_id, uint32_t* id_of_pos)
{
  if (!G) return set_error(LA3G_EINVAL, "null graph");
  const DevGraph& g = G->g;
  if (pos_of_id) LA3G_CUDA(cudaMemcpy(pos_of_id, g.pos_of_id, (size_t) g.nslots * 4, cudaMemcpyDeviceToHost));
  if (id_of_pos) LA3G_CUDA(cudaMemcpy(id_of_pos, g.id_of_pos, (size_t) g.nslots * 4, cudaMemcpyDeviceToHost));
  return LA3G_OK;
}

extern "C" int la3g_graph_device_view(la3g_graph* G, la3g_device_graph* out)
{
  if (!G || !out) return set_error(LA3G_EINVAL, "null graph or output");
  const DevGraph& g = G->g;
  std::memset(out, 0, sizeof(*out));
  out->row_ptr = g.in_ptr;
  out->col = g.in_col;
  out->weight = g.weighted() ? g.in_w : nullptr;
  out->hash_of_pos = g.hash_of_pos;
  out->id_of_pos = g.id_of_pos;
  out->pos_of_id = g.pos_of_id;
  out->nslots = g.nslots;
  out->nregular = g.nreg;
  out->nsink = g.nsink;
  out->nsource = g.nsrc;
  out->flags = g.flags;
  out->nentries = g.nent;
  out->stream = (void*) G->stream;
  return LA3G_OK;
}

extern "C" int la3g_graph_push_view(la3g_graph* G, const uint32_t** out_ptr, const uint32_t** out_row)
{
  if (!G || !out_ptr || !out_row) return set_error(LA3G_EINVAL, "null graph or output");
  const DevGraph& g = G->g;
  if (g.directed()) LA3G_TRY(build_push_csr(G));
  *out_ptr = g.directed() ? g.out_ptr : g.in_ptr;
  *out_row = g.directed() ? g.out_row : g.in_col;
  return LA3G_OK;
}
