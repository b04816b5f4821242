// PageRank: the reference pr app (src/apps/graph_analytics/pr.cpp:11-55,
// pr.h:12-46) on the device.
//
// Reference semantics kept exactly:
//   * degree = number of distinct out-neighbours (DegVertex on the reversed
//     graph, pr.cpp:14-21, degree.h:24-35);
//   * rank starts at alpha = 0.15; x = rank / degree (pr.h:37);
//   * every iteration (the app is stationary) each regular row sums the
//     messages of its in-neighbours, source columns first, then regular
//     columns, each ascending (vertex_program_execute.hpp:479-482,
//     564-603), in FP64, one addition at a time in that order; then
//     rank = alpha + (1 - alpha) * y (pr.h:40-45);
//   * sinks are computed once after the iterations from the final regular
//     ranks (vertex_program_execute.hpp:131-148); sources and isolated
//     vertices keep alpha.
// Every floating-point operation is an explicit round-to-nearest intrinsic,
// so nothing is contracted into an FMA and the result is bit-identical to
// the reference built without contraction.
//
// Kernel layout: the calls run over a copy of the matrix made for them once
// per graph (see "the pull layout"): rows in descending length, columns
// renumbered in descending out-degree.  Rows of at most kShortRow in-edges
// (kShortRowFew on a graph of few rows) go a lane each, longer ones a warp each,
// the longest a block each; FP64 rows are summed in parallel with the result of
// the sequential sum (see "exact sums").
#include <algorithm>
#include <cstring>
#include <vector>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include "la3g_internal.h"

namespace la3g {

static constexpr double kAlpha = 0.15;
static constexpr double kTol = 1e-5;
static constexpr uint32_t kLongRow = 1024;  // longer rows: a block each
// Rows up to this: a lane each.  Of 64, 128, 256 and 512, 256 was fastest for
// FP32 on R-MAT 2^22 (50 iterations: 14.8, 14.5, 13.5, 14.3 ms) and as good as
// any for FP64 on R-MAT 2^16.
static constexpr uint32_t kShortRow = 256;
// On graphs of few rows, which leave SMs idle, a lane's chain of additions is
// what an iteration waits for, and more rows get a warp (limits 256, 64, 32;
// R-MAT, 50 FP32 / 20 FP64 iterations: 1024 x 8, 771, 463, 459 / 336, 297, 295 us;
// 33,001 x 12, 1080, 957, 898 / 507, 460, 494; 65,000 x 16, which has more rows
// than the line, 1305, 1512, 1531 / 596, 632, 648).
static constexpr uint32_t kShortRowFew = 64;
static constexpr uint32_t kFewRows = 1u << 15;
static constexpr int kWarpsPerBlock = 8;

// ---- the pull layout --------------------------------------------------------
//
// A pull is bound by its gathers x[col]: one random 4- or 8-byte read per
// edge, and at R-MAT 2^22 one column in a hundred is behind half of the
// edges.  By position those hot columns are spread over the whole of x, a
// 32-byte sector each, and L1 keeps few of them; numbered by descending
// out-degree ("slots") they share sectors and lines.
// Rows are numbered by descending in-degree ("q"; the regular rows, then the
// sinks), so that 32 neighbouring rows have almost the same length and can go
// a lane each: such a slice is stored column-major (step t of its lanes is
// contiguous), its rows padded to the first one's length with slot N, where x
// is 0.  The longer rows come first, each padded to a multiple of 4 entries
// (16-byte index loads).  Every row keeps the order of its entries, so sums
// come out as over the pull CSR.  FP32, R-MAT 2^22, 50 iterations: 34.0 ms over
// the pull CSR by position, 13.7 ms here (240 G edges/s); what is left is the
// L1 misses of the gathers (36 % hits; neither 32 to 200 KB of the hottest
// messages in shared memory nor L1 eviction hints were faster).
struct PrRange  // q's of one class (regular rows or sinks)
{
  uint32_t q0, q1, q2, q3;  // [q0, q1) above kLongRow, [q1, q2) above the slices' limit, [q2, q3) slices
};

struct PrLayout
{
  uint32_t* qpos = nullptr;  // [nslots] position of row q (identity beyond the rows)
  uint32_t* xi = nullptr;    // [nslots] slot of q's own message
  uint32_t* degq = nullptr;  // [nslots] out-degree of q
  uint64_t* off = nullptr;   // [nrows + 1] first entry of row q; of a slice: of its first row
  uint32_t* col = nullptr;   // the entries' slots
  PrRange reg{}, sink{};
};

struct PrScratch
{
  uint32_t* deg = nullptr;      // [nslots] out-degree by position
  PrLayout L;
  double* rank = nullptr;       // [nslots] by q
  double* x[2] = {nullptr, nullptr};  // [nslots + 1] messages (scatter values) by slot
  int* flag = nullptr;          // any-activated flag
  float* xf[2] = {nullptr, nullptr};  // FP32 study: messages by slot (tiled: by position)
  float* rankf = nullptr;       // by q (tiled: by position until the loop has ended)
  double* resid = nullptr;
  bool ready = false;
  // tiled layout of the regular rows (la3g_pr_f32_tiled), built on first use
  uint32_t ntiles = 0;
  uint64_t tile_ncols = 0, tile_nent = 0;
  uint32_t* tile_col = nullptr;  // [ntiles + 1] first non-empty-column slot of each tile
  uint32_t* tcol = nullptr;      // [ncols] column positions, ascending within a tile
  uint32_t* tptr = nullptr;      // [ncols + 1] first entry of each non-empty column
  uint16_t* trow = nullptr;      // [nent] row of each entry, local to its tile
  uint32_t* tecol = nullptr;     // [nent] column of each entry (the hypersparse tiles' form)
  float* trankf = nullptr;       // [nslots] by position
  float* txf[2] = {nullptr, nullptr};  // [nslots] by position
  int tile_blocks = 0;           // resident blocks per SM of the tiled kernel
  bool tiles_ready = false;
};

static void pr_scratch_free(void* p) { delete (PrScratch*) p; }

__global__ void k_outdeg(const uint32_t* __restrict__ col, uint64_t m, uint32_t* __restrict__ deg)
{
  for (uint64_t e = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x; e < m; e += (uint64_t) gridDim.x * blockDim.x)
    atomicAdd(&deg[col[e]], 1u);
}

// Sort keys of the columns (descending out-degree) and of the rows (regular
// before sinks, descending in-degree); `mask` is at least any degree.
__global__ void k_pr_keys(uint32_t N, uint32_t nrows, uint32_t nreg, uint32_t mask, const uint32_t* __restrict__ ptr,
                          const uint32_t* __restrict__ deg, uint32_t* ckey, uint32_t* rkey, uint32_t* iota)
{
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < N; p += gridDim.x * blockDim.x)
  {
    ckey[p] = mask - deg[p];
    if (p < nrows) rkey[p] = (p < nreg ? 0u : mask + 1) + (mask - (ptr[p + 1] - ptr[p]));
    iota[p] = p;
  }
}

// Row classes from the sorted keys: bounds[0..3] = q1, q2 of the regular rows,
// q1, q2 of the sinks (one thread each).
__global__ void k_pr_bounds(uint32_t nrows, uint32_t nreg, uint32_t mask, uint32_t short_row,
                            const uint32_t* __restrict__ rkey, uint32_t* bounds)
{
  const uint32_t t = threadIdx.x, lim = (t & 1) ? short_row : kLongRow;
  uint32_t lo = t < 2 ? 0 : nreg, hi = t < 2 ? nreg : nrows;
  const uint32_t key = (t < 2 ? 0u : mask + 1) + (mask > lim ? mask - lim : 0u);  // the first row with lim or fewer
  while (lo < hi)
  {
    const uint32_t mid = (lo + hi) >> 1;
    if (rkey[mid] < key) lo = mid + 1;
    else hi = mid;
  }
  bounds[t] = lo;
}

// Slot of each position; the rows' own arrays by q; the entries each row takes
// (a slice: its rows together, 32 or fewer, the first one's length each).
__global__ void k_pr_slots(uint32_t N, const uint32_t* __restrict__ order, uint32_t* slot)
{
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) slot[order[i]] = i;
}

__global__ void k_pr_rows(uint32_t N, uint32_t nrows, uint32_t nreg, uint32_t mask, const uint32_t* __restrict__ rkey,
                          const uint32_t* __restrict__ bounds, const uint32_t* __restrict__ deg,
                          const uint32_t* __restrict__ slot, uint32_t* qpos, uint32_t* xi, uint32_t* degq, uint64_t* take)
{
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < N; q += gridDim.x * blockDim.x)
  {
    if (q >= nrows) qpos[q] = q;
    const uint32_t p = q < nrows ? qpos[q] : q;
    xi[q] = slot[p];
    degq[q] = deg[p];
    if (q > nrows) continue;
    uint64_t n = 0;
    if (q < nrows)
    {
      const uint32_t q2 = bounds[q < nreg ? 1 : 3];
      if (q < q2) n = (mask - (rkey[q] & mask) + 3) & ~3u;
      else
      {
        n = mask - (rkey[q2 + ((q - q2) & ~31u)] & mask);
        // the last slice ends on a multiple of 4, where the sinks' long rows start
        if (q + 1 == (q < nreg ? nreg : nrows)) n += (0 - (((q - q2) & 31u) + 1) * n) & 3;
      }
    }
    take[q] = n;
  }
  if (nrows == N && blockIdx.x == 0 && threadIdx.x == 0) take[N] = 0;
}

// Blocks of a kernel over a PrRange: [0, nlong) a block per row, then nmed a
// warp per row, the rest a warp per slice.
struct PrBlocks
{
  uint32_t nlong, nmed, total;
};

static PrBlocks pr_blocks(const PrRange& r)
{
  PrBlocks b;
  b.nlong = std::min<uint32_t>(r.q1 - r.q0, num_sms() * 4);
  b.nmed = std::min<uint32_t>((r.q2 - r.q1 + kWarpsPerBlock - 1) / kWarpsPerBlock, num_sms() * 8);
  const uint32_t slices = (r.q3 - r.q2 + 31) / 32;
  b.total = b.nlong + b.nmed + std::min<uint32_t>((slices + kWarpsPerBlock - 1) / kWarpsPerBlock, num_sms() * 8);
  return b;
}

__global__ void __launch_bounds__(kWarpsPerBlock * 32)
k_pr_fill(PrRange R, PrBlocks B, const uint32_t* __restrict__ qpos, const uint64_t* __restrict__ off,
          const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ col, const uint32_t* __restrict__ slot,
          uint32_t zero, uint32_t* __restrict__ out)
{
  const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  if (blockIdx.x < B.nlong + B.nmed)
  {
    const bool block = blockIdx.x < B.nlong;  // a block or a warp per row
    const uint32_t step = block ? blockDim.x : 32, at = block ? threadIdx.x : lane;
    const uint32_t hi = block ? R.q1 : R.q2;
    uint32_t q = block ? R.q0 + blockIdx.x : R.q1 + (blockIdx.x - B.nlong) * kWarpsPerBlock + wib;
    for (; q < hi; q += block ? B.nlong : B.nmed * kWarpsPerBlock)
    {
      const uint32_t p = qpos[q], b = ptr[p], n = ptr[p + 1] - b;
      uint32_t* o = out + off[q];
      for (uint32_t i = at; i < ((n + 3) & ~3u); i += step) o[i] = i < n ? slot[col[b + i]] : zero;
    }
    return;
  }
  const uint32_t nw = (gridDim.x - B.nlong - B.nmed) * kWarpsPerBlock;
  for (uint32_t q0 = R.q2 + ((blockIdx.x - B.nlong - B.nmed) * kWarpsPerBlock + wib) * 32; q0 < R.q3; q0 += nw * 32)
  {
    const uint32_t cnt = min(32u, R.q3 - q0);
    uint32_t b = 0, n = 0;
    if (lane < cnt)
    {
      const uint32_t p = qpos[q0 + lane];
      b = ptr[p];
      n = ptr[p + 1] - b;
    }
    const uint32_t width = (uint32_t) (off[q0 + 1] - off[q0]);
    uint32_t* o = out + off[q0];
    if (lane < cnt)
      for (uint32_t t = 0; t < width; t++) o[t * cnt + lane] = t < n ? slot[col[b + t]] : zero;
  }
}

// x: regular and source vertices scatter rank / degree (init(vid, other, s)
// returns true for everyone, pr.h:34-37); sinks and isolated vertices have no
// out-edges and are never read as columns.  Slot N is the padding's.
template <class T>
__global__ void k_pr_init(uint32_t N, uint32_t nreg, uint32_t src_base, uint32_t iso_base,
                          const uint32_t* __restrict__ degq, const uint32_t* __restrict__ xi, T* rank, T* x0, T* x1)
{
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q <= N; q += gridDim.x * blockDim.x)
  {
    T xv = 0;
    if (q < N)
    {
      rank[q] = (T) kAlpha;
      if (q < nreg || (q >= src_base && q < iso_base)) xv = (T) kAlpha / (T) degq[q];
    }
    const uint32_t k = q < N ? xi[q] : N;
    x0[k] = xv;
    x1[k] = xv;
  }
}

// rank = alpha + (1 - alpha) * y with y = 0.0 + partial (combine into A()).
__device__ __forceinline__ double pr_apply(double partial)
{
  double y = __dadd_rn(0.0, partial);
  return __dadd_rn(kAlpha, __dmul_rn(1.0 - kAlpha, y));
}

__device__ __forceinline__ void pr_finish_row(uint32_t q, double acc, const PrLayout& L, double* rank, double* xnext,
                                              int* flag, bool write_x)
{
  double old = rank[q];
  double nr = pr_apply(acc);
  rank[q] = nr;
  if (write_x) xnext[L.xi[q]] = __ddiv_rn(nr, (double) L.degq[q]);
  if (flag && fabs(__dsub_rn(nr, old)) > kTol) *flag = 1;
}

// ---- exact sums --------------------------------------------------------------
//
// acc = RN(acc + v) one value after another, v >= 0, is a serial chain of
// FP64 additions (about 55 cycles each here: a 10k-edge row took 320 us).
// While acc stays inside one binade its ulp 2^e is fixed, and acc = m 2^e with
// an integer m: adding v adds v / 2^e rounded to an integer, which does not
// depend on m except that a tie goes to the even result.  One value is thus a
// function of m's parity, (increment if m is even, increment if m is odd), and
// such functions compose associatively: any stretch of a row that stays in one
// binade can be summed in parallel, in integers, with the sequential result
// bit for bit.  Where m would reach 2^53 (acc enters the next binade, at most
// once per doubling of the sum), the thread that holds that value adds its few
// values with real FP64 additions, and the rest is taken up with the new
// exponent.  On R-MAT 2^16 (1M edges): 328 -> 26 us per iteration.
struct ExactSum
{
  uint64_t m;  // value m 2^(e - 1075); m < 2^53
  int e;       // exponent field of the ulp's binade (1 for denormals); -1 while the sum is 0
};

struct ParityFn  // increments for m even / odd
{
  uint64_t a, b;
};

static constexpr uint64_t kExactTop = 1ull << 53;
// Consecutive values per thread and step: a step costs the functions of a
// thread's values and, at a new binade, as many FP64 additions (R-MAT 2^16, 20
// iterations, the whole call: 8 values 700 us, 4 values 630).
static constexpr int kExactPer = 4;
static constexpr int kAhead = 8;  // entries of a slice's lane per step

__device__ __forceinline__ ExactSum exact_of(double v)
{
  const uint64_t bits = (uint64_t) __double_as_longlong(v), f = bits & ((1ull << 52) - 1);
  const int e = (int) (bits >> 52);  // v >= 0
  if (!bits) return {0, -1};
  return e ? ExactSum{f | (1ull << 52), e} : ExactSum{f, 1};
}

__device__ __forceinline__ double exact_double(uint64_t m, int e)
{
  return m ? __longlong_as_double((long long) (((uint64_t) (e - 1) << 52) + m)) : 0.0;
}

// v as a function of m's parity, with ulp exponent e; an increment of
// kExactTop or more leaves the binade whatever m is.
__device__ __forceinline__ ParityFn exact_fn(double v, int e)
{
  const uint64_t bits = (uint64_t) __double_as_longlong(v);
  int ev = (int) (bits >> 52);
  uint64_t mant = bits & ((1ull << 52) - 1);
  if (ev) mant |= 1ull << 52;
  else ev = 1;
  const int s = e - ev;
  if (s < 0) return mant ? ParityFn{kExactTop, kExactTop} : ParityFn{0, 0};
  if (s > 53) return {0, 0};  // below half an ulp
  const uint64_t f = mant >> s;
  const uint64_t rem = s ? mant << (64 - s) : 0;  // the dropped bits, left-aligned
  const uint64_t up = rem > (1ull << 63), tie = rem == (1ull << 63);
  const uint64_t odd = f & 1;
  return {f + (tie ? odd : up), f + (tie ? odd ^ 1 : up)};
}

__device__ __forceinline__ ParityFn exact_then(ParityFn f, ParityFn g)
{
  return {f.a + ((f.a & 1) ? g.b : g.a), f.b + ((f.b & 1) ? g.a : g.b)};
}

__device__ __forceinline__ ParityFn exact_shfl_up(ParityFn f, int d)
{
  return {__shfl_up_sync(0xffffffffu, f.a, d), __shfl_up_sync(0xffffffffu, f.b, d)};
}

// A thread's kExactPer consecutive values from entry i of a row of n entries
// (both multiples of 4; entries beyond n count as 0, which adds nothing).
__device__ __forceinline__ void exact_load(const uint32_t* __restrict__ col, const double* __restrict__ x, uint32_t i,
                                           uint32_t n, double v[kExactPer])
{
#pragma unroll
  for (int k = 0; k < kExactPer; k += 4)
  {
    const bool in = i + k < n;
    uint4 c = make_uint4(0, 0, 0, 0);
    if (in) c = __ldcs(reinterpret_cast<const uint4*>(col + i + k));
    v[k] = in ? x[c.x] : 0.0;
    v[k + 1] = in ? x[c.y] : 0.0;
    v[k + 2] = in ? x[c.z] : 0.0;
    v[k + 3] = in ? x[c.w] : 0.0;
  }
}

__device__ __forceinline__ ParityFn exact_mine(const double (&v)[kExactPer], int e)
{
  ParityFn f{0, 0};
#pragma unroll
  for (int k = 0; k < kExactPer; k++) f = exact_then(f, exact_fn(v[k], e));
  return f;
}

// Inclusive scan over the warp's lanes, in lane order.
__device__ __forceinline__ ParityFn exact_scan(ParityFn f, int lane)
{
#pragma unroll
  for (int o = 1; o < 32; o <<= 1)
  {
    const ParityFn g = exact_shfl_up(f, o);
    if (lane >= o) f = exact_then(g, f);
  }
  return f;
}

// Adds a warp's entries, kExactPer per lane in lane order, to s.
__device__ __forceinline__ void exact_add_warp(const double (&v)[kExactPer], ExactSum& s, int lane)
{
  int from = 0;  // lanes below are in the sum already
  for (;;)
  {
    const ParityFn f = exact_scan(lane >= from ? exact_mine(v, s.e) : ParityFn{0, 0}, lane);
    const uint64_t incl = s.m + ((s.m & 1) ? f.b : f.a);
    const unsigned over = __ballot_sync(0xffffffffu, incl >= kExactTop);
    if (!over)
    {
      s.m = __shfl_sync(0xffffffffu, incl, 31);
      return;
    }
    const int L = __ffs(over) - 1;
    uint64_t before = __shfl_up_sync(0xffffffffu, incl, 1);
    if (lane == 0) before = s.m;
    double acc = 0.0;
    if (lane == L)
    {
      acc = exact_double(before, s.e);
#pragma unroll
      for (int k = 0; k < kExactPer; k++) acc = __dadd_rn(acc, v[k]);
    }
    s = exact_of(__shfl_sync(0xffffffffu, acc, L));
    from = L + 1;
    if (from == 32) return;
  }
}

// One row of n entries (a multiple of 4) by one warp.
__device__ __forceinline__ double exact_row_warp(const uint32_t* __restrict__ col, const double* __restrict__ x,
                                                 uint32_t n, int lane)
{
  ExactSum s{0, -1};
  double v[kExactPer];
  exact_load(col, x, lane * kExactPer, n, v);
  for (uint32_t base = 0; base < n; base += 32 * kExactPer)  // a warp's rows end at kLongRow
  {
    exact_add_warp(v, s, lane);
    if (base + 32 * kExactPer < n) exact_load(col, x, base + (32 + lane) * kExactPer, n, v);
  }
  return exact_double(s.m, s.e);
}

// One row of n entries (a multiple of 4) by one block (WARPS warps): the warps'
// functions meet in shared memory, every thread composes them and keeps its own
// copy of the sum.
template <int WARPS>
__device__ __forceinline__ double exact_row_block(const uint32_t* __restrict__ col, const double* __restrict__ x,
                                                  uint64_t n)
{
  __shared__ ParityFn s_fn[2][WARPS];
  __shared__ double s_acc;
  __shared__ int s_from;
  constexpr uint32_t kStep = WARPS * 32 * kExactPer;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  ExactSum s{0, -1};
  double v[kExactPer], nv[kExactPer];
  int buf = 0;
  const uint32_t at = threadIdx.x * kExactPer;
  exact_load(col, x, at, (uint32_t) min(n, (uint64_t) kStep), v);
  // the first entries leave a binade every few additions, and each time costs the
  // block two barriers: one warp takes them (20 iterations at 2^16 x 16, which the
  // longest row bounds: 612 us without this, 588 with)
  if (w == 0)
  {
    exact_add_warp(v, s, lane);
    if (lane == 0) s_acc = exact_double(s.m, s.e);
  }
  __syncthreads();
  s = exact_of(s_acc);
  for (uint64_t base = 0; base < n; base += kStep)
  {
    const uint64_t next = base + kStep;
    if (next < n) exact_load(col + next, x, at, (uint32_t) min(n - next, (uint64_t) kStep), nv);
    int from = base ? 0 : 32;
    for (;;)
    {
      const ParityFn f = exact_scan((int) threadIdx.x >= from ? exact_mine(v, s.e) : ParityFn{0, 0}, lane);
      if (lane == 31) s_fn[buf][w] = f;
      __syncthreads();
      uint64_t m = s.m, mine = 0;  // the sum before warp k; before this warp
      int cross = -1;
#pragma unroll
      for (int k = 0; k < WARPS; k++)
      {
        if (k == w) mine = m;
        const ParityFn g = s_fn[buf][k];
        if (cross < 0)
        {
          m += (m & 1) ? g.b : g.a;
          if (m >= kExactTop) cross = k;
        }
      }
      buf ^= 1;
      if (cross < 0)
      {
        s.m = m;
        break;
      }
      if (w == cross)
      {
        const uint64_t incl = mine + ((mine & 1) ? f.b : f.a);
        const int L = __ffs(__ballot_sync(0xffffffffu, incl >= kExactTop)) - 1;
        uint64_t before = __shfl_up_sync(0xffffffffu, incl, 1);
        if (lane == 0) before = mine;
        if (lane == L)
        {
          double acc = exact_double(before, s.e);
#pragma unroll
          for (int k = 0; k < kExactPer; k++) acc = __dadd_rn(acc, v[k]);
          s_acc = acc;
          s_from = w * 32 + L + 1;
        }
      }
      __syncthreads();
      s = exact_of(s_acc);
      from = s_from;
      if (from == WARPS * 32) break;
    }
#pragma unroll
    for (int k = 0; k < kExactPer; k++) v[k] = nv[k];
  }
  __syncthreads();  // s_fn, s_acc and s_from are free for the next row
  return exact_double(s.m, s.e);
}

// One pull over the rows of R.
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
k_pr_pull(PrRange R, PrBlocks B, PrLayout L, uint32_t zero, const double* __restrict__ x, double* __restrict__ xnext,
          double* __restrict__ rank, int* flag, int write_x)
{
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  if (blockIdx.x < B.nlong)
  {
    for (uint32_t q = R.q0 + blockIdx.x; q < R.q1; q += B.nlong)
    {
      const uint64_t o = L.off[q];
      const double acc = exact_row_block<kWarpsPerBlock>(L.col + o, x, L.off[q + 1] - o);
      if (threadIdx.x == 0) pr_finish_row(q, acc, L, rank, xnext, flag, write_x);
    }
    return;
  }
  if (blockIdx.x < B.nlong + B.nmed)
  {
    for (uint32_t q = R.q1 + (blockIdx.x - B.nlong) * kWarpsPerBlock + wib; q < R.q2; q += B.nmed * kWarpsPerBlock)
    {
      const uint64_t o = L.off[q];
      const double acc = exact_row_warp(L.col + o, x, (uint32_t) (L.off[q + 1] - o), lane);
      if (lane == 0) pr_finish_row(q, acc, L, rank, xnext, flag, write_x);
    }
    return;
  }
  const uint32_t first = B.nlong + B.nmed, nw = (gridDim.x - first) * kWarpsPerBlock;
  for (uint32_t q0 = R.q2 + ((blockIdx.x - first) * kWarpsPerBlock + wib) * 32; q0 < R.q3; q0 += nw * 32)
  {
    const uint32_t cnt = min(32u, R.q3 - q0), width = (uint32_t) (L.off[q0 + 1] - L.off[q0]);
    const uint32_t* col = L.col + L.off[q0] + lane;
    if ((uint32_t) lane >= cnt) continue;
    // one step of kAhead additions (a serial chain) while the next step's
    // messages and the slots of the one after are on their way
    double acc = 0.0, v[kAhead];
    uint32_t c[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; u++) c[u] = (uint32_t) u < width ? __ldcs(col + u * cnt) : zero;
#pragma unroll
    for (int u = 0; u < kAhead; u++) v[u] = x[c[u]];
#pragma unroll
    for (int u = 0; u < kAhead; u++) c[u] = kAhead + u < width ? __ldcs(col + (kAhead + u) * cnt) : zero;
    for (uint32_t t = 0; t < width; t += kAhead)
    {
      double nv[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; u++) nv[u] = x[c[u]];
#pragma unroll
      for (int u = 0; u < kAhead; u++) c[u] = t + 2 * kAhead + u < width ? __ldcs(col + (t + 2 * kAhead + u) * cnt) : zero;
#pragma unroll
      for (int u = 0; u < kAhead; u++) acc = __dadd_rn(acc, v[u]);
#pragma unroll
      for (int u = 0; u < kAhead; u++) v[u] = nv[u];
    }
    pr_finish_row(q0 + lane, acc, L, rank, xnext, flag, write_x);
  }
}

// Ranks by id; vertices that are not rows keep alpha (in FP64 in either form).
template <class T>
__global__ void k_rank_by_id(uint32_t N, uint32_t nrows, const uint32_t* __restrict__ qpos, const uint32_t* __restrict__ id_of_pos,
                             const T* __restrict__ rank, double* __restrict__ out)
{
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < N; q += gridDim.x * blockDim.x)
    out[id_of_pos[qpos[q]]] = q < nrows ? (double) rank[q] : kAlpha;
}

__global__ void k_scatter_pos_u32(uint32_t N, const uint32_t* __restrict__ id_of_pos, const uint32_t* __restrict__ val,
                                  uint32_t* __restrict__ out)
{
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < N; p += gridDim.x * blockDim.x) out[id_of_pos[p]] = val[p];
}

static int pr_prepare(la3g_graph* G, PrScratch** out)
{
  DevGraph& g = G->g;
  cudaStream_t s = G->stream;
  PrScratch* ps = (PrScratch*) G->slot[kSlotPr];
  if (ps && ps->ready) { *out = ps; return LA3G_OK; }
  if (!ps)
  {
    ps = new (std::nothrow) PrScratch();
    if (!ps) return set_error(LA3G_ENOMEM, "out of host memory");
    G->slot[kSlotPr] = ps;
    G->slot_free[kSlotPr] = pr_scratch_free;
  }
  const uint32_t N = g.nslots, nrows = g.nrows();
  PrLayout& L = ps->L;
  // Three allocations (an allocation costs 35 us or more, which a first call on a
  // small graph would feel): what is kept, the entries, and the working memory,
  // which holds the temporaries here and the ranks and messages of a call.
  auto round = [](size_t b) { return (b + 255) & ~(size_t) 255; };
  const size_t n4 = round((size_t) N * 4), n8 = round((size_t) N * 8 + 8);
  GallocScope scope(G);
  char* kept = nullptr;
  LA3G_TRY(galloc(G, &kept, 4 * n4 + n8 + 256));
  ps->deg = (uint32_t*) kept;
  L.qpos = (uint32_t*) (kept + n4);
  L.xi = (uint32_t*) (kept + 2 * n4);
  L.degq = (uint32_t*) (kept + 3 * n4);
  L.off = (decltype(L.off)) (kept + 4 * n4);
  ps->flag = (int*) (kept + 4 * n4 + n8);
  ps->resid = (double*) (ps->flag + 4);
  LA3G_CUDA(cudaMemsetAsync(ps->deg, 0, (size_t) N * 4, s));
  if (g.nent)
  {
    ProfileScope ps_("pr_outdeg", s, (double) g.nent * 4);
    k_outdeg<<<grid_for(g.nent, 256), 256, 0, s>>>(g.in_col, g.nent, ps->deg);
    LA3G_LAUNCHED();
  }
  // no self-loops and no duplicates: degrees are below N, which is at most 2^31
  int bits = 1;
  while (((uint64_t) (N - 1) >> bits) != 0) bits++;
  const uint32_t mask = (1u << bits) - 1;
  // temporaries: four key / value arrays and the slots, the rows' entry counts,
  // the class bounds, the library calls' storage
  size_t tb0 = 0, tb1 = 0;
  uint32_t* null32 = nullptr;
  uint64_t* null64 = nullptr;
  LA3G_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb0, null32, null32, null32, null32, (int64_t) N, 0, bits + 1, s));
  LA3G_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb1, null64, null64, (int64_t) nrows + 1, s));
  char* t = nullptr;
  LA3G_TRY(galloc(G, &t, std::max(5 * n4 + n8 + 256 + std::max(tb0, tb1), 3 * n8)));
  uint32_t *key = (uint32_t*) t, *rkey = (uint32_t*) (t + n4), *key2 = (uint32_t*) (t + 2 * n4);
  uint32_t *iota = (uint32_t*) (t + 3 * n4), *slot = (uint32_t*) (t + 4 * n4);
  uint64_t* take = (uint64_t*) (t + 5 * n4);
  uint32_t* bounds = (uint32_t*) (t + 5 * n4 + n8);
  void* lib = t + 5 * n4 + n8 + 256;
  k_pr_keys<<<grid_for(N, 256), 256, 0, s>>>(N, nrows, g.nreg, mask, g.in_ptr, ps->deg, key, rkey, iota);
  LA3G_LAUNCHED();
  uint32_t* order = L.xi;  // the columns' order, until xi is written
  LA3G_CUDA(cub::DeviceRadixSort::SortPairs(lib, tb0, key, key2, iota, order, (int64_t) N, 0, bits, s));
  k_pr_slots<<<grid_for(N, 256), 256, 0, s>>>(N, order, slot);
  LA3G_LAUNCHED();
  if (nrows)
  {
    LA3G_CUDA(cub::DeviceRadixSort::SortPairs(lib, tb0, rkey, key, iota, L.qpos, (int64_t) nrows, 0, bits + 1, s));
    k_pr_bounds<<<1, 4, 0, s>>>(nrows, g.nreg, mask, nrows <= kFewRows ? kShortRowFew : kShortRow, key, bounds);
    LA3G_LAUNCHED();
  }
  k_pr_rows<<<grid_for(N, 256), 256, 0, s>>>(N, nrows, g.nreg, mask, key, bounds, ps->deg, slot, L.qpos, L.xi, L.degq,
                                             take);
  LA3G_LAUNCHED();
  LA3G_CUDA(cub::DeviceScan::ExclusiveSum(lib, tb1, take, L.off, (int64_t) nrows + 1, s));
  uint32_t hb[4] = {0, 0, 0, 0};
  uint64_t total = 0;
  if (nrows) LA3G_CUDA(cudaMemcpyAsync(hb, bounds, 16, cudaMemcpyDeviceToHost, s));
  LA3G_CUDA(cudaMemcpyAsync(&total, L.off + nrows, 8, cudaMemcpyDeviceToHost, s));
  LA3G_CUDA(cudaStreamSynchronize(s));
  L.reg = PrRange{0, hb[0], hb[1], g.nreg};
  L.sink = PrRange{g.nreg, hb[2], hb[3], nrows};
  if (!nrows) L.sink = PrRange{0, 0, 0, 0};
  LA3G_TRY(galloc(G, &L.col, (size_t) total + 4));
  for (const PrRange& r : {L.reg, L.sink})
  {
    if (r.q3 == r.q0) continue;
    const PrBlocks b = pr_blocks(r);
    k_pr_fill<<<b.total, kWarpsPerBlock * 32, 0, s>>>(r, b, L.qpos, L.off, g.in_ptr, g.in_col, slot, N, L.col);
    LA3G_LAUNCHED();
  }
  LA3G_CUDA(cudaStreamSynchronize(s));
  // the FP64 and the FP32 form share the memory: neither leaves anything in it
  // for a later call
  ps->rank = (double*) t;
  ps->x[0] = (double*) (t + n8);
  ps->x[1] = (double*) (t + 2 * n8);
  ps->xf[0] = (float*) t;  // the results by id, 8 B each, take the place of both
  ps->xf[1] = (float*) (t + n8 / 2);
  ps->rankf = (float*) (t + n8);
  ps->ready = true;
  *out = ps;
  return scope.keep();
}

static int pr_launch(la3g_graph* G, PrScratch* ps, const PrRange& r, const double* x, double* xnext, int* flag,
                     bool write_x)
{
  DevGraph& g = G->g;
  const uint32_t rows = r.q3 - r.q0;
  if (!rows) return LA3G_OK;
  const PrBlocks b = pr_blocks(r);
  // algorithmic bytes: 4 B index per edge + per-row ptr, x, rank, xnext
  double bytes = 4.0 * (double) g.nent + 4.0 * (rows + 1) + 8.0 * (double) g.nslots + (write_x ? 16.0 : 8.0) * rows +
                 4.0 * rows;
  ProfileScope p("pr_pull_f64", G->stream, bytes);
  k_pr_pull<<<b.total, kWarpsPerBlock * 32, 0, G->stream>>>(r, b, ps->L, g.nslots, x, xnext, ps->rank, flag,
                                                            write_x ? 1 : 0);
  LA3G_LAUNCHED();
  return LA3G_OK;
}

// ------------------------------------------------------------------ FP32 study

__device__ __forceinline__ float prf_next(float acc) { return (float) kAlpha + (float) (1.0 - kAlpha) * acc; }

__device__ __forceinline__ double prf_finish(uint32_t q, float acc, const PrLayout& L, float* __restrict__ xnext,
                                             float* __restrict__ rankf, int write_x)
{
  const float nr = prf_next(acc);
  const double d = fabs((double) nr - (double) rankf[q]);
  rankf[q] = nr;
  if (write_x) xnext[L.xi[q]] = nr / (float) L.degq[q];
  return d;
}

// One FP32 pull over the rows of R, FP32 accumulation.  A row of at most
// kLongRow entries has four partial sums, entry i in sum i % 4, combined
// (0 + 2) + (1 + 3): a lane holds all four in a slice, a group of four lanes
// one each above the slices' limit.  A longer row has one per thread of its block.
// The L1 residual is reduced in FP64.
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
k_prf_pull(PrRange R, PrBlocks B, PrLayout L, uint32_t zero, const float* __restrict__ x, float* __restrict__ xnext,
           float* __restrict__ rankf, double* resid, int write_x)
{
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  double local = 0.0;
  if (blockIdx.x < B.nlong)
  {
    __shared__ float part[kWarpsPerBlock];
    for (uint32_t q = R.q0 + blockIdx.x; q < R.q1; q += B.nlong)
    {
      const uint64_t o = L.off[q], n = L.off[q + 1] - o;
      const uint32_t* col = L.col + o;
      float acc = 0.0f;
      for (uint64_t i = threadIdx.x; i < n; i += 4 * kWarpsPerBlock * 32)
      {
        float v[4];
#pragma unroll
        for (int u = 0; u < 4; u++)
        {
          const uint64_t k = i + u * kWarpsPerBlock * 32;
          v[u] = x[k < n ? __ldcs(col + k) : zero];
        }
#pragma unroll
        for (int u = 0; u < 4; u++) acc += v[u];
      }
#pragma unroll
      for (int o2 = 16; o2 > 0; o2 >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o2);
      if (lane == 0) part[wib] = acc;
      __syncthreads();
      if (threadIdx.x == 0)
      {
        float t = 0.0f;
        for (int w = 0; w < kWarpsPerBlock; w++) t += part[w];
        local += prf_finish(q, t, L, xnext, rankf, write_x);
      }
      __syncthreads();
    }
  }
  else if (blockIdx.x < B.nlong + B.nmed)
  {
    // eight rows per warp, four lanes each; a warp's lanes go round together
    const uint32_t sub = lane & 3;
    const uint32_t nw = B.nmed * kWarpsPerBlock;
    for (uint32_t q0 = R.q1 + ((blockIdx.x - B.nlong) * kWarpsPerBlock + wib) * 8; q0 < R.q2; q0 += nw * 8)
    {
      const uint32_t q = q0 + (lane >> 2);
      float acc = 0.0f;
      if (q < R.q2)
      {
        const uint64_t o = L.off[q];
        const uint32_t n = (uint32_t) (L.off[q + 1] - o);
        const uint32_t* col = L.col + o;
        for (uint32_t i = sub; i < n; i += 32)
        {
          float v[8];
#pragma unroll
          for (int u = 0; u < 8; u++) v[u] = x[i + 4 * u < n ? __ldcs(col + i + 4 * u) : zero];
#pragma unroll
          for (int u = 0; u < 8; u++) acc += v[u];
        }
      }
      acc += __shfl_xor_sync(0xffffffffu, acc, 2);
      acc += __shfl_xor_sync(0xffffffffu, acc, 1);
      if (q < R.q2 && sub == 0) local += prf_finish(q, acc, L, xnext, rankf, write_x);
    }
  }
  else
  {
    const uint32_t first = B.nlong + B.nmed, nw = (gridDim.x - first) * kWarpsPerBlock;
    for (uint32_t q0 = R.q2 + ((blockIdx.x - first) * kWarpsPerBlock + wib) * 32; q0 < R.q3; q0 += nw * 32)
    {
      const uint32_t cnt = min(32u, R.q3 - q0), width = (uint32_t) (L.off[q0 + 1] - L.off[q0]);
      const uint32_t* col = L.col + L.off[q0] + lane;
      if ((uint32_t) lane >= cnt) continue;
      float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      for (uint32_t t = 0; t < width; t += 8)
      {
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; u++) v[u] = x[t + u < width ? __ldcs(col + (t + u) * cnt) : zero];
#pragma unroll
        for (int u = 0; u < 8; u++) acc[u & 3] += v[u];
      }
      local += prf_finish(q0 + lane, (acc[0] + acc[2]) + (acc[1] + acc[3]), L, xnext, rankf, write_x);
    }
  }
  // one FP64 atomic per block (per-warp atomics on one word serialise)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
  __shared__ double wsum[kWarpsPerBlock];
  if (lane == 0) wsum[wib] = local;
  __syncthreads();
  if (threadIdx.x == 0)
  {
    double t = 0.0;
    for (int w = 0; w < kWarpsPerBlock; w++) t += wsum[w];
    if (t != 0.0) atomicAdd(resid, t);
  }
}

// ------------------------------------------------------------- tiled layout
//
// The regular rows are cut into tiles of kTileRows consecutive rows.  Each
// tile keeps its entries doubly compressed by column (the reference's
// per-tile DCSC, src/utils/csc.h:60-130: only the non-empty columns are
// listed, with their offsets): tcol / tptr over the tile's non-empty columns
// in ascending position, and a 16-bit row inside the tile per entry.  One
// CTA takes a tile at a time with its rows' accumulators in shared memory,
// walks the tile's columns (one thread per column, four columns' messages
// loaded at once; columns with many entries in the tile go to whole warps)
// and adds each column's message into its rows with shared-memory atomics,
// so every message is read once per tile and no row needs a reduction across
// lanes.  Rows with more than kLongRow in-edges stay out of the tiles (their
// thousands of additions would serialise on one shared-memory word) and are
// summed a block each by the first blocks of the same launch.
// Addition order inside a row is free in the FP32 study (the FP64 path keeps
// the reference's order on the flat CSR).
static constexpr uint32_t kTileRows = 2048;    // rows per tile: 8 KB of FP32 accumulators
static constexpr uint32_t kTileThreads = 512;
static constexpr uint32_t kTileBig = 32;       // columns with more entries in a tile go to a warp
static constexpr uint32_t kTileBigCap = 1024;  // such columns queued per tile (the rest run serially)
static constexpr uint32_t kTileDense = 2;      // entries per non-empty column at which a tile walks its DCSC columns

__global__ void k_tile_colof(const uint32_t* __restrict__ ptr, uint32_t ncol, uint32_t* colof)
{
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < ncol; c += gridDim.x * blockDim.x)
    for (uint32_t i = ptr[c]; i < ptr[c + 1]; i++) colof[i] = c;
}

// Tile of each push entry; entries of sink rows and of long regular rows
// (more than kLongRow in-edges: summed by the flat kernel's block-per-row
// path, since thousands of additions into one shared-memory word would
// serialise) sort last and are dropped.
__global__ void k_tile_keys(const uint32_t* __restrict__ row, uint64_t m, uint32_t nreg,
                            const uint32_t* __restrict__ in_ptr, uint32_t* key, uint32_t* idx,
                            unsigned long long* kept)
{
  unsigned long long c = 0;
  for (uint64_t i = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; i < m; i += (uint64_t) gridDim.x * blockDim.x)
  {
    const uint32_t r = row[i];
    const bool keep = r < nreg && in_ptr[r + 1] - in_ptr[r] <= kLongRow;
    key[i] = keep ? r / kTileRows : 0xFFFFFFFFu;
    idx[i] = (uint32_t) i;
    c += keep;
  }
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(kept, c);
}

// Entries in (tile, column, row) order: local rows, and a flag where a new
// (tile, column) pair starts.
__global__ void k_tile_flags(const uint32_t* __restrict__ order, uint64_t n, const uint32_t* __restrict__ colof,
                             const uint32_t* __restrict__ row, uint16_t* trow, uint32_t* tecol, uint32_t* flag)
{
  for (uint64_t e = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; e < n; e += (uint64_t) gridDim.x * blockDim.x)
  {
    const uint32_t i = order[e];
    const uint32_t r = row[i], t = r / kTileRows;
    trow[e] = (uint16_t) (r - t * kTileRows);
    tecol[e] = colof[i];
    bool start = e == 0;
    if (!start)
    {
      const uint32_t j = order[e - 1];
      start = colof[j] != colof[i] || row[j] / kTileRows != t;
    }
    flag[e] = start ? 1u : 0u;
  }
}

__global__ void k_tile_cols(const uint32_t* __restrict__ order, uint64_t n, const uint32_t* __restrict__ colof,
                            const uint32_t* __restrict__ row, const uint32_t* __restrict__ flag,
                            const uint32_t* __restrict__ slot, uint32_t* tcol, uint32_t* tptr, uint32_t* tile_col)
{
  for (uint64_t e = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; e < n; e += (uint64_t) gridDim.x * blockDim.x)
  {
    if (!flag[e]) continue;
    const uint32_t i = order[e], k = slot[e];
    tcol[k] = colof[i];
    tptr[k] = (uint32_t) e;
    const uint32_t t = row[i] / kTileRows;
    if (e == 0 || row[order[e - 1]] / kTileRows != t) tile_col[t] = k;
  }
}

// The push CSR has to be there.
static int pr_build_tiles(la3g_graph* G, PrScratch* ps)
{
  DevGraph& g = G->g;
  cudaStream_t s = G->stream;
  const uint64_t m = g.nent;
  const uint32_t ntiles = (g.nreg + kTileRows - 1) / kTileRows;
  DevBuf colof, key, key2, idx, idx2, flag, slot, tmp, kept;
  LA3G_TRY(kept.alloc(8));
  LA3G_CUDA(cudaMemsetAsync(kept.p, 0, 8, s));
  LA3G_TRY(colof.alloc(m * 4 + 4));
  LA3G_TRY(key.alloc(m * 4 + 4));
  LA3G_TRY(key2.alloc(m * 4 + 4));
  LA3G_TRY(idx.alloc(m * 4 + 4));
  LA3G_TRY(idx2.alloc(m * 4 + 4));
  if (m)
  {
    k_tile_colof<<<grid_for(g.nslots, 256), 256, 0, s>>>(g.out_ptr, g.nslots, colof.as<uint32_t>());
    LA3G_LAUNCHED();
    k_tile_keys<<<grid_for(m, 256), 256, 0, s>>>(g.out_row, m, g.nreg, g.in_ptr, key.as<uint32_t>(), idx.as<uint32_t>(),
                                                 kept.as<unsigned long long>());
    LA3G_LAUNCHED();
    // stable by tile: the push CSR's (column, row) order is kept inside each tile
    size_t tb = 0;
    LA3G_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, key.as<uint32_t>(), key2.as<uint32_t>(), idx.as<uint32_t>(),
                                              idx2.as<uint32_t>(), (int64_t) m, 0, 32, s));
    LA3G_TRY(tmp.alloc(tb));
    LA3G_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, tb, key.as<uint32_t>(), key2.as<uint32_t>(), idx.as<uint32_t>(),
                                              idx2.as<uint32_t>(), (int64_t) m, 0, 32, s));
  }
  // the kept entries sort first
  unsigned long long nkept = 0;
  LA3G_CUDA(cudaMemcpyAsync(&nkept, kept.p, 8, cudaMemcpyDeviceToHost, s));
  LA3G_CUDA(cudaStreamSynchronize(s));
  const uint64_t n = nkept;
  LA3G_TRY(flag.alloc(n * 4 + 4));
  LA3G_TRY(slot.alloc(n * 4 + 4));
  LA3G_TRY(galloc(G, &ps->trow, n + 8));
  LA3G_TRY(galloc(G, &ps->tecol, n + 8));
  uint32_t ncols = 0;
  if (n)
  {
    k_tile_flags<<<grid_for(n, 256), 256, 0, s>>>(idx2.as<uint32_t>(), n, colof.as<uint32_t>(), g.out_row, ps->trow,
                                                  ps->tecol, flag.as<uint32_t>());
    LA3G_LAUNCHED();
    size_t tb = 0;
    LA3G_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, flag.as<uint32_t>(), slot.as<uint32_t>(), (int64_t) n, s));
    LA3G_TRY(tmp.alloc(tb));
    LA3G_CUDA(cub::DeviceScan::ExclusiveSum(tmp.p, tb, flag.as<uint32_t>(), slot.as<uint32_t>(), (int64_t) n, s));
    uint32_t last[2];
    LA3G_CUDA(cudaMemcpyAsync(&last[0], slot.as<uint32_t>() + n - 1, 4, cudaMemcpyDeviceToHost, s));
    LA3G_CUDA(cudaMemcpyAsync(&last[1], flag.as<uint32_t>() + n - 1, 4, cudaMemcpyDeviceToHost, s));
    LA3G_CUDA(cudaStreamSynchronize(s));
    ncols = last[0] + last[1];
  }
  LA3G_TRY(galloc(G, &ps->tcol, (size_t) ncols + 1));
  LA3G_TRY(galloc(G, &ps->tptr, (size_t) ncols + 1));
  LA3G_TRY(galloc(G, &ps->tile_col, (size_t) ntiles + 1));
  std::vector<uint32_t> tc(ntiles + 1, ncols);
  LA3G_CUDA(cudaMemcpyAsync(ps->tile_col, tc.data(), tc.size() * 4, cudaMemcpyHostToDevice, s));
  if (n)
  {
    k_tile_cols<<<grid_for(n, 256), 256, 0, s>>>(idx2.as<uint32_t>(), n, colof.as<uint32_t>(), g.out_row,
                                                 flag.as<uint32_t>(), slot.as<uint32_t>(), ps->tcol, ps->tptr,
                                                 ps->tile_col);
    LA3G_LAUNCHED();
  }
  const uint32_t end = (uint32_t) n;
  LA3G_CUDA(cudaMemcpyAsync(ps->tptr + ncols, &end, 4, cudaMemcpyHostToDevice, s));
  // empty tiles start where the next tile starts
  LA3G_CUDA(cudaMemcpyAsync(tc.data(), ps->tile_col, tc.size() * 4, cudaMemcpyDeviceToHost, s));
  LA3G_CUDA(cudaStreamSynchronize(s));
  for (int64_t t = (int64_t) ntiles - 1; t >= 0; t--) tc[t] = std::min(tc[t], tc[t + 1]);
  LA3G_CUDA(cudaMemcpyAsync(ps->tile_col, tc.data(), tc.size() * 4, cudaMemcpyHostToDevice, s));
  LA3G_CUDA(cudaStreamSynchronize(s));
  ps->ntiles = ntiles;
  ps->tile_ncols = ncols;
  ps->tile_nent = n;
  return LA3G_OK;
}

__global__ void k_prf_tile_init(uint32_t N, uint32_t nreg, uint32_t src_base, uint32_t iso_base,
                                const uint32_t* __restrict__ deg, float* rankf, float* x0, float* x1)
{
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < N; p += gridDim.x * blockDim.x)
  {
    rankf[p] = (float) kAlpha;
    const bool scat = p < nreg || (p >= src_base && p < iso_base);
    x0[p] = x1[p] = scat ? (float) kAlpha / (float) deg[p] : 0.0f;
  }
}

__device__ __forceinline__ double prf_tile_finish(uint32_t p, float acc, float* __restrict__ xnext,
                                                  float* __restrict__ rankf, const uint32_t* __restrict__ deg)
{
  const float nr = prf_next(acc);
  const double d = fabs((double) nr - (double) rankf[p]);
  rankf[p] = nr;
  xnext[p] = nr / (float) deg[p];
  return d;
}

// The tiled loop's results in the pull layout, for the sink pass and the output.
__global__ void k_prf_from_tiles(uint32_t N, const uint32_t* __restrict__ qpos, const uint32_t* __restrict__ xi,
                                 const float* __restrict__ trankf, const float* __restrict__ tx, float* rankf, float* x)
{
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q <= N; q += gridDim.x * blockDim.x)
  {
    if (q == N)
    {
      x[N] = 0.0f;
      continue;
    }
    const uint32_t p = qpos[q];
    rankf[q] = trankf[p];
    x[xi[q]] = tx[p];
  }
}

__global__ void __launch_bounds__(kTileThreads)
k_prf_tiles(const uint32_t* __restrict__ tile_col, const uint32_t* __restrict__ tcol,
            const uint32_t* __restrict__ tptr, const uint16_t* __restrict__ trow,
            const uint32_t* __restrict__ tecol, uint32_t ntiles, uint32_t nreg,
            const uint32_t* __restrict__ in_ptr, const uint32_t* __restrict__ in_col,
            const uint32_t* __restrict__ long_rows, uint32_t nlong, uint32_t long_blocks,
            const float* __restrict__ x, float* __restrict__ xnext, float* __restrict__ rankf,
            const uint32_t* __restrict__ deg, double* resid)
{
  extern __shared__ float ys[];  // kTileRows accumulators
  __shared__ uint32_t s_big[kTileBigCap];
  __shared__ uint32_t s_nbig;
  __shared__ double s_part[kTileThreads / 32];
  __shared__ float s_lpart[kTileThreads / 32];
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double local = 0.0;
  // the first long_blocks blocks: the long rows, a block each, from the flat CSR
  for (uint32_t k = blockIdx.x; blockIdx.x < long_blocks && k < nlong; k += long_blocks)
  {
    const uint32_t r = long_rows[k];
    float acc = 0.0f;
    for (uint32_t i = in_ptr[r] + tid; i < in_ptr[r + 1]; i += kTileThreads) acc += x[in_col[i]];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) s_lpart[warp] = acc;
    __syncthreads();
    if (tid == 0)
    {
      float t = 0.0f;
      for (uint32_t w = 0; w < kTileThreads / 32; w++) t += s_lpart[w];
      local += prf_tile_finish(r, t, xnext, rankf, deg);
    }
    __syncthreads();
  }
  const uint32_t tblocks = gridDim.x - long_blocks;
  for (uint32_t t = blockIdx.x - long_blocks; blockIdx.x >= long_blocks && t < ntiles; t += tblocks)
  {
    const uint32_t r0 = t * kTileRows, nr = min(kTileRows, nreg - r0);
    for (uint32_t i = tid; i < nr; i += kTileThreads) ys[i] = 0.0f;
    if (tid == 0) s_nbig = 0;
    __syncthreads();
    const uint32_t k0 = tile_col[t], k1 = tile_col[t + 1];
    const uint32_t e0 = tptr[k0], e1 = tptr[k1];
    // hypersparse tile (fewer than kTileDense entries per non-empty column):
    // a thread per entry, its column from the per-entry form, four entries in
    // flight; denser tiles walk their DCSC columns, each message read once
    const bool by_entry = (uint64_t) (e1 - e0) < (uint64_t) kTileDense * (k1 - k0);
    for (uint32_t eb = e0; by_entry && eb < e1; eb += 4 * kTileThreads)
    {
      float xv[4];
      uint32_t rr[4];
#pragma unroll
      for (int u = 0; u < 4; u++)
      {
        const uint32_t e = eb + u * kTileThreads + tid;
        rr[u] = e < e1 ? trow[e] : 0xFFFFFFFFu;
        xv[u] = e < e1 ? x[tecol[e]] : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (rr[u] != 0xFFFFFFFFu) atomicAdd(&ys[rr[u]], xv[u]);
    }
    // a thread per column, four columns' messages in flight
    for (uint32_t kb = k0; !by_entry && kb < k1; kb += 4 * kTileThreads)
    {
      uint32_t b[4], e[4];
      float xv[4];
#pragma unroll
      for (int u = 0; u < 4; u++)
      {
        const uint32_t k = kb + u * kTileThreads + tid;
        b[u] = e[u] = 0;
        if (k < k1)
        {
          b[u] = tptr[k];
          e[u] = tptr[k + 1];
        }
      }
#pragma unroll
      for (int u = 0; u < 4; u++)
      {
        const uint32_t k = kb + u * kTileThreads + tid;
        xv[u] = (k < k1 && e[u] - b[u] <= kTileBig) ? x[tcol[k]] : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < 4; u++)
      {
        const uint32_t k = kb + u * kTileThreads + tid;
        if (k >= k1) continue;
        if (e[u] - b[u] > kTileBig)
        {
          const uint32_t q = atomicAdd(&s_nbig, 1u);
          if (q < kTileBigCap)
          {
            s_big[q] = k;
            continue;
          }
          xv[u] = x[tcol[k]];  // queue full: this thread adds the column itself
        }
        for (uint32_t j = b[u]; j < e[u]; j++) atomicAdd(&ys[trow[j]], xv[u]);
      }
    }
    __syncthreads();
    const uint32_t nb = min(s_nbig, kTileBigCap);
    for (uint32_t q = warp; q < nb; q += kTileThreads / 32)
    {
      const uint32_t k = s_big[q];
      const float v = x[tcol[k]];
      for (uint32_t j = tptr[k] + lane; j < tptr[k + 1]; j += 32) atomicAdd(&ys[trow[j]], v);
    }
    __syncthreads();
    for (uint32_t i = tid; i < nr; i += kTileThreads)
      if (in_ptr[r0 + i + 1] - in_ptr[r0 + i] <= kLongRow)  // long rows are finished by the flat kernel
        local += prf_tile_finish(r0 + i, ys[i], xnext, rankf, deg);
    __syncthreads();
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
  if (lane == 0) s_part[warp] = local;
  __syncthreads();
  if (tid == 0)
  {
    double sum = 0.0;
    for (uint32_t w = 0; w < kTileThreads / 32; w++) sum += s_part[w];
    if (sum != 0.0) atomicAdd(resid, sum);
  }
}

}  // namespace la3g

using namespace la3g;

extern "C" int la3g_pr(la3g_graph* G, uint32_t iters, double* rank_out, uint32_t* degree_out, la3g_stats* st)
{
  if (!G) return set_error(LA3G_EINVAL, "null graph");
  DevGraph& g = G->g;
  if (!g.directed() || (g.flags & (LA3G_REVERSE | LA3G_ACYCLIC | LA3G_BIPARTITE)))
    return set_error(LA3G_EINVAL, "pagerank needs a graph loaded with LA3G_DIRECTED only");
  CallTimer T(G, st);
  PrScratch* ps = nullptr;
  LA3G_TRY(pr_prepare(G, &ps));
  cudaStream_t s = G->stream;
  const uint32_t N = g.nslots;
  T.device_begin();
  k_pr_init<double><<<grid_for((uint64_t) N + 1, 256), 256, 0, s>>>(N, g.nreg, g.src_base(), g.iso_base(), ps->L.degq,
                                                                    ps->L.xi, ps->rank, ps->x[0], ps->x[1]);
  LA3G_LAUNCHED();
  tls_launches++;
  uint32_t it = 0;
  int cur = 0;
  const bool until = iters == 0;
  for (;;)
  {
    if (!until && it >= iters) break;
    if (until) LA3G_CUDA(cudaMemsetAsync(ps->flag, 0, 4, s));
    LA3G_TRY(pr_launch(G, ps, ps->L.reg, ps->x[cur], ps->x[cur ^ 1], until ? ps->flag : nullptr, true));
    cur ^= 1;
    it++;
    if (until)
    {
      int f = 0;
      LA3G_CUDA(cudaMemcpyAsync(&f, ps->flag, 4, cudaMemcpyDeviceToHost, s));
      LA3G_CUDA(cudaStreamSynchronize(s));
      if (!f) break;
    }
  }
  // sink pass from the final messages (vertex_program_execute.hpp:131-148)
  LA3G_TRY(pr_launch(G, ps, ps->L.sink, ps->x[cur], ps->x[cur ^ 1], nullptr, false));
  T.device_end();
  if (st)
  {
    st->iterations = it;
    st->teps_edges = (uint64_t) it * g.nent;
    st->edges_examined = (uint64_t) it * g.nent + g.nent;
    st->algo_bytes = (uint64_t) ((4.0 * g.nent + 28.0 * N) * it);
  }
  // the results by id, in the message buffers, which are free now (a buffer for
  // each call cost its allocation and release, 65 us of a 680 us call at 2^16)
  if (rank_out)
  {
    k_rank_by_id<double><<<grid_for(N, 256), 256, 0, s>>>(N, g.nrows(), ps->L.qpos, g.id_of_pos, ps->rank, ps->x[0]);
    LA3G_LAUNCHED();
    LA3G_CUDA(cudaMemcpyAsync(rank_out, ps->x[0], (size_t) N * 8, cudaMemcpyDeviceToHost, s));
  }
  if (degree_out)
  {
    uint32_t* out = (uint32_t*) ps->x[1];
    k_scatter_pos_u32<<<grid_for(N, 256), 256, 0, s>>>(N, g.id_of_pos, ps->deg, out);
    LA3G_LAUNCHED();
    LA3G_CUDA(cudaMemcpyAsync(degree_out, out, (size_t) N * 4, cudaMemcpyDeviceToHost, s));
  }
  return T.finish();
}

static int pr_f32_run(la3g_graph* G, uint32_t iters, double tol, double* rank_out, double* residual_out,
                      la3g_stats* st, bool tiled)
{
  if (!G) return set_error(LA3G_EINVAL, "null graph");
  DevGraph& g = G->g;
  if (!g.directed() || (g.flags & (LA3G_REVERSE | LA3G_ACYCLIC | LA3G_BIPARTITE)))
    return set_error(LA3G_EINVAL, "pagerank needs a graph loaded with LA3G_DIRECTED only");
  if (iters == 0) return set_error(LA3G_EINVAL, "iters must be > 0");
  CallTimer T(G, st);
  PrScratch* ps = nullptr;
  LA3G_TRY(pr_prepare(G, &ps));
  cudaStream_t s = G->stream;
  const uint32_t N = g.nslots;
  if (tiled && !ps->tiles_ready)
  {
    LA3G_TRY(build_push_csr(G));
    GallocScope scope(G);
    LA3G_TRY(pr_build_tiles(G, ps));
    LA3G_CUDA(cudaFuncSetAttribute(k_prf_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) (kTileRows * 4)));
    LA3G_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ps->tile_blocks, k_prf_tiles, kTileThreads,
                                                            kTileRows * 4));
    LA3G_TRY(galloc(G, &ps->trankf, N));
    LA3G_TRY(galloc(G, &ps->txf[0], N));
    LA3G_TRY(galloc(G, &ps->txf[1], N));
    ps->tiles_ready = true;
    scope.keep();
  }
  const PrLayout& L = ps->L;
  const uint32_t nlong = L.reg.q1;  // regular rows above kLongRow: qpos[0 .. nlong)
  T.device_begin();
  if (tiled)
    k_prf_tile_init<<<grid_for(N, 256), 256, 0, s>>>(N, g.nreg, g.src_base(), g.iso_base(), ps->deg, ps->trankf,
                                                     ps->txf[0], ps->txf[1]);
  else
    k_pr_init<float><<<grid_for((uint64_t) N + 1, 256), 256, 0, s>>>(N, g.nreg, g.src_base(), g.iso_base(), L.degq, L.xi,
                                                                     ps->rankf, ps->xf[0], ps->xf[1]);
  LA3G_LAUNCHED();
  tls_launches++;
  int cur = 0;
  uint32_t it = 0;
  double res = 0.0;
  const PrBlocks rb = pr_blocks(L.reg), sb = pr_blocks(L.sink);
  // algorithmic bytes per iteration (FP32 form of the FP64 count): column
  // index per edge, row offsets, x read, rank read + write, next x write
  const double it_bytes = 4.0 * g.nent + 4.0 * (g.nreg + 1) + 4.0 * N + 8.0 * g.nreg + 8.0 * g.nreg + 4.0 * g.nreg;
  for (; it < iters;)
  {
    // the residual is looked at after every iteration, or after the last one only
    if (tol > 0 || it + 1 == iters) LA3G_CUDA(cudaMemsetAsync(ps->resid, 0, 8, s));
    if (tiled)
    {
      // per tile: its non-empty columns (index, offset, message) and 2 B per
      // entry, then the rows' rank read + write and next message write
      ProfileScope p("pr_tiles_f32", s, 12.0 * ps->tile_ncols + 2.0 * ps->tile_nent + 4.0 * (g.nreg + 1) + 8.0 * g.nreg +
                                            8.0 * g.nreg + 4.0 * g.nreg);
      // long rows first (a block each), then the tiles
      const uint32_t lblocks = std::min<uint32_t>(nlong, num_sms());
      const unsigned tgrid = std::min<unsigned>(std::max<uint32_t>(ps->ntiles, 1), num_sms() * std::max(ps->tile_blocks, 1));
      k_prf_tiles<<<lblocks + tgrid, kTileThreads, kTileRows * 4, s>>>(
          ps->tile_col, ps->tcol, ps->tptr, ps->trow, ps->tecol, ps->ntiles, g.nreg, g.in_ptr, g.in_col, L.qpos, nlong,
          lblocks, ps->txf[cur], ps->txf[cur ^ 1], ps->trankf, ps->deg, ps->resid);
      LA3G_LAUNCHED();
    }
    else if (g.nreg)
    {
      ProfileScope p("pr_pull_f32", s, it_bytes);
      k_prf_pull<<<rb.total, kWarpsPerBlock * 32, 0, s>>>(L.reg, rb, L, N, ps->xf[cur], ps->xf[cur ^ 1], ps->rankf,
                                                          ps->resid, 1);
      LA3G_LAUNCHED();
    }
    cur ^= 1;
    it++;
    if (tol > 0)
    {
      LA3G_CUDA(cudaMemcpyAsync(&res, ps->resid, 8, cudaMemcpyDeviceToHost, s));
      LA3G_CUDA(cudaStreamSynchronize(s));
      if (res < tol) break;
    }
  }
  // the residual of the last iteration (the sink pass below reuses the counter)
  if (tol <= 0) LA3G_CUDA(cudaMemcpyAsync(&res, ps->resid, 8, cudaMemcpyDeviceToHost, s));
  if (tiled)
  {
    k_prf_from_tiles<<<grid_for((uint64_t) N + 1, 256), 256, 0, s>>>(N, L.qpos, L.xi, ps->trankf, ps->txf[cur],
                                                                     ps->rankf, ps->xf[cur]);
    LA3G_LAUNCHED();
  }
  if (g.nsink)
  {
    LA3G_CUDA(cudaMemsetAsync(ps->resid, 0, 8, s));
    k_prf_pull<<<sb.total, kWarpsPerBlock * 32, 0, s>>>(L.sink, sb, L, N, ps->xf[cur], ps->xf[cur ^ 1], ps->rankf,
                                                        ps->resid, 0);
    LA3G_LAUNCHED();
  }
  T.device_end();
  if (st)
  {
    st->iterations = it;
    st->teps_edges = (uint64_t) it * g.nent;
    st->edges_examined = (uint64_t) it * g.nent;
    st->algo_bytes = (uint64_t) ((4.0 * g.nent + 20.0 * N) * it);
  }
  if (rank_out)
  {
    double* out = (double*) ps->xf[0];  // the messages are no longer needed
    k_rank_by_id<float><<<grid_for(N, 256), 256, 0, s>>>(N, g.nrows(), L.qpos, g.id_of_pos, ps->rankf, out);
    LA3G_LAUNCHED();
    LA3G_CUDA(cudaMemcpyAsync(rank_out, out, (size_t) N * 8, cudaMemcpyDeviceToHost, s));
  }
  LA3G_TRY(T.finish());
  if (residual_out) *residual_out = res;
  return LA3G_OK;
}

extern "C" int la3g_pr_f32(la3g_graph* G, uint32_t iters, double tol, double* rank_out, double* residual_out,
                           la3g_stats* st)
{
  return pr_f32_run(G, iters, tol, rank_out, residual_out, st, false);
}

extern "C" int la3g_pr_f32_tiled(la3g_graph* G, uint32_t iters, double tol, double* rank_out, double* residual_out,
                                 la3g_stats* st)
{
  return pr_f32_run(G, iters, tol, rank_out, residual_out, st, true);
}
