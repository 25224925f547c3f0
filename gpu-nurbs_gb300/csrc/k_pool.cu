// Batched inversion over a pool of many surfaces of uneven degree, net size and query count,
// in one persistent launch.
//
// The batch is cut on the host into tiles (surface, query range), listed surface by surface.  A CTA
// takes a tile, or a few consecutive small ones, from a counter; consecutive tiles of one surface are
// one run of queries.  The surface of a run is staged once for the CTA's four warps, which take equal
// portions of the run from a cursor in shared memory and stream them through their slots as in the
// single-surface kernel (invert_core.cuh).  Degree dispatch: (p,q) in {2,3,5}^2 run degree-specialised
// code, other degrees a run-time-degree path.  Tile size and CTAs per SM are chosen by the pool's
// autotuner.
#include <algorithm>

#include "invert_core.cuh"

namespace gnurbs {
namespace {

using namespace inv;

// The queries from `begin` to `qend`, handed out to the CTA's warps by a cursor in shared memory,
// `portion` at a time.
struct CtaRange {
  unsigned long long* cursor;  // queries handed out
  int64_t begin, qend;
  int portion;
  __device__ __forceinline__ int grab(int want, int64_t& q0) {
    const int k = min(portion, want);
    unsigned long long a = 0;
    if ((threadIdx.x & 31) == 0) a = atomicAdd(cursor, (unsigned long long)k);
    q0 = begin + (int64_t)__shfl_sync(0xffffffffu, a, 0);
    const int64_t left = qend - q0;
    return left < k ? (left > 0 ? (int)left : 0) : k;
  }
};

// Each degree variant is its own (not inlined) function, so that it keeps its own register
// allocation instead of the kernel taking the union of all variants' live ranges.
template <int P, int Q, int MODE, int KS, class Source>
__device__ __noinline__ void stream_variant(Staged<KS, MODE>& sm, WarpWork<MODE>& ww,
                                            const double* __restrict__ P_, Source& src, double* __restrict__ uv,
                                            int* __restrict__ st, double* __restrict__ res) {
  invert_stream<P, Q, MODE, KS, false>(sm, ww, P_, src, uv, st, res);
}

template <int MODE, int KS, class Source>
__device__ __forceinline__ void dispatch_stream(Staged<KS, MODE>& sm, WarpWork<MODE>& ww,
                                                const double* __restrict__ P, Source src, double* __restrict__ uv,
                                                int* __restrict__ st, double* __restrict__ res) {
#define GN_CASE(A, B)                                                   \
  if (sm.ctx.p == A && sm.ctx.q == B) {                                         \
    stream_variant<A, B, MODE, KS>(sm, ww, P, src, uv, st, res);    \
    return;                                                             \
  }
  GN_CASE(3, 3)
  GN_CASE(2, 2)
  GN_CASE(5, 5)
  GN_CASE(2, 3)
  GN_CASE(3, 2)
  GN_CASE(2, 5)
  GN_CASE(5, 2)
  GN_CASE(3, 5)
  GN_CASE(5, 3)
#undef GN_CASE
  stream_variant<0, 0, MODE, KS>(sm, ww, P, src, uv, st, res);
}

// The consecutive tiles [t, return value) that continue tile t: the same surface, adjoining
// queries.  begin, end: their queries.
__device__ __forceinline__ int tile_run(const InvTile* __restrict__ tiles, int t, int t1, int& surf, int64_t& begin,
                                        int64_t& end) {
  const InvTile T = tiles[t];
  surf = T.surf;
  begin = T.begin;
  end = T.begin + T.count;
  for (++t; t < t1 && tiles[t].surf == surf && tiles[t].begin == end; ++t) end += tiles[t].count;
  return t;
}

// Batched FP64 evaluation over tiles: one CTA per tile, one thread per (u,v), run-time degrees.
template <int ORDER>
__global__ void __launch_bounds__(128) k_eval_pool(const SurfDev* __restrict__ table, const InvTile* __restrict__ tiles,
                                                   const double* __restrict__ uv, int64_t n, unsigned mask,
                                                   double* __restrict__ out) {
  const InvTile T = tiles[blockIdx.x];
  const SurfDev s = table[T.surf];
  const fast::Locator<double> L = fast::global_locator<double>(s);
  for (int k = threadIdx.x; k < T.count; k += blockDim.x) {
    const int64_t i = T.begin + k;
    int hu = 0, hv = 0;
    fast::SDer<double> d = fast::eval_at<double, 0, 0, ORDER>(L, s.m64, s.p, s.q, uv[2 * i], uv[2 * i + 1], hu, hv);
    int o = 0;
    auto put = [&](const v3<double>& a) {
      out[(int64_t)(3 * o + 0) * n + i] = a.x;
      out[(int64_t)(3 * o + 1) * n + i] = a.y;
      out[(int64_t)(3 * o + 2) * n + i] = a.z;
      ++o;
    };
    if (mask & 1u) put(d.S);
    if (ORDER >= 1) {
      if (mask & 2u) put(d.Su);
      if (mask & 4u) put(d.Sv);
    }
    if (ORDER >= 2) {
      if (mask & 8u) put(d.Suu);
      if (mask & 16u) put(d.Suv);
      if (mask & 32u) put(d.Svv);
    }
  }
}

constexpr int kCtaSpans = 256;      // breakpoint tables staged up to this many spans
// Small tiles are taken together up to this many queries.  32 / 64 / 128 / 256, tiles of 16, mixed: 63,000
// queries of 130 surfaces 1,901 / 1,786 / 1,488 / 1,394 us, 200,000 of 200 4,054 / 3,888 / 4,074 / 4,536; FP64,
// 63,000 of 130 10,976 / 12,004 / 14,066 / 13,887.
constexpr int kGroupQueries = 128;
constexpr int kCtasPerSm = 4;

// Register budget: 4 CTAs per SM (6 / 5 / 4: 6.95 / 6.32 / 6.01 ms on 160 uneven faces in tiles of 128;
// every tile ends with its warps waiting for the last one, so latency counts).  Small tiles (32 queries
// at most, for latency) are CTA work too: with a warp per tile, a batch's warps ran up to nine degree
// variants side by side, each with a staged surface and a drain of its own.  Mixed, tiles of 16:
// 1,000 queries of 3 surfaces 538 -> 221 us, 14,000 of 25 565 -> 450, 63,000 of 130 2348 -> 1317.
template <int MODE>
__global__ void __launch_bounds__(kThreads, kCtasPerSm)
    k_invert_pool_cta(const SurfDev* __restrict__ table, const InvTile* __restrict__ tiles, int ntiles,
                      int* __restrict__ counter, const double* __restrict__ P, double* __restrict__ uv,
                      int* __restrict__ st, double* __restrict__ res, int group) {
  __shared__ Staged<kCtaSpans, MODE> sm;
  __shared__ WarpWork<MODE> ww[kWarps];
  __shared__ int s_tile;
  __shared__ unsigned long long s_cursor;
  int cur = -1;
  const int warp = threadIdx.x >> 5;
  for (;;) {
    if (threadIdx.x == 0) s_tile = atomicAdd(counter, group);
    __syncthreads();
    const int t0 = s_tile;
    if (t0 >= ntiles) break;
    const int t1 = min(t0 + group, ntiles);
    for (int t = t0; t < t1;) {
      int surf;
      int64_t begin, end;
      t = tile_run(tiles, t, t1, surf, begin, end);
      if (threadIdx.x == 0) s_cursor = 0;
      if (surf != cur) {
        const SurfDev s = table[surf];
        stage_surface<kCtaSpans>(s, sm, threadIdx.x, blockDim.x);
        cur = surf;
      }
      __syncthreads();
      const int64_t part = (end - begin + kWarps - 1) / kWarps;
      const int portion = (int)(part < 32 ? part : 32);  // an equal part for each warp
      dispatch_stream<MODE>(sm, ww[warp], P, CtaRange{&s_cursor, begin, end, portion}, uv, st, res);
      __syncthreads();
    }
  }
}

}  // namespace

cudaError_t launch_eval_pool(const SurfDev* table, const InvTile* tiles, int ntiles, const double* uv, int64_t n,
                             unsigned mask, double* out, cudaStream_t st) {
  if (ntiles <= 0) return cudaSuccess;
  int order = (mask & 56u) ? 2 : ((mask & 6u) ? 1 : 0);
  if (order == 0) k_eval_pool<0><<<ntiles, 128, 0, st>>>(table, tiles, uv, n, mask, out);
  else if (order == 1) k_eval_pool<1><<<ntiles, 128, 0, st>>>(table, tiles, uv, n, mask, out);
  else k_eval_pool<2><<<ntiles, 128, 0, st>>>(table, tiles, uv, n, mask, out);
  return cudaGetLastError();
}

int pool_ctas_per_sm(int precision) {
  static int cached[2][64] = {};
  const int mode = precision == 1 ? 1 : 0;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  int& c = cached[mode][dev];
  if (!c) {
    int fit = 0;
    if (mode) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k_invert_pool_cta<kModeMixed>, kThreads, 0);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k_invert_pool_cta<kModeFP64>, kThreads, 0);
    c = fit > 0 ? fit : 1;
  }
  return c;
}

cudaError_t launch_invert_pool(const SurfDev* table, const InvTile* tiles, int ntiles, int* counter, const double* P,
                               double* uv, int* status, double* residual, int precision, int ctas, int tile_queries,
                               cudaStream_t st) {
  if (ntiles <= 0) return cudaSuccess;
  cudaError_t e = cudaMemsetAsync(counter, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  if (ctas > ntiles) ctas = ntiles;
  // Tiles per grab: small tiles together, up to kGroupQueries queries, while every resident CTA gets a
  // grab.  Larger tiles one by one: groups of 8 / 2 / 1 tiles of 128 take 41.3 / 35.8 / 32.8 ms on 600
  // surfaces with 4.4 M queries (the last groups are the launch's tail), and the same on 300 with 1 M.
  const int resident = std::min(ctas, kCtasPerSm * 152);
  const int group = std::max(1, std::min(ntiles / resident, kGroupQueries / tile_queries));
  if (precision == 1)
    k_invert_pool_cta<kModeMixed><<<ctas, kThreads, 0, st>>>(table, tiles, ntiles, counter, P, uv, status, residual,
                                                             group);
  else
    k_invert_pool_cta<kModeFP64><<<ctas, kThreads, 0, st>>>(table, tiles, ntiles, counter, P, uv, status, residual,
                                                            group);
  return cudaGetLastError();
}

}  // namespace gnurbs
