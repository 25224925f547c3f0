// Batched inversion over a pool of many surfaces of uneven degree, net size and query count,
// in one persistent launch.
//
// The batch is cut on the host into tiles (surface, query range), listed surface by surface; a
// group of consecutive tiles of one surface is one run of queries.  Large tiles go to CTAs: the
// surface is staged once for four warps, which take equal portions of the run from a cursor in
// shared memory.  Tiles of at most 32 queries (latency) go to warps, each staging the surface in its
// own shared-memory area; warps never wait for one another, so a batch of a few thousand queries
// spreads over all SMs.  Either way the queries stream through the warp's slots as in the
// single-surface kernel (invert_core.cuh).  Degree dispatch: (p,q) in {2,3,5}^2 run
// degree-specialised code, other degrees a run-time-degree path.  Tile size and CTAs per SM
// are chosen by the pool's autotuner.
#include "invert_core.cuh"

namespace gnurbs {
namespace {

using namespace inv;

// Each degree variant is its own (not inlined) function, so that it keeps its own register
// allocation instead of the kernel taking the union of all variants' live ranges.
constexpr int kPoolSpans = 64;  // breakpoint tables staged per warp up to this many spans

// The queries [q, qend), handed to one warp.
struct WarpRange {
  int64_t q, qend;
  __device__ __forceinline__ int grab(int want, int64_t& q0) {
    q0 = q;
    const int64_t left = qend - q;
    const int k = left < want ? (int)left : want;
    q += k;
    return k;
  }
};

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

template <int MODE>
__global__ void __launch_bounds__(kThreads, 4) k_invert_pool(const SurfDev* __restrict__ table,
                                                          const InvTile* __restrict__ tiles, int ntiles,
                                                          int* __restrict__ counter, const double* __restrict__ P,
                                                          double* __restrict__ uv, int* __restrict__ st,
                                                          double* __restrict__ res, int group) {
  __shared__ Staged<kPoolSpans, MODE> sm[kWarps];
  __shared__ WarpWork<MODE> ww[kWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int cur = -1;
  for (;;) {
    // a group of consecutive chunks (mostly of one surface: chunks are listed surface by
    // surface) per grab, so a warp restages rarely
    int t0 = 0;
    if (lane == 0) t0 = atomicAdd(counter, group);
    t0 = __shfl_sync(0xffffffffu, t0, 0);
    if (t0 >= ntiles) break;
    const int t1 = min(t0 + group, ntiles);
    for (int t = t0; t < t1;) {
      int surf;
      int64_t begin, end;
      t = tile_run(tiles, t, t1, surf, begin, end);
      if (surf != cur) {
        __syncwarp();
        const SurfDev s = table[surf];
        stage_surface<kPoolSpans>(s, sm[warp], lane, 32);
        cur = surf;
        __syncwarp();
      }
      dispatch_stream<MODE>(sm[warp], ww[warp], P, WarpRange{begin, end}, uv, st, res);
      __syncwarp();
    }
  }
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

// CTA-granular schedule for large batches: a CTA takes a group of consecutive tiles, stages the
// surface of each run of tiles once for its four warps, and the warps share the run's queries.
constexpr int kCtaSpans = 256;

// Register budget: 4 CTAs per SM (6 / 5 / 4: 6.95 / 6.32 / 6.01 ms on 160 uneven faces in tiles of 128;
// every tile ends with its warps waiting for the last one, so latency counts).
template <int MODE>
__global__ void __launch_bounds__(kThreads, 4)
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

cudaError_t launch_invert_pool(const SurfDev* table, const InvTile* tiles, int ntiles, int* counter, const double* P,
                               double* uv, int* status, double* residual, int precision, int ctas, int tile_queries,
                               cudaStream_t st) {
  if (ntiles <= 0) return cudaSuccess;
  cudaError_t e = cudaMemsetAsync(counter, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  if (tile_queries > 32) {  // CTA tiles
    if (ctas > ntiles) ctas = ntiles;
    int group = ntiles / (ctas * 8);
    group = group < 1 ? 1 : (group > 8 ? 8 : group);
    if (precision == 1)
      k_invert_pool_cta<kModeMixed><<<ctas, kThreads, 0, st>>>(table, tiles, ntiles, counter, P, uv, status, residual,
                                                                group);
    else
      k_invert_pool_cta<kModeFP64><<<ctas, kThreads, 0, st>>>(table, tiles, ntiles, counter, P, uv, status, residual,
                                                               group);
    return cudaGetLastError();
  }
  const int warps_needed = ntiles;
  if (ctas * kWarps > warps_needed) ctas = (warps_needed + kWarps - 1) / kWarps;
  // chunks per grab: large batches take up to 8 at a time, while every warp still gets about
  // eight grabs so the tail stays short
  int group = ntiles / (ctas * kWarps * 8);
  group = group < 1 ? 1 : (group > 8 ? 8 : group);
  if (precision == 1)
    k_invert_pool<kModeMixed><<<ctas, kThreads, 0, st>>>(table, tiles, ntiles, counter, P, uv, status, residual,
                                                          group);
  else
    k_invert_pool<kModeFP64><<<ctas, kThreads, 0, st>>>(table, tiles, ntiles, counter, P, uv, status, residual,
                                                         group);
  return cudaGetLastError();
}

}  // namespace gnurbs
