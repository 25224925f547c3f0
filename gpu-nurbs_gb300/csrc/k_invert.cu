// Stage d: candidate culling + Gauss-Newton point inversion (K4 invert), one fused kernel.
//
// Replaces NewInverse + GaussNewton (src/kernel/kernel.cu:433-469, 151-249).  Per query:
//   1. cull: the built tree nodes sit in shared memory as FP32 boxes rounded outward (a point
//      outside is outside the exact box) and inward (a point strictly inside is inside it); only
//      coordinates within an FP32 ulp of a face are decided by the exact FP64 box, so the
//      candidate set equals the reference's NewBoundingBoxCheck scan bit for bit;
//   2. each candidate is seeded at its node's uv-centre (kernel.cu:154) and iterated with the
//      reference's Gauss-Newton update  C <- C - (J^T J)^-1 J^T (S(C) - P)  (kernel.cu:195-243)
//      until the step is small, then with Newton steps (Hessian J^T J + sum r_k d2S_k) whose
//      fixed point is the same stationary point but which converge quadratically;
//   3. results inside the knot domain are kept; the closest wins.
//
// Work distribution.  A query has anywhere from 0 to 65 candidate seeds and a seed needs from 2 to 24
// iterations, so one thread per query leaves most lanes of a warp idle.  The grid is persistent (as
// many CTAs as fit, fewer for small launches); each warp holds up to 32 queries in slots, flattens
// their (query, seed) pairs into a task list, and its lanes pull the next tasks as their seeds
// converge or fail, in batches of a few free lanes (the start and the merge of results are divergent
// work, cheaper done once for several lanes than every iteration for the two or three that just
// finished).  When the list runs out, the finished queries leave and new ones from a global counter
// take their slots while the last seeds of the others still run, so a warp's lanes idle only at the
// end of the launch.  A warp takes its share of what is left of the launch, and at least queries for
// a few seeds per lane (invert_core.cuh: least_grab).
//
// Against chunks of 32 queries run to their end one after the other (with the lookup grid of the
// staged breakpoints and the merges in batches; us, before and after):
//   64x64 surface, mixed   1,500 queries  671 -> 147;   20,000  812 -> 480;   2^20  9051 -> 8230
//   8x8 surface, mixed     1,500 queries  107 ->  73;   60,000  133 -> 122;   2^20  1365 -> 1250
//   64x64 surface, FP64    2,000 queries 3245 -> 820;   50,021  7390 -> 6670
//   quintic 256x256        20,000 queries 1212 -> 872;  300,007 6370 -> 5630
//
// Every seed runs to its own end (convergence, failure, the iteration cap, or an FP32 iterate two
// domain extents outside the domain), decided by the seed alone, so a query's result does not depend
// on which other queries share its warp: results are the same alone and in any batch.
//
// Precision schedules (template MODE):
//   FP64  — every evaluation, solve and update in FP64.  Bound by the FP64 pipe, which a warp's
//           instruction occupies for 64 clocks whatever its active lanes: so a seed's end takes its
//           residual from its last step instead of another evaluation, seeds start in batches,
//           reciprocals are three FP64 operations and comparisons run on the integer pipe (64x64
//           surface, 50,021 queries: 10.1 -> 7.4 ms; 4.9 -> 6.8 M queries/s).
//   MIXED — the seed exploration in FP32 (FP32 span matrices, FP32 breakpoints); the best
//           minimum (plus a distinct runner-up within 5 % of its distance, and the closest
//           minimum just outside the domain when as close) then takes the final Newton steps in
//           FP64: S, Su, Sv and the gradient J^T r in FP64, for the first three steps the
//           Hessian's curvature term from FP32 second derivatives (it only sets the convergence
//           rate; two steps normally reach the tolerance), the 2x2 solve and the residual
//           |S - P| at the returned point in FP64 (from the last step's S, Su, Sv and the step, a
//           first-order update whose error is far below FP64 rounding).  Later steps (at most 24
//           in all) take the curvature in FP64 too, for nearly degenerate minima.
#include "invert_core.cuh"

namespace gnurbs {
namespace {

using namespace inv;

// Register budget.  Mixed: 6 CTAs per SM (80 registers, some spills) hide the exploration's latencies
// best when every warp refills its slots several times; a launch of at most one slot set per warp of
// 4 CTAs per SM is bound by the latency of its seeds, and spills lengthen that (64x64 surface, 6 / 4
// CTAs: 6,000 queries 230 / 204 us, 60,000 835 / 789 us, 2^18 2457 / 2505 us, 2^20 8.26 / 8.63 ms).
// Degree 5 and the run-time-degree variant keep 128 registers (4 CTAs per SM): their larger Horner
// state spills heavily at 80.
template <int P, int Q, int MODE, int CTAS>
__global__ void __launch_bounds__(kThreads, CTAS)
    k_invert(SurfDev s, const double* __restrict__ Pq, int64_t n, double* __restrict__ uv_out,
             int* __restrict__ st_out, double* __restrict__ res_out, unsigned long long* __restrict__ counter,
             StreamGrid grid) {
  __shared__ Staged<kSmemSpans, MODE> sm;           // one surface for the whole CTA
  __shared__ WarpWork<MODE> ww[kWarps];
  stage_surface<kSmemSpans>(s, sm, threadIdx.x, blockDim.x);
  __syncthreads();
  QueryCounter src{counter, n, 0, grid.share, grid.least};
  invert_stream<P, Q, MODE, kSmemSpans, false>(sm, ww[threadIdx.x >> 5], Pq, src, uv_out, st_out, res_out);
}

// The work-counting variant: the same per-query computation, FP32/FP64 seed iterations and final
// FP64 polishes added to counts[0..1].  Diagnostic only.
template <int P, int Q, int MODE>
__global__ void __launch_bounds__(kThreads, 4)
    k_invert_count(SurfDev s, const double* __restrict__ Pq, int64_t n, double* __restrict__ uv_out,
                   int* __restrict__ st_out, double* __restrict__ res_out, unsigned long long* __restrict__ counter,
                   StreamGrid grid, unsigned long long* __restrict__ counts) {
  __shared__ Staged<kSmemSpans, MODE> sm;
  __shared__ WarpWork<MODE> ww[kWarps];
  stage_surface<kSmemSpans>(s, sm, threadIdx.x, blockDim.x);
  __syncthreads();
  QueryCounter src{counter, n, 0, grid.share, grid.least};
  invert_stream<P, Q, MODE, kSmemSpans, true>(sm, ww[threadIdx.x >> 5], Pq, src, uv_out, st_out, res_out, counts);
}

template <int P, int Q, int MODE>
cudaError_t launch_count_mode(const SurfDev& s, const double* P_, int64_t n, double* uv, int* st_, double* res,
                              unsigned long long* counter, unsigned long long* counts, cudaStream_t st) {
  if ((n + 31) / 32 > 0x3fffffffLL) return cudaErrorInvalidValue;
  int sms = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const StreamGrid g = stream_grid<MODE>(s, n, (int64_t)(sms > 0 ? sms : 1) * 4);
  k_invert_count<P, Q, MODE><<<g.blocks, kThreads, 0, st>>>(s, P_, n, uv, st_, res, counter, g, counts);
  return cudaGetLastError();
}

template <int P, int Q>
cudaError_t launch_count_pq(const SurfDev& s, const double* P_, int64_t n, double* uv, int* st_, double* res,
                            int prec, unsigned long long* counter, unsigned long long* counts, cudaStream_t st) {
  if (prec == 1) return launch_count_mode<P, Q, kModeMixed>(s, P_, n, uv, st_, res, counter, counts, st);
  return launch_count_mode<P, Q, kModeFP64>(s, P_, n, uv, st_, res, counter, counts, st);
}

// CTAs of a kernel that fit on the current GPU at once (queried once per kernel and device).
template <int P, int Q, int MODE, int CTAS>
int64_t resident_ctas() {
  static int cached[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (!cached[dev]) {
    int sms = 0, per_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_invert<P, Q, MODE, CTAS>, kThreads, 0);
    cached[dev] = (sms > 0 ? sms : 1) * (per_sm > 0 ? per_sm : 1);
  }
  return cached[dev];
}

template <int P, int Q, int MODE, int CTAS>
cudaError_t launch_budget(const SurfDev& s, const double* P_, int64_t n, double* uv, int* st_, double* res,
                          unsigned long long* counter, cudaStream_t st) {
  const StreamGrid g = stream_grid<MODE>(s, n, resident_ctas<P, Q, MODE, CTAS>());
  k_invert<P, Q, MODE, CTAS><<<g.blocks, kThreads, 0, st>>>(s, P_, n, uv, st_, res, counter, g);
  return cudaGetLastError();
}

template <int P, int Q, int MODE>
cudaError_t launch_mode(const SurfDev& s, const double* P_, int64_t n, double* uv, int* st_, double* res,
                        unsigned long long* counter, cudaStream_t st) {
  if ((n + 31) / 32 > 0x3fffffffLL) return cudaErrorInvalidValue;
  if constexpr (MODE == kModeMixed && (P == 2 || P == 3)) {
    if (n > (int64_t)32 * 4 * kWarps * kSchedulers / 4)
      return launch_budget<P, Q, MODE, 6>(s, P_, n, uv, st_, res, counter, st);
  }
  return launch_budget<P, Q, MODE, 4>(s, P_, n, uv, st_, res, counter, st);
}

template <int P, int Q>
cudaError_t launch_pq(const SurfDev& s, const double* P_, int64_t n, double* uv, int* st_, double* res, int prec,
                      unsigned long long* counter, cudaStream_t st) {
  if (prec == 1) return launch_mode<P, Q, kModeMixed>(s, P_, n, uv, st_, res, counter, st);
  return launch_mode<P, Q, kModeFP64>(s, P_, n, uv, st_, res, counter, st);
}

// S, Su, Sv at the uv-centre of every built node, FP32 and FP64: the first iteration of every
// seed starts there, and its evaluation does not depend on the query.  Computed with the same
// device functions and arguments as the seed iterations, so the values are the same bits.  Then the
// average number of candidate nodes of these points, by which the inversion sizes its work
// (cd32[9 * kTreeNodes]).  96 threads.
template <int P, int Q>
__device__ __forceinline__ void centre_of(const SurfDev& s, int k, int& hits) {
  const TreeNodeDev& T = s.tree[k];
  const double cu = (T.uv_lb[0] + T.uv_rt[0]) / 2, cv = (T.uv_lb[1] + T.uv_rt[1]) / 2;  // kernel.cu:154
  const fast::Locator<float> L32 = fast::global_locator<float>(s);
  const fast::Locator<double> L64 = fast::global_locator<double>(s);
  int hu = 0, hv = 0;
  fast::SDer<float> d = fast::eval_at<float, P, Q, 2, true>(L32, s.m32, s.p, s.q, (float)cu, (float)cv, hu, hv);
  hu = hv = 0;
  fast::SDer<double> e = fast::eval_at<double, P, Q, 2>(L64, s.m64, s.p, s.q, cu, cv, hu, hv);
  const float f[9] = {d.S.x, d.S.y, d.S.z, d.Su.x, d.Su.y, d.Su.z, d.Sv.x, d.Sv.y, d.Sv.z};
  const double g[9] = {e.S.x, e.S.y, e.S.z, e.Su.x, e.Su.y, e.Su.z, e.Sv.x, e.Sv.y, e.Sv.z};
  for (int c = 0; c < 9; ++c) {
    s.cd32[9 * k + c] = f[c];
    s.cd64[9 * k + c] = g[c];
  }
  const long long x = fast::order_key(g[0]), y = fast::order_key(g[1]), z = fast::order_key(g[2]);
  for (int j = 0; j < kTreeNodes; ++j) {
    const TreeNodeDev& B = s.tree[j];
    if (s.built[j] && x >= fast::order_key(B.lb[0]) && x <= fast::order_key(B.rt[0]) &&
        y >= fast::order_key(B.lb[1]) && y <= fast::order_key(B.rt[1]) && z >= fast::order_key(B.lb[2]) &&
        z <= fast::order_key(B.rt[2]))
      ++hits;
  }
}
template <int P, int Q>
__device__ void centre_ders(const SurfDev& s, int k) {
  __shared__ int s_hits, s_built;
  if (k == 0) s_hits = s_built = 0;
  __syncthreads();
  if (k < kTreeNodes && s.built[k]) {
    int hits = 0;
    centre_of<P, Q>(s, k, hits);
    atomicAdd(&s_hits, hits);
    atomicAdd(&s_built, 1);
  }
  __syncthreads();
  if (k == 0) s.cd32[9 * kTreeNodes] = (float)s_hits / (float)(s_built > 0 ? s_built : 1);
}

template <int P, int Q>
__global__ void k_centre_ders(SurfDev s) {
  centre_ders<P, Q>(s, threadIdx.x);
}

__global__ void k_centre_ders_batched(const SurfDev* __restrict__ table, const int* __restrict__ ids) {
  const SurfDev s = table[ids[blockIdx.x]];
  if (s.p == 3 && s.q == 3) centre_ders<3, 3>(s, threadIdx.x);
  else if (s.p == 5 && s.q == 5) centre_ders<5, 5>(s, threadIdx.x);
  else if (s.p == 2 && s.q == 2) centre_ders<2, 2>(s, threadIdx.x);
  else centre_ders<0, 0>(s, threadIdx.x);
}

}  // namespace

cudaError_t launch_centre_ders(const SurfDev& s, cudaStream_t st) {
  if (s.p == 3 && s.q == 3) k_centre_ders<3, 3><<<1, 96, 0, st>>>(s);
  else if (s.p == 5 && s.q == 5) k_centre_ders<5, 5><<<1, 96, 0, st>>>(s);
  else if (s.p == 2 && s.q == 2) k_centre_ders<2, 2><<<1, 96, 0, st>>>(s);
  else k_centre_ders<0, 0><<<1, 96, 0, st>>>(s);
  return cudaGetLastError();
}

cudaError_t launch_centre_ders_batched(const SurfDev* table, const int* ids, int count, cudaStream_t st) {
  for (int off = 0; off < count; off += 65535) {
    const int c = count - off < 65535 ? count - off : 65535;
    k_centre_ders_batched<<<c, 96, 0, st>>>(table, ids + off);
  }
  return cudaGetLastError();
}

cudaError_t launch_invert_count(const SurfDev& s, const double* P, int64_t n, double* uv, int* status,
                                double* residual, int precision, unsigned long long* counter, unsigned long long* counts,
                                cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if (s.p == 3 && s.q == 3) return launch_count_pq<3, 3>(s, P, n, uv, status, residual, precision, counter, counts, st);
  if (s.p == 5 && s.q == 5) return launch_count_pq<5, 5>(s, P, n, uv, status, residual, precision, counter, counts, st);
  return launch_count_pq<0, 0>(s, P, n, uv, status, residual, precision, counter, counts, st);
}

cudaError_t launch_invert(const SurfDev& s, const double* P, int64_t n, double* uv, int* status, double* residual,
                          int precision, unsigned long long* counter, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if (s.p == 3 && s.q == 3) return launch_pq<3, 3>(s, P, n, uv, status, residual, precision, counter, st);
  if (s.p == 5 && s.q == 5) return launch_pq<5, 5>(s, P, n, uv, status, residual, precision, counter, st);
  if (s.p == 2 && s.q == 2) return launch_pq<2, 2>(s, P, n, uv, status, residual, precision, counter, st);
  return launch_pq<0, 0>(s, P, n, uv, status, residual, precision, counter, st);
}

}  // namespace gnurbs
