// Device core of the point inversion (stage d), shared by the single-surface kernel
// (k_invert.cu) and the pooled persistent kernel (k_pool.cu): per-seed FP32/FP64 iterations,
// the per-warp task scheduler over (query, seed) pairs and the final FP64 steps.  The
// algorithm and its precision schedules are described in k_invert.cu.
#pragma once
#include <type_traits>

#include "nurbs_internal.h"
#include "nurbs_math.cuh"

namespace gnurbs {
namespace inv {

constexpr int kModeFP64 = 0;
constexpr int kModeMixed = 1;

constexpr int kWarps = 4;          // warps per CTA
constexpr int kThreads = 32 * kWarps;
constexpr int kMaxIter32 = 40;     // FP32 iterations per seed (the FP64 cap: the oracle's too)
constexpr int kMaxIter64 = 40;     // FP64-mode iterations per seed
constexpr int kMaxFinal64 = 24;    // MIXED: FP64 steps (2 normally)
constexpr int kFinal32Curv = 3;    // MIXED: FP64 steps with the FP32 curvature term before the FP64 one
constexpr float kPolishMargin = 0.05f;  // MIXED: a runner-up this close to the best also takes the FP64 steps
constexpr double kNewtonSwitch = 1e-2;  // GN while the step is larger, Newton below
constexpr float kTol32 = 3e-7f;
constexpr double kTolNewton64 = 1e-10;  // a Newton step this small leaves < 1e-19 error
constexpr double kTolAny64 = 1e-14;
constexpr double kDistinct = 1e-7;      // FP64 minima: grid cell size, times the domain's extent
constexpr float kDistinct32 = 1e-4f;    // FP32 minima: the same
// Every seed runs to its own end, decided by the seed alone.  Stopping a seed once it nears a
// minimum its query already found saves ~15-20 % of the iterations, but whether that other seed
// has finished first depends on the other queries sharing the warp, so results would depend on
// the batch.
constexpr int kSols = 4;                // FP64 mode: distinct minima kept per query
constexpr int kSmemSpans = 256;         // breakpoint tables staged in shared memory up to this
// MIXED: lanes whose seed has ended wait until this many are free (or no lane still iterates)
// and then merge their results and start their next seeds together, so that the divergent start (task decode, the first
// step from the node centre) runs once for several lanes instead of every iteration for ~3.
// Which lane runs which seed, and when, does not change any seed's arithmetic, and the
// records are independent of arrival order, so results are the same for every value.
constexpr int kStartBatch = 8;
// The FP64 schedule's (50,021 queries of the 64x64 surface: 1 / 3 / 6 / 10 take 7.52 / 7.38 / 7.47 /
// 7.73 ms).
constexpr int kStartBatch64 = 3;
// Slots free or finished before the task list is refilled while seeds still run.  A refill of the
// mixed schedule passes its finished queries through the final FP64 steps, as long for one lane as
// for all: 24 / 28 / 29 slots take 1.52 / 1.39 / 1.42 ms on the 8x8 surface (2^20 queries), the same on
// the 64x64 one.  The FP64 schedule has no such pass.
constexpr int kRefillMixed = 28;
constexpr int kRefill64 = 8;
// Seeds a warp's least portion holds (least_grab).  Mixed, 32 / 64: 64x64 surface, 6,000 queries 230 /
// 210 us; 8x8 surface, 60,000 queries 145 / 126 us; FP64 64 / 128: 50,021 queries 6.73 / 6.67 ms.
constexpr float kGrabSeedsMixed = 64, kGrabSeeds64 = 128;

// Arithmetic below writes every product that feeds a sum as an explicit FMA (the translation
// units are compiled with --fmad=false), so a seed's trajectory is the same bit for bit in
// every kernel that runs it: results do not depend on the kernel, the batch or the schedule.
template <typename T>
__device__ __forceinline__ T dot3(const v3<T>& a, const v3<T>& b) {
  return fast::mad(a.z, b.z, fast::mad(a.y, b.y, a.x * b.x));
}
template <typename T, typename TH>
__device__ __forceinline__ T dot3c(const v3<T>& a, const v3<TH>& b) {  // b converted to T
  return fast::mad(a.z, (T)b.z, fast::mad(a.y, (T)b.y, a.x * (T)b.x));
}
template <typename T>
__device__ __forceinline__ T det2(T h00, T h01, T h11) {
  return fast::mad(h00, h11, -(h01 * h01));
}

// One (Gauss-)Newton step from the derivatives at C.  Newton uses H = J^T J + r.d2S when that
// H is positive definite, else the Gauss-Newton matrix J^T J (the reference's update,
// kernel.cu:195-243).  Returns kSingular when the system is singular, kStepGN or kStepNewton
// for the matrix it used.  FAST: FP32 reciprocal by the hardware approximation.
enum StepKind { kSingular = 0, kStepGN = 1, kStepNewton = 2 };
template <typename T, typename TH, bool FAST>
__device__ __forceinline__ int solve_step(const v3<T>& r, const v3<T>& Su, const v3<T>& Sv, const v3<TH>& Suu,
                                          const v3<TH>& Suv, const v3<TH>& Svv, bool newton, T& du, T& dv) {
  T h00 = dot3(Su, Su), h01 = dot3(Su, Sv), h11 = dot3(Sv, Sv);
  const T g0 = dot3(Su, r), g1 = dot3(Sv, r);
  int kind = kStepGN;
  if (newton) {
    const T n00 = h00 + dot3c(r, Suu), n01 = h01 + dot3c(r, Suv), n11 = h11 + dot3c(r, Svv);
    if (fast::is_positive(n00) && fast::is_positive(det2(n00, n01, n11))) {
      h00 = n00;
      h01 = n01;
      h11 = n11;
      kind = kStepNewton;
    }
  }
  const T det = det2(h00, h01, h11);
  if (!fast::is_positive(det)) return kSingular;
  const T inv = fast::rcp<FAST>(det);
  du = fast::mad(h11, g0, -(h01 * g1)) * inv;
  dv = fast::mad(h00, g1, -(h01 * g0)) * inv;
  return kind;
}

// Where one kernel finds the span tables: breakpoints in shared memory when they fit.
struct Ctx {
  fast::Locator<float> L32;
  fast::Locator<double> L64;
  const float* m32;
  const double* m64;
  int p, q;
  double dom_u0, dom_u1, dom_v0, dom_v1;
  double iru, irv;   // 1 / knot range
};

// |S - P|^2 at (u - du, v - dv) from r = S - P, Su, Sv at (u, v): S(u - du, v - dv) = S - Su du -
// Sv dv + O(|S''| 1e-20) for the steps a seed ends with (1e-10 at most), below the rounding of S
// itself.  Su and Sv are scaled by the knot range (kernel.cu:167): du and dv are the steps divided by
// it, or the range is 1.
__device__ __forceinline__ double dist2_after(const v3<double>& r, const v3<double>& Su, const v3<double>& Sv,
                                              double du, double dv) {
  const v3<double> r2 = {fast::mad(-Sv.x, dv, fast::mad(-Su.x, du, r.x)),
                         fast::mad(-Sv.y, dv, fast::mad(-Su.y, du, r.y)),
                         fast::mad(-Sv.z, dv, fast::mad(-Su.z, du, r.z))};
  return dot3(r2, r2);
}

// The FP32 evaluation of S..Svv that the explorations iterate with, from a context's tables
// (GlobalEval: breakpoints by bisection from the last span) or from a staged surface (StagedEval).
template <int P, int Q>
struct GlobalEval {
  const Ctx& c;
  __device__ __forceinline__ void spans(float u, float v, int& hu, int& hv) const {
    hu = fast::find_seg_hint(c.L32.bu, c.L32.ns_u, u, hu);
    hv = fast::find_seg_hint(c.L32.bv, c.L32.ns_v, v, hv);
  }
  template <int ORDER>
  __device__ __forceinline__ fast::SDer<float> at(float u, float v, int& hu, int& hv) const {
    return fast::eval_at<float, P, Q, ORDER, true>(c.L32, c.m32, c.p, c.q, u, v, hu, hv);
  }
};

// The same at an FP64 seed's end (u, v) on a knot range other than 1: evaluated, where the ends are taken
// up.  (Dividing the steps inside the iterations, in which some lane ends in nearly every turn, cost them
// up to 2 % on every range.)
template <int P, int Q>
__device__ __forceinline__ void evaluate_dist2(const Ctx& c, double px, double py, double pz, double u, double v, int hu,
                                               int hv, double& dist2) {
  const long long one = 0x3ff0000000000000ll;
  if (__double_as_longlong(c.iru) == one && __double_as_longlong(c.irv) == one) return;
  const fast::SDer<double> d = fast::eval_at<double, P, Q, 0>(c.L64, c.m64, c.p, c.q, u, v, hu, hv);
  const v3<double> r = {d.S.x - px, d.S.y - py, d.S.z - pz};
  dist2 = dot3(r, r);
}

// Per-seed iteration state (hu/hv: span hints for the warm-started span search).
template <typename T>
struct Seed {
  T u, v, prev;
  int it, hu, hv;
  bool newton;
};

enum StepResult { kContinue = 0, kConverged = 1, kFailed = 2 };

// One FP32 iteration of a seed.  Convergence: the step is at the FP32 resolution of the
// parameters (the change of S it makes, |Su du + Sv dv|, is within 8 ulp(|S|)), or Newton steps
// (with a positive definite Hessian) stop shrinking.  Where the Hessian is not
// positive definite the iterate is near a saddle of the distance, from which the GN steps creep
// away slowly: steps that do not shrink there are no sign of convergence.  dist2 = |S - P|^2
// before the step.
template <class Eval>
__device__ __forceinline__ int iterate32(const Eval& ev, float px, float py, float pz, Seed<float>& st, float& dist2) {
  fast::SDer<float> d = ev.template at<2>(st.u, st.v, st.hu, st.hv);
  v3<float> r = {d.S.x - px, d.S.y - py, d.S.z - pz};
  float du, dv;
  const int kind = solve_step<float, float, true>(r, d.Su, d.Sv, d.Suu, d.Suv, d.Svv, st.newton, du, dv);
  if (kind == kSingular) return kFailed;
  if (!(isfinite(du) && isfinite(dv))) return kFailed;
  st.u -= du;
  st.v -= dv;
  float step = fmaxf(fabsf(du), fabsf(dv));
  dist2 = dot3(r, r);
  float smag = fmaxf(fmaxf(fabsf(d.S.x), fabsf(d.S.y)), fmaxf(fabsf(d.S.z), 1.0f));
  const v3<float> dS = {fast::mad(d.Sv.x, dv, d.Su.x * du), fast::mad(d.Sv.y, dv, d.Su.y * du),
                        fast::mad(d.Sv.z, dv, d.Su.z * du)};
  float fl = 8.0f * 5.96e-8f * smag;
  if (step <= kTol32 || dot3(dS, dS) <= fl * fl) return kConverged;
  if (kind == kStepNewton && step < 1e-4f && step > 0.5f * st.prev) return kConverged;
  st.prev = step;
  st.newton = step < (float)kNewtonSwitch;
  if (++st.it >= kMaxIter32) return kFailed;
  return kContinue;
}

// One FP64 iteration of a seed (FP64 mode).  dist2, when the seed converges: |S - P|^2 at the new
// (u, v) from this step's S, Su, Sv (another evaluation for the few lanes whose seeds just ended would
// cost the warp as much as one for all lanes), for a knot range of 1 (evaluate_dist2).
template <int P, int Q>
__device__ __forceinline__ int iterate64(const Ctx& c, double px, double py, double pz, Seed<double>& st,
                                         double& dist2) {
  fast::SDer<double> d = fast::eval_at<double, P, Q, 2>(c.L64, c.m64, c.p, c.q, st.u, st.v, st.hu, st.hv);
  v3<double> r = {d.S.x - px, d.S.y - py, d.S.z - pz};
  double du, dv;
  if (!solve_step<double, double, false>(r, d.Su, d.Sv, d.Suu, d.Suv, d.Svv, st.newton, du, dv)) return kFailed;
  if (!(fast::is_finite(du) && fast::is_finite(dv))) return kFailed;
  st.u -= du;
  st.v -= dv;
  const double step = fast::max_abs(du, dv);
  if ((st.newton && fast::le_nonneg(step, kTolNewton64)) || fast::le_nonneg(step, kTolAny64)) {
    dist2 = dist2_after(r, d.Su, d.Sv, du, dv);
    return kConverged;
  }
  st.prev = step;
  st.newton = fast::lt_nonneg(step, kNewtonSwitch);
  if (++st.it >= kMaxIter64) return kFailed;
  return kContinue;
}

// An FP64 seed's end counts when it lies in the domain at a finite distance.
__device__ __forceinline__ bool in_domain64(const Ctx& c, double u, double v, double dist2) {
  const long long ku = fast::order_key(u), kv = fast::order_key(v);
  return ku >= fast::order_key(c.dom_u0) && ku <= fast::order_key(c.dom_u1) && kv >= fast::order_key(c.dom_v0) &&
         kv <= fast::order_key(c.dom_v1) && fast::is_finite(dist2);
}

// The first iteration of a seed from its node centre's precomputed S, Su, Sv (cd = 9 values,
// the same bits the evaluation there gives): the seed advances to its second iteration when the
// first one continues it, and is left at the centre otherwise, for iterate32/iterate64 to repeat
// that first iteration and end the seed.  The step is the GN update (the Newton phase starts
// after a step below kNewtonSwitch).
template <typename T>
__device__ __forceinline__ void first_step(const T* __restrict__ cd, T px, T py, T pz, const float far[4],
                                           Seed<T>& st) {
  const v3<T> S = {cd[0], cd[1], cd[2]}, Su = {cd[3], cd[4], cd[5]}, Sv = {cd[6], cd[7], cd[8]};
  const v3<T> r = {S.x - px, S.y - py, S.z - pz};
  T du, dv;
  if (solve_step<T, T, sizeof(T) == 4>(r, Su, Sv, Su, Su, Su, false, du, dv) == kSingular) return;
  const T u = st.u - du, v = st.v - dv;
  T step;
  if constexpr (sizeof(T) == 4) {
    if (!(isfinite(du) && isfinite(dv))) return;
    step = fmaxf(fabsf(du), fabsf(dv));
  } else {
    if (!(fast::is_finite(du) && fast::is_finite(dv))) return;
    step = fast::max_abs(du, dv);
  }
  if constexpr (sizeof(T) == 4) {
    const float smag = fmaxf(fmaxf(fabsf(S.x), fabsf(S.y)), fmaxf(fabsf(S.z), 1.0f));
    const v3<float> dS = {fast::mad(Sv.x, dv, Su.x * du), fast::mad(Sv.y, dv, Su.y * du),
                          fast::mad(Sv.z, dv, Su.z * du)};
    const float fl = 8.0f * 5.96e-8f * smag;
    if (step <= kTol32 || dot3(dS, dS) <= fl * fl) return;  // converged at once: left to iterate32
    if (!(u >= far[0] && u <= far[1] && v >= far[2] && v <= far[3])) return;
  } else {
    if (fast::le_nonneg(step, kTolAny64)) return;
  }
  st.u = u;
  st.v = v;
  st.prev = step;
  if constexpr (sizeof(T) == 4) st.newton = step < (T)kNewtonSwitch;
  else st.newton = fast::lt_nonneg(step, kNewtonSwitch);
  st.it = 1;
}

// MIXED: the final FP64 Newton steps from an FP32 minimum, then the residual.  The first
// kFinal32Curv steps take the Hessian's curvature term from FP32 second derivatives (it only
// sets the rate of convergence, and two steps normally reach the tolerance); later steps take
// it in FP64, which converges where the minimum is nearly degenerate (a flat valley, where the
// FP32 term's error is comparable to the Hessian's smallest eigenvalue).
struct Final {
  double u, v;
  int it, hu, hv, hu32, hv32;
};
template <class Eval>
__device__ __forceinline__ void final_start(const Eval& ev, double u, double v, Final& f) {
  f.u = u;
  f.v = v;
  f.it = 0;
  // span hints from the FP32 tables (shared memory when staged): the FP64 search then only
  // confirms them with two reads instead of bisecting the FP64 tables in global memory
  f.hu = f.hv = 0;
  ev.spans((float)u, (float)v, f.hu, f.hv);
  f.hu32 = f.hu;
  f.hv32 = f.hv;
}
// One step: kConverged (in the domain, res the residual), kFailed or kContinue.
template <int P, int Q, class Eval>
__device__ __forceinline__ int final_step(const Ctx& c, const Eval& ev, double px, double py, double pz, Final& f,
                                          double& res) {
  fast::SDer<double> d;
  double du, dv;
  int kind;
  v3<double> r;
  if (f.it < kFinal32Curv) {
    d = fast::eval_at<double, P, Q, 1>(c.L64, c.m64, c.p, c.q, f.u, f.v, f.hu, f.hv);
    fast::SDer<float> e = ev.template at<2>((float)f.u, (float)f.v, f.hu32, f.hv32);
    r = {d.S.x - px, d.S.y - py, d.S.z - pz};
    kind = solve_step<double, float, false>(r, d.Su, d.Sv, e.Suu, e.Suv, e.Svv, true, du, dv);
  } else {
    d = fast::eval_at<double, P, Q, 2>(c.L64, c.m64, c.p, c.q, f.u, f.v, f.hu, f.hv);
    r = {d.S.x - px, d.S.y - py, d.S.z - pz};
    kind = solve_step<double, double, false>(r, d.Su, d.Sv, d.Suu, d.Suv, d.Svv, true, du, dv);
  }
  if (kind == kSingular) return kFailed;
  if (!(fast::is_finite(du) && fast::is_finite(dv))) return kFailed;
  f.u -= du;
  f.v -= dv;
  if (fast::le_nonneg(fast::max_abs(du, dv), kTolNewton64)) {
    const double dist2 = dist2_after(r, d.Su, d.Sv, du * c.iru, dv * c.irv);
    res = sqrt(dist2);
    return in_domain64(c, f.u, f.v, dist2) ? kConverged : kFailed;
  }
  return ++f.it < kMaxFinal64 ? kContinue : kFailed;
}
template <int P, int Q, class Eval>
__device__ __forceinline__ bool final64(const Ctx& c, const Eval& ev, double px, double py, double pz, double& u,
                                        double& v, double& res) {
  Final f;
  final_start(ev, u, v, f);
  int r = kContinue;
  while (r == kContinue) r = final_step<P, Q>(c, ev, px, py, pz, f, res);
  u = f.u;
  v = f.v;
  return r == kConverged;
}

// Position of the k-th (0-based) set bit of m, which has more than k set bits: a fixed
// five-step bisection on bit counts of the lower half of each window.
__device__ __forceinline__ int select_bit(uint64_t m, int k) {
  const unsigned lo = (unsigned)m;
  const int clo = __popc(lo);
  unsigned w32 = k < clo ? lo : (unsigned)(m >> 32);
  int pos = k < clo ? 0 : 32;
  if (k >= clo) k -= clo;
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) {
    const int c = __popc(w32 & ((1u << w) - 1u));
    if (k >= c) {
      k -= c;
      w32 >>= w;
      pos += w;
    }
  }
  return pos;
}

struct Rec32 {  // per-query FP32 record: best and best distinct runner-up (squared distances)
  float u1, v1, d1, u2, v2, d2;
  int cu1, cv1;  // grid cell of the best
  float ue, ve, de;  // the closest FP32 minimum just outside the domain (edge record)
};

// Total order on results (distance, then u, then v): the minimum of a set does not depend on
// the order in which its members arrive, so per-query records are schedule independent.
template <typename T>
__device__ __forceinline__ bool before(T d, T u, T v, T d0, T u0, T v0) {
  const auto kd = fast::order_key(d), kd0 = fast::order_key(d0);
  if (kd != kd0) return kd < kd0;
  const auto ku = fast::order_key(u), ku0 = fast::order_key(u0);
  return ku < ku0 || (ku == ku0 && fast::order_key(v) < fast::order_key(v0));
}
struct Rec64 {  // per-query FP64 record: distinct minima (r: squared distances) and their grid cells
  double u[kSols], v[kSols], r[kSols];
  int cu[kSols], cv[kSols];
  int n;
};

// Results are grouped into minima by a fixed grid over the parameter domain (cells of
// kDistinct32 / kDistinct times the domain's extent): a grouping that depends on each result
// alone, unlike "within a distance of the current representative", so the records below hold
// the same values whatever order the seeds finish in.
template <typename T>
struct Cells {
  T u0, v0, iu, iv;  // domain origin, cells per parameter unit
};
// cell indices of an in-domain result (rounded down; saturating)
__device__ __forceinline__ int cell_index(float x) { return __float2int_rd(x); }
__device__ __forceinline__ int cell_index(double x) { return __double2int_rd(x); }
template <typename T>
__device__ __forceinline__ void cell_of(const Cells<T>& g, T u, T v, int& cu, int& cv) {
  cu = cell_index((u - g.u0) * g.iu);
  cv = cell_index((v - g.v0) * g.iv);
}

// R.1 = the minimum of all results (total order); R.2 = the minimum of the results outside
// R.1's cell.  Exact for any arrival order: a new overall minimum in another cell makes the
// old minimum (smaller than everything else seen) the runner-up.
__device__ __forceinline__ void merge32(Rec32& R, int cu, int cv, float u, float v, float d) {
  if (R.d1 < INFINITY && cu == R.cu1 && cv == R.cv1) {
    if (before(d, u, v, R.d1, R.u1, R.v1)) { R.u1 = u; R.v1 = v; R.d1 = d; }
  } else if (before(d, u, v, R.d1, R.u1, R.v1)) {
    R.u2 = R.u1; R.v2 = R.v1; R.d2 = R.d1;
    R.u1 = u; R.v1 = v; R.d1 = d; R.cu1 = cu; R.cv1 = cv;
  } else if (before(d, u, v, R.d2, R.u2, R.v2)) {
    R.u2 = u; R.v2 = v; R.d2 = d;
  }
}

// The kSols cells with the smallest minima, each with its minimum.  A cell evicted earlier can
// only come back with a smaller value than the one it was evicted with, so the kept values are
// exact cell minima whatever the arrival order.
__device__ __forceinline__ void merge64(Rec64& R, int cu, int cv, double u, double v, double r) {
  for (int k = 0; k < R.n; ++k)
    if (cu == R.cu[k] && cv == R.cv[k]) {
      if (before(r, u, v, R.r[k], R.u[k], R.v[k])) { R.u[k] = u; R.v[k] = v; R.r[k] = r; }
      return;
    }
  int slot = R.n;
  if (R.n >= kSols) {
    slot = 0;
    for (int k = 1; k < kSols; ++k)
      if (before(R.r[slot], R.u[slot], R.v[slot], R.r[k], R.u[k], R.v[k])) slot = k;
    if (!before(r, u, v, R.r[slot], R.u[slot], R.v[slot])) return;
  } else {
    ++R.n;
  }
  R.u[slot] = u; R.v[slot] = v; R.r[slot] = r; R.cu[slot] = cu; R.cv[slot] = cv;
}

// best minimum and status (FOUND / AMBIGUOUS): FOUND unless another distinct minimum is as
// close within 1e-6 relative
// A minimum within (tu, tv) of the best is the same minimum: results that converged to one
// point can fall on both sides of a grid-cell boundary (an exact parameter such as 0.5 is one).
__device__ __forceinline__ int finish_status(const double* us, const double* vs, const double* rs, int n, double tu,
                                             double tv, double& u, double& v, double& r) {
  int bi = 0;
  for (int k = 1; k < n; ++k)
    if (before(rs[k], us[k], vs[k], rs[bi], us[bi], vs[bi])) bi = k;
  u = us[bi];
  v = vs[bi];
  r = rs[bi];
  for (int k = 0; k < n; ++k)
    if (k != bi && rs[k] <= r * (1 + 1e-6) + 1e-12 && (fabs(us[k] - u) > tu || fabs(vs[k] - v) > tv))
      return 1;  // NURBS_INV_AMBIGUOUS
  return 0;
}

// A surface's context and FP32 breakpoint tables staged in shared memory, when the surface has at
// most KS spans per direction.
template <int KS>
struct SpanTables {
  static_assert(kGridBuckets % KS == 0, "the staged grid is a thinned one");
  Ctx ctx;    // one copy for all threads, its fields read where they are used
  bool fits;  // breakpoint tables staged
  // FP32 breakpoints and inverse span lengths, and a lookup grid over the domain: KS equal buckets,
  // each with the span of its left end (or one before)
  float2 seg[2][KS + 1];
  float g0[2], gs[2];  // bucket of x: (x - g0) * gs
  unsigned char grid[2][KS];

  // The span of x, as find_seg_hint's: two or three dependent shared-memory reads instead of a
  // bisection's 6 to 8 (which the whole warp runs as soon as one lane has left its last span; the
  // bisections took a quarter of an iteration of the exploration).
  __device__ __forceinline__ int span(int dir, int ns, float x) const {
    const int i = min(max((int)((x - g0[dir]) * gs[dir]), 0), KS - 1);
    int k = grid[dir][i];
    for (int n = 0; k < ns - 1 && x >= seg[dir][k + 1].x; ++n) {
      ++k;
      if (n == 3) {  // clustered knots
        for (int step = 1 << (31 - __clz(ns)); step > 0; step >>= 1)
          if (k + step < ns && seg[dir][k + step].x <= x) k += step;
        break;
      }
    }
    return k;
  }
};

// Cooperative over `nthreads` threads (index tid); the callers synchronise before and after.
template <int KS>
__device__ __forceinline__ void stage_tables(const SurfDev& s, SpanTables<KS>& sm, int tid, int nthreads) {
  const bool smem_tables = s.ns_u <= KS && s.ns_v <= KS;
  if (smem_tables) {
    for (int dir = 0; dir < 2; ++dir) {
      const float *b = dir ? s.bv32 : s.bu32, *inv = dir ? s.inv_dv32 : s.inv_du32;
      const int ns = dir ? s.ns_v : s.ns_u;
      for (int k = tid; k <= ns; k += nthreads) sm.seg[dir][k] = make_float2(b[k], k < ns ? inv[k] : 0.f);
      // the surface's lookup grid, thinned to KS buckets
      const unsigned char* grid = dir ? s.grid_v : s.grid_u;
      for (int i = tid; i < KS; i += nthreads) sm.grid[dir][i] = grid[i * (kGridBuckets / KS)];
      if (tid == 0) {
        sm.g0[dir] = dir ? s.g0_v : s.g0_u;
        sm.gs[dir] = (dir ? s.gs_v : s.gs_u) * ((float)KS / kGridBuckets);
      }
    }
  }
  if (tid == 0) {
    Ctx& cx = sm.ctx;
    sm.fits = smem_tables;
    cx.L32 = fast::global_locator<float>(s);
    cx.L64 = fast::global_locator<double>(s);
    cx.m32 = s.m32;
    cx.m64 = s.m64;
    cx.p = s.p;
    cx.q = s.q;
    cx.dom_u0 = s.dom_u0; cx.dom_u1 = s.dom_u1; cx.dom_v0 = s.dom_v0; cx.dom_v1 = s.dom_v1;
    cx.iru = s.inv_range_u; cx.irv = s.inv_range_v;
  }
}

// One surface staged in shared memory: tree boxes (FP32 outward-rounded and exact FP64), seed
// centres, domain, and breakpoint tables when the surface has at most KS spans per direction.
// FP64 breakpoint tables are staged only for the FP64 schedule: the mixed schedule reads them in
// its few final FP64 steps from global memory, which leaves more of the SM's memory to L1.
template <int KS, int MODE>
struct Staged : SpanTables<KS> {
  static constexpr int KS64 = MODE == kModeMixed ? 1 : KS;
  float box32[kTreeNodes][6];   // rounded outward: a point outside is outside the exact box
  float box32i[kTreeNodes][6];  // rounded inward: a point strictly inside is inside the exact box
  const TreeNodeDev* tree;     // exact FP64 boxes, read only near a face (global memory, L2)
  double ctr[kTreeNodes][2];
  float ctr32[kTreeNodes][2];
  double org[3];    // origin of the FP32 tables: FP32 iterations see P - org
  const float* cd32;   // S, Su, Sv at the node centres (FP32, relative to org), 9 per node
  const double* cd64;  // the same in FP64
  float dom32[4];
  float near32[4];  // 1 % of the extent around the domain: FP32 minima here are edge records
  float far32[4];  // two domain extents around the domain: an FP32 iterate beyond is abandoned
  Cells<float> cell32;
  Cells<double> cell64;
  int nb;
  double sb64[2][KS64 + 1], si64[2][KS64];
};

template <int P, int Q, int KS>
struct StagedEval {
  const SpanTables<KS>& sm;
  __device__ __forceinline__ void spans(float u, float v, int& hu, int& hv) const {
    if (sm.fits) {
      hu = sm.span(0, sm.ctx.L32.ns_u, u);
      hv = sm.span(1, sm.ctx.L32.ns_v, v);
    } else {
      GlobalEval<P, Q>{sm.ctx}.spans(u, v, hu, hv);
    }
  }
  template <int ORDER>
  __device__ __forceinline__ fast::SDer<float> at(float u, float v, int& hu, int& hv) const {
    const fast::Locator<float>& L = sm.ctx.L32;
    float bu, bv, iu, iv;
    spans(u, v, hu, hv);
    if (sm.fits) {
      const float2 a = sm.seg[0][hu], b = sm.seg[1][hv];
      bu = a.x;
      iu = a.y;
      bv = b.x;
      iv = b.y;
    } else {
      bu = L.bu[hu];
      iu = L.iu[hu];
      bv = L.bv[hv];
      iv = L.iv[hv];
    }
    const float lu = (u - bu) * iu, lv = (v - bv) * iv;
    return fast::eval_span<float, P, Q, ORDER, true>(sm.ctx.m32, sm.ctx.p, sm.ctx.q, L.ns_v, hu, hv, lu, lv, L.ru * iu,
                                                     L.rv * iv);
  }
};

// Per-warp bookkeeping of the task scheduler: the warp's 32 query slots.
template <int MODE>
struct WarpWork {
  long long sq[32];              // query index of the slot
  unsigned long long smask0[32]; // candidate nodes 0..63 of the slots in the current task list
  int slpref[32];                // exclusive prefix of the slots' task counts
  int sleft[32];                 // seeds of the slot's query that have not ended
  typename std::conditional<MODE == kModeMixed, Rec32, Rec64>::type rec[32];
  float sp32[MODE == kModeMixed ? 32 : 1][3];
  double sp64[MODE == kModeMixed ? 1 : 32][3];
};

// Queries a warp takes at least at a time: enough for a few seeds per lane (by the surface's average
// number of candidates, SurfDev::seeds), since a warp is busy until its longest seed ends and a refill
// ends with a pass of the final FP64 steps, as long with one query as with 32; but no more than
// `spread`, with which the launch has a warp on every scheduler.
template <int MODE>
__host__ __device__ inline int least_grab(float seeds, int64_t spread) {
  const float want = MODE == kModeMixed ? kGrabSeedsMixed : kGrabSeeds64;
  const int by_seeds = (int)(want / (seeds > 1.0f ? seeds : 1.0f)) + 1;
  const int k = (int)(spread < 1 ? 1 : (spread < (int64_t)by_seeds ? spread : (int64_t)by_seeds));
  return k < 32 ? k : 32;
}

// Where a warp of a persistent launch takes its next queries from: a global counter.  A warp asks
// for as many queries as it has free slots and gets its share of what is left, or `least`, so that
// a small launch spreads over all warps and a large one ends with all warps on their last queries.
struct QueryCounter {
  unsigned long long* next;
  int64_t n, seen;
  float share;  // 1 / resident warps
  int least;
  __device__ __forceinline__ int grab(int want, int64_t& q0) {
    const float fair = (float)(n - seen) * share;
    int k = fair < (float)want ? (int)fair + 1 : want;
    k = max(k, least);
    k = min(k, want);
    unsigned long long a = 0;
    if ((threadIdx.x & 31) == 0) a = atomicAdd(next, (unsigned long long)k);
    q0 = (int64_t)__shfl_sync(0xffffffffu, a, 0);
    seen = q0 + k;
    const int64_t left = n - q0;
    return left < k ? (left > 0 ? (int)left : 0) : k;
  }
};
// A launch's grid: as many warps as take their first queries at once (more would race for them, and
// leave some schedulers with several warps' queries and others with none), at most the resident ones.
struct StreamGrid {
  unsigned blocks;
  float share;
  int least;
};
template <int MODE>
inline StreamGrid stream_grid(const SurfDev& s, int64_t n, int64_t resident_ctas) {
  StreamGrid g;
  g.least = least_grab<MODE>(s.seeds, n / kSchedulers);
  const int64_t warps = (n + g.least - 1) / g.least, blocks = (warps + kWarps - 1) / kWarps;
  g.blocks = (unsigned)(blocks < resident_ctas ? blocks : resident_ctas);
  g.share = 1.0f / (float)((int64_t)g.blocks * kWarps);
  return g;
}

// Cooperative over `nthreads` threads (index tid): stages one surface and its context.
// The callers synchronise the participating threads before and after.
template <int KS, int MODE>
__device__ __forceinline__ void stage_surface(const SurfDev& s, Staged<KS, MODE>& sm, int tid, int nthreads) {
  constexpr int KS64 = Staged<KS, MODE>::KS64;
  stage_tables(s, sm, tid, nthreads);
  if (s.ns_u <= KS64 && s.ns_v <= KS64) {
    for (int dir = 0; dir < 2; ++dir) {
      const double *b64 = dir ? s.bv : s.bu, *inv64 = dir ? s.inv_dv : s.inv_du;
      const int ns = dir ? s.ns_v : s.ns_u;
      for (int k = tid; k <= ns; k += nthreads) {
        sm.sb64[dir][k] = b64[k];
        if (k < ns) sm.si64[dir][k] = inv64[k];
      }
    }
    if (tid == 0) {
      Ctx& cx = sm.ctx;
      cx.L64.bu = sm.sb64[0]; cx.L64.bv = sm.sb64[1]; cx.L64.iu = sm.si64[0]; cx.L64.iv = sm.si64[1];
    }
  }
  // built nodes are the root alone, or the root and all 64 children (the children of the
  // 2-level tree are built together when the root is divided), so node k keeps index k
  const int nb = s.built[1] ? kTreeNodes : (s.built[0] ? 1 : 0);
  for (int k = tid; k < nb; k += nthreads) {
    const TreeNodeDev& T = s.tree[k];
    for (int j = 0; j < 3; ++j) {
      sm.box32[k][j] = __double2float_rd(T.lb[j]);
      sm.box32[k][3 + j] = __double2float_ru(T.rt[j]);
      sm.box32i[k][j] = __double2float_ru(T.lb[j]);
      sm.box32i[k][3 + j] = __double2float_rd(T.rt[j]);
    }
    sm.ctr[k][0] = (T.uv_lb[0] + T.uv_rt[0]) / 2;  // kernel.cu:154
    sm.ctr[k][1] = (T.uv_lb[1] + T.uv_rt[1]) / 2;
    sm.ctr32[k][0] = (float)sm.ctr[k][0];
    sm.ctr32[k][1] = (float)sm.ctr[k][1];
  }
  if (tid == 0) {
    sm.nb = nb;
    sm.tree = s.tree;
    sm.cd32 = s.cd32;
    sm.cd64 = s.cd64;
    sm.org[0] = s.org[0];
    sm.org[1] = s.org[1];
    sm.org[2] = s.org[2];
    const float slack = 1e-4f;  // FP32 domain test is a prefilter; the FP64 phase decides
    sm.dom32[0] = (float)s.dom_u0 - slack;
    sm.dom32[1] = (float)s.dom_u1 + slack;
    sm.dom32[2] = (float)s.dom_v0 - slack;
    sm.dom32[3] = (float)s.dom_v1 + slack;
    const float fu = 2.0f * (float)(s.dom_u1 - s.dom_u0), fv = 2.0f * (float)(s.dom_v1 - s.dom_v0);
    sm.near32[0] = (float)s.dom_u0 - 5e-3f * fu;
    sm.near32[1] = (float)s.dom_u1 + 5e-3f * fu;
    sm.near32[2] = (float)s.dom_v0 - 5e-3f * fv;
    sm.near32[3] = (float)s.dom_v1 + 5e-3f * fv;
    sm.far32[0] = (float)s.dom_u0 - fu;
    sm.far32[1] = (float)s.dom_u1 + fu;
    sm.far32[2] = (float)s.dom_v0 - fv;
    sm.far32[3] = (float)s.dom_v1 + fv;
    const double eu = s.dom_u1 - s.dom_u0, ev = s.dom_v1 - s.dom_v0;
    sm.cell32 = {(float)s.dom_u0, (float)s.dom_v0, (float)(1.0 / ((double)kDistinct32 * eu)),
                 (float)(1.0 / ((double)kDistinct32 * ev))};
    sm.cell64 = {s.dom_u0, s.dom_v0, 1.0 / (kDistinct * eu), 1.0 / (kDistinct * ev)};
  }
}

// One warp inverts the queries that `src` hands out (src.grab), of the staged surface.
//
// The warp holds up to 32 queries in slots and its lanes run their (query, seed) pairs.  When the
// lanes have started every seed of the task list, the slots whose seeds have all ended get their
// final FP64 steps and results, and new queries take their place while the other slots' last
// seeds still run: the warp's lanes idle only at the end of the whole launch.  (With chunks of 32
// queries run to their end one after the other, every chunk ended with a few lanes on its longest
// seeds, and a launch of fewer than ~32 queries per resident warp left warps without work.)
// Which lane, slot or warp runs a seed, and when, does not change its arithmetic, and the
// per-query records do not depend on the order in which seeds end.
//
// COUNT: the work-counting variant (nurbs_invert_count): seed iterations and final FP64 polishes
// are added to counts[0] and counts[1]; the results are the same.
template <int P, int Q, int MODE, int KS, bool COUNT, class Source>
__device__ __forceinline__ void invert_stream(Staged<KS, MODE>& sm, WarpWork<MODE>& ww, const double* __restrict__ Pq,
                                              Source& src,
                                              double* __restrict__ uv_out, int* __restrict__ st_out,
                                              double* __restrict__ res_out,
                                              unsigned long long* __restrict__ counts = nullptr) {
  typedef typename std::conditional<MODE == kModeMixed, float, double>::type T;
  const Ctx& cx = sm.ctx;
  const StagedEval<P, Q, KS> ev{sm};
  unsigned n_iter = 0, n_final = 0;
  const int lane = threadIdx.x & 31;
  const unsigned FULL = 0xffffffffu;
  const unsigned lt_mask = (1u << lane) - 1u;
  constexpr int kBatch = MODE == kModeMixed ? kStartBatch : kStartBatch64;
  constexpr int kRefill = MODE == kModeMixed ? kRefillMixed : kRefill64;

  bool more = true;                    // src may have queries left
  bool used = false;                   // this lane's slot holds a query
  int total = 0, next = 0;             // task list: tasks, and how many have been started
  bool waiting = true;                 // this lane wants a seed (it runs one otherwise)
  int ql = 0;                          // its slot
  Seed<T> sd;
  T tx = 0, ty = 0, tz = 0;
  int end = kContinue;                 // how its last seed ended, until that is merged
  T dist = 0;                          // and the squared distance there

  // this lane's slot: the final FP64 steps (MIXED) and the result of its query
  auto finish_query = [&]() {
    const int64_t q = ww.sq[lane];
    int status;
    double ou = __longlong_as_double(0x7ff8000000000000ll), ov = ou, orr = ou;
    if constexpr (MODE == kModeMixed) {
      const double px = Pq[3 * q], py = Pq[3 * q + 1], pz = Pq[3 * q + 2];
      double us[3], vs[3], rs[3];
      int ns = 0;
      // FP64 minima reached from the records; two within kDistinct are one minimum (split by a
      // cell boundary), which keeps its smaller residual
      auto add = [&](double u, double v, double r) {
        for (int k = 0; k < ns; ++k)
          if (fabs(u - us[k]) <= kDistinct && fabs(v - vs[k]) <= kDistinct) {
            if (r < rs[k]) { us[k] = u; vs[k] = v; rs[k] = r; }
            return;
          }
        us[ns] = u; vs[ns] = v; rs[ns] = r; ++ns;
      };
      const Rec32& R = ww.rec[lane];
      const float dbest = fminf(R.d1, R.de);
      if (dbest < INFINITY) {
        // the runner-up also takes the FP64 steps when the best fails there, or when it is within
        // kPolishMargin of the best (an FP32 iterate that stopped in a flat valley overstates its
        // minimum's distance); one next to the best is the same minimum split by a cell boundary.
        // The edge record takes them when it is within the same margin.
        const float e1 = sqrtf(dbest) * (1.0f + kPolishMargin) + 1e-5f;
        const bool first = R.d1 < INFINITY;
        const bool second =
            first && R.d2 < INFINITY && !(fabsf(R.u2 - R.u1) <= kDistinct32 && fabsf(R.v2 - R.v1) <= kDistinct32);
        const bool tie = second && R.d2 <= e1 * e1, edge = R.de <= e1 * e1;
        // One loop over the lane's candidates, the next one taken up in the very iteration after the
        // last one's end: the warp's steps are the longest sum over a lane's candidates, not the sum
        // of the longest of the best, of the runners-up and of the edge records.
        int cand = first ? 0 : 2;
        Final f;
        final_start(ev, first ? R.u1 : R.ue, first ? R.v1 : R.ve, f);
        if constexpr (COUNT) ++n_final;
        while (cand < 3) {
          double r;
          const int end = final_step<P, Q>(cx, ev, px, py, pz, f, r);
          if (end == kContinue) continue;
          if (end == kConverged) add(f.u, f.v, r);
          const bool more2 = cand == 0 && (end == kConverged ? tie : second);
          cand = more2 ? 1 : (cand < 2 && edge ? 2 : 3);
          if (cand < 3) {
            final_start(ev, more2 ? R.u2 : R.ue, more2 ? R.v2 : R.ve, f);
            if constexpr (COUNT) ++n_final;
          }
        }
      }
      status = ns == 0 ? 3 : finish_status(us, vs, rs, ns, kDistinct, kDistinct, ou, ov, orr);
    } else {
      const Rec64& R = ww.rec[lane];
      double rs[kSols];
      for (int k = 0; k < kSols; ++k) rs[k] = k < R.n ? sqrt(R.r[k]) : 0.0;
      status = R.n == 0 ? 3 : finish_status(R.u, R.v, rs, R.n, 2.0 / sm.cell64.iu, 2.0 / sm.cell64.iv, ou, ov, orr);
    }
    uv_out[2 * q] = ou;
    uv_out[2 * q + 1] = ov;
    st_out[q] = status;
    res_out[q] = orr;
  };

  // A new query for this lane's slot: its candidates and an empty record.  Returns the number of
  // candidates; a query without any is answered at once.
  auto load_query = [&](int64_t q) {
    const double px = Pq[3 * q], py = Pq[3 * q + 1], pz = Pq[3 * q + 2];
    const float fx = (float)px, fy = (float)py, fz = (float)pz;
    // ---- cull (exact candidate set, ascending node order).  With f = fl(x) rounded to nearest,
    // f < rd(lb) implies x < lb and f > ru(lb) implies x > lb (rounding is monotone), so the
    // FP64 comparison only runs for coordinates within an FP32 ulp of a box face.
    uint64_t m0 = 0;
    unsigned m1 = 0;
    const int nbl = sm.nb;
    for (int k = 0; k < nbl; ++k) {
      if (fx >= sm.box32[k][0] && fy >= sm.box32[k][1] && fz >= sm.box32[k][2] && fx <= sm.box32[k][3] &&
          fy <= sm.box32[k][4] && fz <= sm.box32[k][5]) {
        const bool surely = fx > sm.box32i[k][0] && fy > sm.box32i[k][1] && fz > sm.box32i[k][2] &&
                            fx < sm.box32i[k][3] && fy < sm.box32i[k][4] && fz < sm.box32i[k][5];
        const TreeNodeDev* B = sm.tree + k;
        if (surely || (px >= B->lb[0] && py >= B->lb[1] && pz >= B->lb[2] && px <= B->rt[0] && py <= B->rt[1] &&
                       pz <= B->rt[2])) {
          if (k < 64) m0 |= 1ull << k;
          else m1 = 1u;
        }
      }
    }
    const int cnt = __popcll(m0) + (int)m1;
    if (cnt == 0) {
      const double nan = __longlong_as_double(0x7ff8000000000000ll);
      uv_out[2 * q] = nan;
      uv_out[2 * q + 1] = nan;
      st_out[q] = 2;  // NURBS_INV_NO_CANDIDATE
      res_out[q] = nan;
      return 0;
    }
    ww.sq[lane] = q;
    ww.smask0[lane] = m0;
    ww.sleft[lane] = cnt;
    if constexpr (MODE == kModeMixed) {
      // the FP32 iterations work relative to the FP32 tables' origin
      ww.sp32[lane][0] = (float)(px - sm.org[0]);
      ww.sp32[lane][1] = (float)(py - sm.org[1]);
      ww.sp32[lane][2] = (float)(pz - sm.org[2]);
      Rec32& R = ww.rec[lane];
      R.d1 = INFINITY;
      R.d2 = INFINITY;
      R.de = INFINITY;
      R.u1 = R.v1 = R.u2 = R.v2 = R.ue = R.ve = 0.f;
      R.cu1 = R.cv1 = 0;
    } else {
      ww.sp64[lane][0] = px;
      ww.sp64[lane][1] = py;
      ww.sp64[lane][2] = pz;
      ww.rec[lane].n = 0;
    }
    return cnt;
  };

  // Finishes the slots whose seeds have all ended, fills the free slots with new queries and lists
  // their tasks, a query's seeds consecutive in ascending node order.  When src has no queries left
  // the finished slots wait for the last ones (`last`): one pass of the final steps for all of them.
  auto refill = [&](bool last) {
    const bool ended = used && ww.sleft[lane] == 0;
    const unsigned fm = __ballot_sync(FULL, !used || ended);
    int64_t q0 = 0;
    int k = 0;
    if (more) {
      k = src.grab(__popc(fm), q0);
      more = k > 0;
    }
    if (ended && (more || last)) {
      finish_query();
      used = false;
    }
    int cnt = 0;
    const int r = __popc(fm & lt_mask);
    if (!used && r < k) {
      cnt = load_query(q0 + r);
      used = cnt > 0;
    }
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += t;
    }
    ww.slpref[lane] = incl - cnt;
    total = __shfl_sync(FULL, incl, 31);
    next = 0;
    __syncwarp();
  };

  // starts task t: its slot is the largest lane whose exclusive prefix is <= t (a lane without
  // tasks shares its prefix with the next lane and is never the largest)
  auto start = [&](int t) {
    int lo = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1)
      if (ww.slpref[lo + step] <= t) lo += step;
    ql = lo;
    const uint64_t mm = ww.smask0[ql];
    const int k = t - ww.slpref[lo];
    const int node = k < __popcll(mm) ? select_bit(mm, k) : 64;
    if constexpr (MODE == kModeMixed) {
      tx = ww.sp32[ql][0];
      ty = ww.sp32[ql][1];
      tz = ww.sp32[ql][2];
      sd.u = sm.ctr32[node][0];
      sd.v = sm.ctr32[node][1];
    } else {
      tx = ww.sp64[ql][0];
      ty = ww.sp64[ql][1];
      tz = ww.sp64[ql][2];
      sd.u = sm.ctr[node][0];
      sd.v = sm.ctr[node][1];
    }
    sd.prev = INFINITY;
    sd.it = 0;
    sd.hu = 0;
    sd.hv = 0;
    sd.newton = false;
    if constexpr (MODE == kModeMixed) first_step<float>(sm.cd32 + 9 * node, tx, ty, tz, sm.far32, sd);
    else first_step<double>(sm.cd64 + 9 * node, tx, ty, tz, sm.far32, sd);
  };

  bool none = true;  // no lane runs a seed
  for (;;) {
    refill(none);
    if (total == 0 && !more && !__any_sync(FULL, used)) break;
    // ---- seeds, until the lanes that want one find the list exhausted and enough slots are done
    for (;;) {
      const unsigned wm = __ballot_sync(FULL, waiting);
      none = wm == FULL;
      if (__popc(wm) >= kBatch || none) {
        // ---- the ended seeds' results, and the next seeds
        if (end != kContinue) atomicSub(&ww.sleft[ql], 1);
        int cu = 0, cv = 0;
        bool upd, edge = false;
        if constexpr (MODE == kModeMixed) {
          upd = end == kConverged && sd.u >= sm.dom32[0] && sd.u <= sm.dom32[1] && sd.v >= sm.dom32[2] &&
                sd.v <= sm.dom32[3];
          // An FP32 minimum within 1 % of the extent outside the domain: near an edge FP32 arithmetic
          // can end outside while FP64 steps from there reach a minimum inside.  The closest such
          // result of a query is kept apart and takes the final FP64 steps too when it is close.
          edge = end == kConverged && !upd && sd.u >= sm.near32[0] && sd.u <= sm.near32[1] && sd.v >= sm.near32[2] &&
                 sd.v <= sm.near32[3];
          if (upd) {
            // Records only improve, so a result that cannot change its query's record now never
            // will: only the others are merged, one lane at a time.
            cell_of(sm.cell32, sd.u, sd.v, cu, cv);
            const Rec32& R = ww.rec[ql];
            if (R.d1 < INFINITY && cu == R.cu1 && cv == R.cv1)
              upd = before(dist, sd.u, sd.v, R.d1, R.u1, R.v1);
            else
              upd = before(dist, sd.u, sd.v, R.d1, R.u1, R.v1) || before(dist, sd.u, sd.v, R.d2, R.u2, R.v2);
          }
          edge = edge && before(dist, sd.u, sd.v, ww.rec[ql].de, ww.rec[ql].ue, ww.rec[ql].ve);
        } else {
          if (end == kConverged) evaluate_dist2<P, Q>(cx, tx, ty, tz, sd.u, sd.v, sd.hu, sd.hv, dist);
          upd = end == kConverged && in_domain64(cx, sd.u, sd.v, dist);
          if (upd) cell_of(sm.cell64, sd.u, sd.v, cu, cv);
        }
        unsigned fm = __ballot_sync(FULL, upd || edge);
        while (fm) {
          const int j = __ffs(fm) - 1;
          if (lane == j) {
            if constexpr (MODE == kModeMixed) {
              Rec32& R = ww.rec[ql];
              if (upd) merge32(R, cu, cv, sd.u, sd.v, dist);
              else if (before(dist, sd.u, sd.v, R.de, R.ue, R.ve)) { R.ue = sd.u; R.ve = sd.v; R.de = dist; }
            } else {
              merge64(ww.rec[ql], cu, cv, sd.u, sd.v, dist);
            }
          }
          __syncwarp();
          fm &= fm - 1;
        }
        end = kContinue;
        __syncwarp();
        if (next < total) {
          const int t = next + __popc(wm & lt_mask);
          if (waiting && t < total) {
            waiting = false;
            start(t);
          }
          next += __popc(wm);
        } else {
          if (none) break;
          if (more && __popc(__ballot_sync(FULL, !used || ww.sleft[lane] == 0)) >= kRefill) break;
        }
      }
      if (!waiting) {
        int res;
        if constexpr (MODE == kModeMixed) {
          res = iterate32(ev, tx, ty, tz, sd, dist);
          if (res == kContinue &&
              !(sd.u >= sm.far32[0] && sd.u <= sm.far32[1] && sd.v >= sm.far32[2] && sd.v <= sm.far32[3]))
            res = kFailed;
        } else {
          res = iterate64<P, Q>(cx, tx, ty, tz, sd, dist);
        }
        if constexpr (COUNT) ++n_iter;
        if (res != kContinue) {
          end = res;
          waiting = true;
        }
      }
      __syncwarp();
    }
  }
  if constexpr (COUNT) {
    unsigned long long a = n_iter, b = n_final;
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if ((threadIdx.x & 31) == 0) {
      atomicAdd(counts, a);
      atomicAdd(counts + 1, b);
    }
  }
}

}  // namespace inv
}  // namespace gnurbs
