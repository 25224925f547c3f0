// Point projection (nurbs_project): the closest point of the surface over its closed knot domain,
// for query points near the surface or far from it.
//
// Replaces the reference's unfinished projection (Project, src/kernel/kernel.cu:471-485, a
// <<<1,1>>> launch for one constant point; NormalBoundingBoxCheck :487-513; NormalBoundingBox
// :623-704; NormalBoxToNormalTreeNode :1613-1636) with one fused persistent kernel:
//   1. cull (FP32, relative to the control net's centre, the same operations and roundings as
//      the oracle's cull, so both select the same nodes): the distance bound UB is the
//      least distance from P to the 3x3 sub-lattice surface points of every built node; a node is
//      a candidate when its bound box is within UB of P and its normal cone, taken with both
//      signs, can face P from some point of the box's bounding ball;
//   2. each candidate is seeded at its 9x9 lattice point closest to P and iterated with projected
//      Newton steps and a line search inside the domain (the full Hessian J^T J + r.d2S where it
//      is positive definite, J^T J elsewhere; a coordinate held at a bound whose descent points
//      out of the domain, the other taking the 1-D step; every step halved until |S - P| does not
//      grow), so minima on the boundary, where S - P is not normal to the surface, are found too;
//   3. the converged results are merged into per-query records (grid cells of the domain, as in
//      the inversion) and the closest wins; AMBIGUOUS when another minimum is as close.
// Queries stream through a warp's slots and its lanes run their (query, seed) pairs, as the
// inversion's do (invert_core.cuh); one evaluation per lane and turn, a line search's trial points
// included, and the few seeds and final steps that need hundreds of them by the whole warp, 31
// halvings at once: one such query took as long as the rest of a launch.  The closest lattice point is
// searched per candidate, a candidate per lane, when a warp's tasks are listed.  Two schedules (template
// MODE): FP64 — every trajectory in FP64; MIXED — the trajectories in FP32 (tables relative to
// the control net's centre; steps below kWholeStep32 skip the line search, whose distance
// comparisons are rounding noise there), each query's best result and best of another grid cell
// kept, then FP64 projected Newton steps from the best, and from the other when it is within
// kPolishMargin of it or the best fails (project_polish_step, the FP64 schedule's iteration where
// those steps do not converge).  64x64 surface, 2^18 points, 20 % of them far: mixed 3.80 -> 2.23 ms,
// 3,000 points 1.09 -> 0.57 ms; FP64 20,000 points 3.36 -> 1.95 ms (against chunks of 32 queries with
// the line search inside an iteration).
#include "invert_core.cuh"

namespace gnurbs {
namespace {

using namespace inv;

constexpr int kMaxIterProj = 40;  // projected Newton iterations per seed (the oracle's cap)
constexpr int kMaxHalvings = 30;  // line-search halvings per iteration
// a Newton move this small ends a seed (far points have flat minima, where Newton converges
// slowly: the inversion's 1e-10 would leave the parameters ~1e-9 from the minimum)
constexpr double kTolNewtonProj = 1e-12;
constexpr double kWholeStep = 1e-6;  // steps below this skip the line search
constexpr int kLattice = kPts * kPts;

struct ProjStaged {
  float cone[kTreeNodes][kConeStride];
  float sub[kTreeNodes][9][3];  // the 3x3 sub-lattice (1, 4, 7)^2 of every node
};

template <int MODE>
struct ProjWarp {  // the warp's 32 query slots (as the inversion's)
  long long sq[32];
  unsigned long long smask0[32];
  int slpref[32], sleft[32];
  unsigned char psub[32][kTreeNodes];  // seed lattice index of (slot, node)
  typename std::conditional<MODE == kModeMixed, Rec32, Rec64>::type rec[32];
  double sp64[MODE == kModeMixed ? 1 : 32][3];  // the query
  float sp32[32][3];   // the query relative to the control net's centre, FP32
};

__device__ __forceinline__ float fdot3(const float* a, const float* b) {
  return (a[0] * b[0] + a[1] * b[1]) + a[2] * b[2];
}
__device__ __forceinline__ double clampd(double x, double lo, double hi) { return x < lo ? lo : (x > hi ? hi : x); }

constexpr float kWholeStep32 = 3e-4f;  // mixed: FP32 steps below this skip the line search
constexpr float kTolMove32 = 1e-6f;    // mixed: an FP32 move this small ends the exploration

__device__ __forceinline__ float clampv(float x, float lo, float hi) { return fminf(fmaxf(x, lo), hi); }
__device__ __forceinline__ double clampv(double x, double lo, double hi) { return clampd(x, lo, hi); }

// A seed of the projected Newton iteration: its point (u, v) with the squared distance f there, and
// the point to evaluate next: itself, or the trial point of its line search (step alpha (d0, d1)).
template <typename T>
struct PSeed {
  T u, v, un, vn, f, d0, d1, alpha;
  int it, ls;
  bool trial, newton;
  __device__ __forceinline__ void start(T u0, T v0) {
    u = un = u0;
    v = vn = v0;
    it = ls = 0;
    trial = newton = false;
    f = d0 = d1 = alpha = T(0);
  }
};

// One evaluation of a seed (S to second order at (un, vn), d) and what follows from it: a trial point
// that does not decrease the distance halves the step; any other point is the seed's next one, whose
// derivatives are then at hand for its Newton step.  Each trial is evaluated once, with derivatives,
// and every lane does one evaluation per call: a line search inside the iteration would evaluate the
// accepted point twice and hold up the warp for its longest search.  dist2: the squared distance, FP32
// before the last step, FP64 at the end point (for a knot range of 1: evaluate_dist2).
template <typename T>
__device__ __forceinline__ int project_advance(const fast::SDer<T>& d, const T dom[4], T px, T py, T pz, PSeed<T>& st,
                                               T& dist2) {
  constexpr bool kFp32 = sizeof(T) == 4;
  const v3<T> r = {d.S.x - px, d.S.y - py, d.S.z - pz};
  const T fn = dot3(r, r);
  auto moved_to = [&]() {  // (u, v) becomes (un, vn)
    T m;
    if constexpr (kFp32) m = fmaxf(fabsf(st.un - st.u), fabsf(st.vn - st.v));
    else m = fast::max_abs(st.un - st.u, st.vn - st.v);
    st.u = st.un;
    st.v = st.vn;
    if constexpr (kFp32) return m <= kTolMove32;
    else return fast::le_nonneg(m, kTolAny64) || (st.newton && fast::le_nonneg(m, kTolNewtonProj));
  };
  if (st.trial) {
    if (!(fn <= st.f) && st.ls < kMaxHalvings) {
      ++st.ls;
      st.alpha *= T(0.5);
      st.un = clampv(st.u - st.alpha * st.d0, dom[0], dom[1]);
      st.vn = clampv(st.v - st.alpha * st.d1, dom[2], dom[3]);
      return kContinue;
    }
    dist2 = kFp32 ? st.f : fn;
    if (moved_to()) return kConverged;
    if (++st.it >= kMaxIterProj) return kFailed;
  }
  st.f = fn;
  dist2 = fn;
  const T g0 = dot3(d.Su, r), g1 = dot3(d.Sv, r);
  const T a00 = dot3(d.Su, d.Su), a01 = dot3(d.Su, d.Sv), a11 = dot3(d.Sv, d.Sv);
  const T n00 = a00 + dot3(r, d.Suu), n01 = a01 + dot3(r, d.Suv), n11 = a11 + dot3(r, d.Svv);
  const auto ku = fast::order_key(st.u), kv = fast::order_key(st.v);
  const bool fu = !((ku <= fast::order_key(dom[0]) && fast::is_positive(g0)) ||
                    (ku >= fast::order_key(dom[1]) && fast::is_positive(-g0)));
  const bool fv = !((kv <= fast::order_key(dom[2]) && fast::is_positive(g1)) ||
                    (kv >= fast::order_key(dom[3]) && fast::is_positive(-g1)));
  T d0 = 0, d1 = 0;
  if (fu && fv) {
    st.newton = fast::is_positive(n00) && fast::is_positive(det2(n00, n01, n11));
    const T h00 = st.newton ? n00 : a00, h01 = st.newton ? n01 : a01, h11 = st.newton ? n11 : a11;
    const T det = det2(h00, h01, h11);
    if (!fast::is_positive(det)) return kFailed;
    const T inv = fast::rcp<kFp32>(det);
    d0 = fast::mad(h11, g0, -(h01 * g1)) * inv;
    d1 = fast::mad(h00, g1, -(h01 * g0)) * inv;
  } else if (fu) {
    st.newton = fast::is_positive(n00);
    const T h = st.newton ? n00 : a00;
    if (!fast::is_positive(h)) return kFailed;
    d0 = g0 / h;
  } else if (fv) {
    st.newton = fast::is_positive(n11);
    const T h = st.newton ? n11 : a11;
    if (!fast::is_positive(h)) return kFailed;
    d1 = g1 / h;
  } else {
    return kConverged;  // a corner where the distance grows into the domain
  }
  T step;
  if constexpr (kFp32) {
    if (!(isfinite(d0) && isfinite(d1))) return kFailed;
    step = fmaxf(fabsf(d0), fabsf(d1));
  } else {
    if (!(fast::is_finite(d0) && fast::is_finite(d1))) return kFailed;
    step = fast::max_abs(d0, d1);
  }
  st.un = clampv(st.u - d0, dom[0], dom[1]);
  st.vn = clampv(st.v - d1, dom[2], dom[3]);
  // a step below kWholeStep is taken whole (its decrease is below the rounding of the distance, so
  // comparing distances would stop it at random near the minimum)
  if (kFp32 ? step > (T)kWholeStep32 : step > (T)kWholeStep) {
    st.d0 = d0;
    st.d1 = d1;
    st.alpha = T(1);
    st.ls = 0;
    st.trial = true;
    return kContinue;
  }
  st.trial = false;
  const T du = st.u - st.un, dv = st.v - st.vn;
  if (moved_to()) {
    if constexpr (!kFp32) dist2 = dist2_after(r, d.Su, d.Sv, du, dv);
    return kConverged;
  }
  return ++st.it >= kMaxIterProj ? kFailed : kContinue;
}

// The evaluations of one precision: S to the given order at (u, v).
template <int P, int Q, int KS, typename T>
struct ProjEval {
  const SpanTables<KS>& sm;
  template <int ORDER>
  __device__ __forceinline__ fast::SDer<T> at(T u, T v, int& hu, int& hv) const {
    if constexpr (sizeof(T) == 4) return StagedEval<P, Q, KS>{sm}.template at<ORDER>(u, v, hu, hv);
    else return fast::eval_at<double, P, Q, ORDER>(sm.ctx.L64, sm.ctx.m64, sm.ctx.p, sm.ctx.q, u, v, hu, hv);
  }
};

// Runs lane j's seed to its end with the whole warp: every trial point of a line search at once, one
// per lane, the first that decreases the distance (or the last) taken, as one after the other would.
// For the few seeds that need hundreds of trials, which otherwise hold up their launch.  Returns how
// the seed ended; its state and dist2 come back in lane j's (and every lane's) st and dist2.
template <typename T, class Eval>
__device__ __forceinline__ int project_by_warp(const Eval& ev, const T dom[4], int j, T px, T py, T pz, PSeed<T>& st,
                                               T& dist2) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  auto from = [&](T x) { return __shfl_sync(FULL, x, j); };
  px = from(px);
  py = from(py);
  pz = from(pz);
  st.u = from(st.u);
  st.v = from(st.v);
  st.un = from(st.un);
  st.vn = from(st.vn);
  st.f = from(st.f);
  st.d0 = from(st.d0);
  st.d1 = from(st.d1);
  st.alpha = from(st.alpha);
  st.it = __shfl_sync(FULL, st.it, j);
  st.ls = __shfl_sync(FULL, st.ls, j);
  st.trial = __shfl_sync(FULL, (int)st.trial, j) != 0;
  st.newton = __shfl_sync(FULL, (int)st.newton, j) != 0;
  int hu = 0, hv = 0;
  for (;;) {
    if (st.trial) {
      const T alpha = sizeof(T) == 4 ? (T)__int_as_float((127 - lane) << 23) : (T)__hiloint2double((1023 - lane) << 20, 0);
      const T tu = clampv(st.u - alpha * st.d0, dom[0], dom[1]), tv = clampv(st.v - alpha * st.d1, dom[2], dom[3]);
      const fast::SDer<T> e = ev.template at<0>(tu, tv, hu, hv);
      const v3<T> r = {e.S.x - px, e.S.y - py, e.S.z - pz};
      const bool ok = lane >= st.ls && lane <= kMaxHalvings && (dot3(r, r) <= st.f || lane == kMaxHalvings);
      const int first = __ffs(__ballot_sync(FULL, ok)) - 1;
      st.un = __shfl_sync(FULL, tu, first);
      st.vn = __shfl_sync(FULL, tv, first);
      st.ls = kMaxHalvings;  // taken
    }
    const int res = project_advance(ev.template at<2>(st.un, st.vn, hu, hv), dom, px, py, pz, st, dist2);
    if (res != kContinue) return res;
  }
}

// MIXED: the final FP64 steps from an FP32 result, as the inversion's (final64): S, Su, Sv in FP64
// and the Hessian's curvature term from FP32 second derivatives, projected onto the domain as the
// trajectories are, without a line search (the FP32 result lies in its minimum's basin); at most
// kPolishSteps, converged at a move <= kTolNewtonProj, the residual from the last step's S, Su, Sv.
// False when it does not converge: the caller then runs the FP64 schedule's iteration.
constexpr int kPolishSteps = 8;
// One such step: kConverged (res the residual), kFailed or kContinue.
template <int P, int Q, class Eval>
__device__ __forceinline__ int project_polish_step(const Ctx& c, const Eval& ev, double px, double py, double pz,
                                                   Final& f, double& res) {
  const fast::SDer<double> d = fast::eval_at<double, P, Q, 1>(c.L64, c.m64, c.p, c.q, f.u, f.v, f.hu, f.hv);
  const fast::SDer<float> e = ev.template at<2>((float)f.u, (float)f.v, f.hu32, f.hv32);
  const v3<double> r = {d.S.x - px, d.S.y - py, d.S.z - pz};
  const double g0 = dot3(d.Su, r), g1 = dot3(d.Sv, r);
  const double a00 = dot3(d.Su, d.Su), a01 = dot3(d.Su, d.Sv), a11 = dot3(d.Sv, d.Sv);
  const double n00 = a00 + dot3c(r, e.Suu), n01 = a01 + dot3c(r, e.Suv), n11 = a11 + dot3c(r, e.Svv);
  const long long ku = fast::order_key(f.u), kv = fast::order_key(f.v);
  const bool fu = !((ku <= fast::order_key(c.dom_u0) && fast::is_positive(g0)) ||
                    (ku >= fast::order_key(c.dom_u1) && fast::is_positive(-g0)));
  const bool fv = !((kv <= fast::order_key(c.dom_v0) && fast::is_positive(g1)) ||
                    (kv >= fast::order_key(c.dom_v1) && fast::is_positive(-g1)));
  double d0 = 0, d1 = 0;
  if (fu && fv) {
    const bool newton = fast::is_positive(n00) && fast::is_positive(det2(n00, n01, n11));
    const double h00 = newton ? n00 : a00, h01 = newton ? n01 : a01, h11 = newton ? n11 : a11;
    const double det = det2(h00, h01, h11);
    if (!fast::is_positive(det)) return kFailed;
    const double inv = fast::rcp<false>(det);
    d0 = fast::mad(h11, g0, -(h01 * g1)) * inv;
    d1 = fast::mad(h00, g1, -(h01 * g0)) * inv;
  } else if (fu) {
    const double h = fast::is_positive(n00) ? n00 : a00;
    if (!fast::is_positive(h)) return kFailed;
    d0 = g0 * fast::rcp<false>(h);
  } else if (fv) {
    const double h = fast::is_positive(n11) ? n11 : a11;
    if (!fast::is_positive(h)) return kFailed;
    d1 = g1 * fast::rcp<false>(h);
  }
  if (!(fast::is_finite(d0) && fast::is_finite(d1))) return kFailed;
  const double un = clampd(f.u - d0, c.dom_u0, c.dom_u1), vn = clampd(f.v - d1, c.dom_v0, c.dom_v1);
  const double du = f.u - un, dv = f.v - vn;
  f.u = un;
  f.v = vn;
  if (fast::le_nonneg(fast::max_abs(du, dv), kTolNewtonProj)) {
    const double dist2 = dist2_after(r, d.Su, d.Sv, du * c.iru, dv * c.irv);
    res = sqrt(dist2);
    return fast::is_finite(dist2) ? kConverged : kFailed;
  }
  return ++f.it < kPolishSteps ? kContinue : kFailed;
}

// Slots free or finished before the task list is refilled (invert_core.cuh: a refill culls its new
// queries and takes the finished ones through the final FP64 steps).  16 / 24 / 28 / 30: 2,254 / 2,266 /
// 2,155 / 2,186 us on 262,147 points of the 64x64 surface, mixed; the same within 2 % on 30,000 and below.
constexpr int kRefillProj = 28;
// At the end of a launch, this many running seeds of a warp are taken over by the whole warp, one after
// the other.  0 / 2 / 4 / 8: 64x64 surface, mixed, 262,147 points 2,070 / 2,152 / 2,155 / 2,201 us, 500
// points 146 / 145 / 153 / 171; FP64, 3,000 points 1,576 / 1,196 / 1,385 / 1,653, 20,000 points 1,976 /
// 1,397 / 1,599 / 1,973; 8x8 surface, FP64, 3,000 points 1,170 / 684 / 1,474 / 1,712; quintic 64x64, FP64,
// 3,000 points 1,964 / 1,121 / 1,676 / 2,978; 300x40 net, FP64, 6,000 points 2,822 / 1,770 with 2 / 4.  The
// launch is then as long as one warp's last seeds, and no value is best everywhere.
constexpr int kByWarp = 4;

// One warp projects the queries that `src` hands out, streaming them through its slots as the
// inversion does (invert_stream).
template <int P, int Q, int MODE, class Source>
__device__ __forceinline__ void project_stream(const Staged<kSmemSpans, MODE>& sm, const ProjStaged& ps,
                                               const float* __restrict__ lattice, ProjWarp<MODE>& ww,
                                               const double* __restrict__ Pq, Source& src, double* __restrict__ uv_out,
                                               int* __restrict__ st_out, double* __restrict__ res_out) {
  typedef typename std::conditional<MODE == kModeMixed, float, double>::type T;
  constexpr int kBatch = MODE == kModeMixed ? kStartBatch : kStartBatch64;
  const Ctx& cx = sm.ctx;
  const ProjEval<P, Q, kSmemSpans, T> ev{sm};
  const int lane = threadIdx.x & 31;
  const unsigned FULL = 0xffffffffu;
  const unsigned lt_mask = (1u << lane) - 1u;
  const T dom[4] = {(T)cx.dom_u0, (T)cx.dom_u1, (T)cx.dom_v0, (T)cx.dom_v1};
  const double nan = __longlong_as_double(0x7ff8000000000000ll);

  bool more = true, used = false, waiting = true, none = true;
  int total = 0, next = 0, ql = 0;
  int end = kContinue;
  PSeed<T> sd;
  sd.start(T(0), T(0));
  T tx = 0, ty = 0, tz = 0, dist = 0;
  int hu = 0, hv = 0;

  auto write = [&](int64_t q, int status, double u, double v, double r) {
    uv_out[2 * q] = u;
    uv_out[2 * q + 1] = v;
    st_out[q] = status;
    res_out[q] = r;
  };

  // the final steps and results of the lanes' slots (all lanes call it; fin: this lane's is finished)
  auto finish_queries = [&](bool fin) {
    double ou = nan, ov = nan, orr = nan;
    int status = 3;
    const int64_t q = fin ? ww.sq[lane] : 0;
    if constexpr (MODE == kModeMixed) {
      // the FP64 projected Newton steps from the best FP32 result, and from the best outside its cell
      // when that one is as close within kPolishMargin, or when the best fails
      const StagedEval<P, Q, kSmemSpans> e32{sm};
      const ProjEval<P, Q, kSmemSpans, double> e64{sm};
      const double dom64[4] = {cx.dom_u0, cx.dom_u1, cx.dom_v0, cx.dom_v1};
      double px = 0, py = 0, pz = 0, us[2], vs[2], rs[2];
      int ns = 0, cand = 2;
      const Rec32& R = ww.rec[lane];
      bool second = false, tie = false;
      Final f;
      f.u = f.v = 0;
      f.it = f.hu = f.hv = f.hu32 = f.hv32 = 0;
      if (fin && R.d1 < INFINITY) {
        px = Pq[3 * q];
        py = Pq[3 * q + 1];
        pz = Pq[3 * q + 2];
        const float e1 = sqrtf(R.d1) * (1.0f + kPolishMargin) + 1e-5f;
        second = R.d2 < INFINITY && !(fabsf(R.u2 - R.u1) <= kDistinct32 && fabsf(R.v2 - R.v1) <= kDistinct32);
        tie = second && R.d2 <= e1 * e1;
        cand = 0;
        final_start(e32, R.u1, R.v1, f);
      }
      // one loop over the lanes' candidates, as the inversion's: the second is taken up in the very
      // iteration after the first one's end
      while (__any_sync(FULL, cand < 2)) {
        int res = kContinue;
        double rr = 0;
        if (cand < 2) res = project_polish_step<P, Q>(cx, e32, px, py, pz, f, rr);
        for (unsigned fm = __ballot_sync(FULL, res == kFailed); fm; fm &= fm - 1) {
          // where the steps do not converge: the FP64 schedule's iteration from the FP32 result
          const int j = __ffs(fm) - 1;
          PSeed<double> s64;
          s64.start(cand == 0 ? R.u1 : R.u2, cand == 0 ? R.v1 : R.v2);
          double d2 = 0;
          const int r = project_by_warp(e64, dom64, j, px, py, pz, s64, d2);
          if (lane == j) {
            if (r == kConverged) evaluate_dist2<P, Q>(cx, px, py, pz, s64.u, s64.v, 0, 0, d2);
            res = r == kConverged && fast::is_finite(d2) ? kConverged : kFailed;
            f.u = s64.u;
            f.v = s64.v;
            rr = sqrt(d2);
          }
        }
        if (res != kContinue) {
          if (res == kConverged) {
            if (ns == 1 && fabs(f.u - us[0]) <= kDistinct && fabs(f.v - vs[0]) <= kDistinct) {
              if (rr < rs[0]) { us[0] = f.u; vs[0] = f.v; rs[0] = rr; }
            } else {
              us[ns] = f.u;
              vs[ns] = f.v;
              rs[ns] = rr;
              ++ns;
            }
          }
          cand = cand == 0 && (res == kConverged ? tie : second) ? 1 : 2;
          if (cand == 1) final_start(e32, R.u2, R.v2, f);
        }
      }
      if (ns > 0) status = finish_status(us, vs, rs, ns, kDistinct, kDistinct, ou, ov, orr);
    } else if (fin) {
      const Rec64& R = ww.rec[lane];
      double rs[kSols];
      for (int k = 0; k < kSols; ++k) rs[k] = k < R.n ? sqrt(R.r[k]) : 0.0;
      if (R.n > 0)
        status = finish_status(R.u, R.v, rs, R.n, 2.0 / sm.cell64.iu, 2.0 / sm.cell64.iv, ou, ov, orr);
    }
    if (fin) write(q, status, ou, ov, orr);
  };

  // a new query for this lane's slot: its candidates (the oracle's arithmetic, operation for
  // operation) and an empty record; a query without any (a non-finite one) is answered at once
  auto load_query = [&](int64_t q) {
    const double px = Pq[3 * q], py = Pq[3 * q + 1], pz = Pq[3 * q + 2];
    const float Pf[3] = {(float)(px - sm.org[0]), (float)(py - sm.org[1]), (float)(pz - sm.org[2])};
    const int nbl = sm.nb;
    uint64_t m0 = 0;
    unsigned m1 = 0;
    float ub2 = INFINITY;
    for (int k = 0; k < nbl; ++k)
      for (int j = 0; j < 9; ++j) {
        const float dd3[3] = {ps.sub[k][j][0] - Pf[0], ps.sub[k][j][1] - Pf[1], ps.sub[k][j][2] - Pf[2]};
        const float dd = fdot3(dd3, dd3);
        ub2 = ub2 < dd ? ub2 : dd;
      }
    ub2 = ub2 * (1.0f + 0x1p-10f);
    for (int k = 0; k < nbl; ++k) {
      const float* rc = ps.cone[k];
      float g[3];
      for (int c = 0; c < 3; ++c) {
        const float lo = rc[9 + c] - Pf[c], hi = Pf[c] - rc[12 + c];
        g[c] = lo > hi ? lo : hi;
        g[c] = g[c] > 0.0f ? g[c] : 0.0f;
      }
      const bool nearb = fdot3(g, g) <= ub2;
      const float dv[3] = {Pf[0] - rc[0], Pf[1] - rc[1], Pf[2] - rc[2]};
      const float dd = fdot3(dv, dv), r = rc[3];
      float e = dd - r * r;
      e = e > 0.0f ? e : 0.0f;
      const bool seen = rc[7] * sqrtf(e) <= fabsf(fdot3(dv, rc + 4)) + rc[8] * r;
      if (nearb && seen) {
        if (k < 64) m0 |= 1ull << k;
        else m1 = 1u;
      }
    }
    const int cnt = __popcll(m0) + (int)m1;
    if (cnt == 0) {
      write(q, 2, nan, nan, nan);  // NURBS_INV_NO_CANDIDATE
      return 0;
    }
    ww.sq[lane] = q;
    ww.smask0[lane] = m0;
    ww.sleft[lane] = cnt;
    ww.sp32[lane][0] = Pf[0];
    ww.sp32[lane][1] = Pf[1];
    ww.sp32[lane][2] = Pf[2];
    if constexpr (MODE == kModeMixed) {
      Rec32& R = ww.rec[lane];
      R.d1 = R.d2 = R.de = INFINITY;
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

  // task t of the list: its slot and node (invert_stream's)
  auto decode = [&](int t, int& slot, int& node) {
    int lo = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1)
      if (ww.slpref[lo + step] <= t) lo += step;
    slot = lo;
    const uint64_t mm = ww.smask0[lo];
    const int k = t - ww.slpref[lo];
    node = k < __popcll(mm) ? select_bit(mm, k) : 64;
  };

  auto refill = [&](bool last) {
    const bool ended = used && ww.sleft[lane] == 0;
    const unsigned fm = __ballot_sync(FULL, !used || ended);
    int64_t q0 = 0;
    int k = 0;
    if (more) {
      k = src.grab(__popc(fm), q0);
      more = k > 0;
    }
    if (more || last) {
      finish_queries(ended);
      if (ended) used = false;
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
    // the seeds: per task the node's lattice point closest to P (first of equals), a task per lane
    for (int t = lane; t < total; t += 32) {
      int slot, node;
      decode(t, slot, node);
      const float x0 = ww.sp32[slot][0], x1 = ww.sp32[slot][1], x2 = ww.sp32[slot][2];
      const float* L = lattice + (size_t)node * kLattice * 3;
      float best = INFINITY;
      int bi = 0;
#pragma unroll 9
      for (int j = 0; j < kLattice; ++j) {
        const float x[3] = {__ldg(L + 3 * j) - x0, __ldg(L + 3 * j + 1) - x1, __ldg(L + 3 * j + 2) - x2};
        const float ee = fdot3(x, x);
        if (ee < best) {
          best = ee;
          bi = j;
        }
      }
      ww.psub[slot][node] = (unsigned char)bi;
    }
    __syncwarp();
  };

  auto start = [&](int t) {
    int node;
    decode(t, ql, node);
    if constexpr (MODE == kModeMixed) {
      tx = ww.sp32[ql][0];
      ty = ww.sp32[ql][1];
      tz = ww.sp32[ql][2];
    } else {
      tx = ww.sp64[ql][0];
      ty = ww.sp64[ql][1];
      tz = ww.sp64[ql][2];
    }
    // the lattice point's parameters, as the samples compute them
    const int j = ww.psub[ql][node];
    const unsigned bx = node == 0 ? 0u : (unsigned)(node - 1) / kGap, by = node == 0 ? 0u : (unsigned)(node - 1) % kGap;
    const double base_unit = node == 0 ? 1.0 : 1.0 / kGap, unit = base_unit * (1.0 / kGap);
    const double u = clampd(base_unit * bx + (j / kPts) * unit, cx.dom_u0, cx.dom_u1);
    const double v = clampd(base_unit * by + (j % kPts) * unit, cx.dom_v0, cx.dom_v1);
    sd.start(clampv((T)u, dom[0], dom[1]), clampv((T)v, dom[2], dom[3]));
    hu = hv = 0;
  };

  for (;;) {
    refill(none);
    if (total == 0 && !more && !__any_sync(FULL, used)) break;
    for (;;) {
      unsigned wm = __ballot_sync(FULL, waiting);
      if (!more && next >= total && wm != FULL && __popc(~wm) <= kByWarp) {
        // the last seeds of the launch
        for (unsigned am = ~wm; am; am &= am - 1) {
          const int j = __ffs(am) - 1;
          PSeed<T> one = sd;
          T d2 = dist;
          const int r = project_by_warp(ev, dom, j, tx, ty, tz, one, d2);
          if (lane == j) {
            sd = one;
            dist = d2;
            end = r;
            waiting = true;
          }
        }
        wm = FULL;
      }
      none = wm == FULL;
      if (__popc(wm) >= kBatch || none) {
        if (end != kContinue) atomicSub(&ww.sleft[ql], 1);
        int cu = 0, cv = 0;
        bool upd = end == kConverged;
        if constexpr (MODE == kModeMixed) {
          if (upd) {
            cell_of(sm.cell32, sd.u, sd.v, cu, cv);
            const Rec32& R = ww.rec[ql];
            if (R.d1 < INFINITY && cu == R.cu1 && cv == R.cv1)
              upd = before(dist, sd.u, sd.v, R.d1, R.u1, R.v1);
            else
              upd = before(dist, sd.u, sd.v, R.d1, R.u1, R.v1) || before(dist, sd.u, sd.v, R.d2, R.u2, R.v2);
          }
        } else {
          if (upd) evaluate_dist2<P, Q>(cx, tx, ty, tz, sd.u, sd.v, hu, hv, dist);
          upd = upd && fast::is_finite(dist);
          if (upd) cell_of(sm.cell64, sd.u, sd.v, cu, cv);
        }
        unsigned fm = __ballot_sync(FULL, upd);
        while (fm) {
          const int j = __ffs(fm) - 1;
          if (lane == j) {
            if constexpr (MODE == kModeMixed) merge32(ww.rec[ql], cu, cv, sd.u, sd.v, dist);
            else merge64(ww.rec[ql], cu, cv, sd.u, sd.v, dist);
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
          if (more && __popc(__ballot_sync(FULL, !used || ww.sleft[lane] == 0)) >= kRefillProj) break;
        }
      }
      if (!waiting) {
        const int res = project_advance(ev.template at<2>(sd.un, sd.vn, hu, hv), dom, tx, ty, tz, sd, dist);
        if (res != kContinue) {
          end = res;
          waiting = true;
        }
      }
      __syncwarp();
    }
  }
}

// Shared memory (dynamic, above the 48 KB of static allocations): the staged surface, the cone
// records and sub-lattice points, and the warps' bookkeeping.
template <int MODE>
struct ProjSmem {
  static constexpr size_t ps = (sizeof(Staged<kSmemSpans, MODE>) + 15) / 16 * 16;
  static constexpr size_t ww = ps + (sizeof(ProjStaged) + 15) / 16 * 16;
  static constexpr size_t bytes = ww + sizeof(ProjWarp<MODE>) * kWarps;
};

// Register budget: the FP64 schedule and the run-time degrees keep 168 registers (3 CTAs per SM); the
// mixed one of a compiled degree 128 (4 / 5 / 6 CTAs per SM: 2.23 / 2.45 / 2.57 ms on 2^18 points of the
// 64x64 surface).
template <int P, int Q, int MODE>
__global__ void __launch_bounds__(kThreads, (MODE == kModeMixed && P != 0) ? 4 : 3)
    k_project(SurfDev s, const double* __restrict__ Pq, int64_t n, double* __restrict__ uv_out,
              int* __restrict__ st_out, double* __restrict__ res_out, unsigned long long* __restrict__ counter,
              float share, int least) {
  extern __shared__ __align__(16) unsigned char smem[];
  Staged<kSmemSpans, MODE>& sm = *reinterpret_cast<Staged<kSmemSpans, MODE>*>(smem);
  ProjStaged& ps = *reinterpret_cast<ProjStaged*>(smem + ProjSmem<MODE>::ps);
  ProjWarp<MODE>* ww = reinterpret_cast<ProjWarp<MODE>*>(smem + ProjSmem<MODE>::ww);
  stage_surface<kSmemSpans>(s, sm, threadIdx.x, blockDim.x);
  for (int e = threadIdx.x; e < kTreeNodes * kConeStride; e += blockDim.x)
    ps.cone[e / kConeStride][e % kConeStride] = s.cone[e];
  for (int e = threadIdx.x; e < kTreeNodes * 9; e += blockDim.x) {
    const int k = e / 9, j = e % 9, a = 1 + 3 * (j / 3), b = 1 + 3 * (j % 3);
    const float* x = s.lattice + ((size_t)k * kLattice + kPts * a + b) * 3;
    ps.sub[k][j][0] = x[0];
    ps.sub[k][j][1] = x[1];
    ps.sub[k][j][2] = x[2];
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5;
  QueryCounter src{counter, n, 0, share, least};
  project_stream<P, Q, MODE>(sm, ps, s.lattice, ww[warp], Pq, src, uv_out, st_out, res_out);
}

template <int P, int Q, int MODE>
cudaError_t launch_project_mode(const SurfDev& s, const double* P_, int64_t n, double* uv, int* st_, double* res,
                                unsigned long long* counter, cudaStream_t st) {
  if ((n + 31) / 32 > 0x3fffffffLL) return cudaErrorInvalidValue;  // far beyond any device's memory
  constexpr size_t bytes = ProjSmem<MODE>::bytes;
  static int cached[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (!cached[dev]) {
    cudaError_t e = cudaFuncSetAttribute(k_project<P, Q, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    int sms = 0, per_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_project<P, Q, MODE>, kThreads, bytes);
    cached[dev] = (sms > 0 ? sms : 1) * (per_sm > 0 ? per_sm : 1);
  }
  // at least what puts a warp on every scheduler, up to 16: culling and final steps cost a warp about
  // as much for one query (8 / 16 / 32: 64x64 surface, FP64, 20,000 points 1,707 / 1,599 / 1,550 us, 8x8
  // 1,742 / 1,467 / 1,556; mixed the same within 3 %)
  const int64_t spread = n / kSchedulers;
  const int least = (int)(spread < 1 ? 1 : (spread < 16 ? spread : 16));
  int64_t blocks = ((n + least - 1) / least + kWarps - 1) / kWarps;
  if (blocks > cached[dev]) blocks = cached[dev];
  k_project<P, Q, MODE><<<(unsigned)blocks, kThreads, bytes, st>>>(s, P_, n, uv, st_, res, counter,
                                                                    1.0f / (float)(blocks * kWarps), least);
  return cudaGetLastError();
}

template <int P, int Q>
cudaError_t launch_project_pq(const SurfDev& s, const double* P_, int64_t n, double* uv, int* st_, double* res,
                              int precision, unsigned long long* counter, cudaStream_t st) {
  if (precision == kModeMixed) return launch_project_mode<P, Q, kModeMixed>(s, P_, n, uv, st_, res, counter, st);
  return launch_project_mode<P, Q, kModeFP64>(s, P_, n, uv, st_, res, counter, st);
}

}  // namespace

cudaError_t launch_project(const SurfDev& s, const double* P, int64_t n, double* uv, int* status, double* residual,
                           int precision, unsigned long long* counter, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if (s.p == 3 && s.q == 3) return launch_project_pq<3, 3>(s, P, n, uv, status, residual, precision, counter, st);
  if (s.p == 5 && s.q == 5) return launch_project_pq<5, 5>(s, P, n, uv, status, residual, precision, counter, st);
  return launch_project_pq<0, 0>(s, P, n, uv, status, residual, precision, counter, st);
}

}  // namespace gnurbs
