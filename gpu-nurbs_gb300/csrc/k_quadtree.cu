// Adaptive quadtree inversion (nurbs_invert_quadtree): the reference's first inversion, which
// needs no tree build — per query a breadth-first quadtree over the parameter domain, culled by
// control-net boxes (Inverse, src/kernel/kernel.cu:4-104; BoundingBoxCheck :106-149;
// getSplitType :251-298; NODE_MAX_SIZE 64, src/kernel/kernel.cuh:13).
//
// Per query, layer by layer: the nodes whose control-point box (widened by max_edge) holds P run a
// trajectory from their centre; a result counts when it converged inside the domain within max_edge
// of P; the first layer with a result answers (its closest result; AMBIGUOUS as in the inversion);
// otherwise each passing node is split by the reference's getSplitType and its children are the next
// layer, in the reference's order.  The box checks and split decisions are exact (minima and maxima,
// and getSplitType decided in FP32 only where its lengths are clearly off max_edge and else with the
// reference-order FP64 functions; this translation unit is compiled with --fmad=false), so the tree
// is the oracle's; the v-length uses the v-derivative, which the reference takes with
// MatrixSurfaceDerivativeU.  With MODE mixed every node's trajectory runs in FP32 and its end takes
// FP64 Newton steps (the mixed inversion's final steps).  Culled nodes are not split (their
// control-point box does not hold P, so neither does their surface); a layer of more than 64 nodes or
// 60 layers ends the query unanswered.
//
// Work distribution.  A persistent grid whose warps take portions of queries from a counter:
//   1. root: the trajectories from the domain's centre stream through the warp's lanes (a lane whose
//      query ended takes the portion's next one), their ends take the final FP64 steps 32 at a time.
//      This answers most queries.
//   2. the others collect in a queue; 32 at a time they are searched lane per query from the root's
//      children on (the root's split does not depend on the query and is decided once per warp).
//      Layers hold about one passing node, so a warp that searched one query at a time kept 1 lane
//      in 32 busy.
//   3. a query that meets a node of many control points, and the last one or two, are searched by the
//      whole warp: lanes stride over a node's control points and take a node's trajectory each.
// Measured on 2^18 points near the 64x64 surface (a search for 5 of every 32 queries), mixed:
// 3.2 ms with the warp per query, 1.7 ms so.
#include "invert_core.cuh"

namespace gnurbs {
namespace {

using namespace inv;

constexpr int kQtMax = 64;     // nodes per layer (NODE_MAX_SIZE)
constexpr int kQtLayers = 60;
constexpr int kPortion = 128;   // queries a warp takes at a time, at most
constexpr int kLaneCps = 512;   // control points of a node a lane scans alone

struct QtWarp {
  float ru[kPortion], rv[kPortion];   // mixed: ends of the root trajectories
  unsigned char list[kPortion], end[kPortion];
  long long rest[64];             // queries the root did not answer
  double node[2][kQtMax + 4][4];  // two layers: lb.u, lb.v, rt.u, rt.v
  int code[2][kQtMax + 4];        // index of the node's precomputed box, -1 when it has none
  double su[kQtMax], sv[kQtMax], sr[kQtMax];
  unsigned char pass[kQtMax], ok[kQtMax];
};

__device__ __forceinline__ int knot_span(const int* knot_idx, const double* b, int ns, double x) {
  return knot_idx[exact::find_seg(b, ns, x)];  // findSpan (Evaluate.cu:504-533) over the breakpoints
}

// getSplitType: 0 NOT_SPLIT, 1 SPLIT_V, 2 SPLIT_U, 3 SPLIT_UV
__device__ int split_type(const SurfDev& s, const double* nd, double max_edge) {
  const int p = s.p, q = s.q, k2 = q + 1, k12 = (p + 1) * (q + 1);
  const double iu = (nd[2] - nd[0]) / 4, iv = (nd[3] - nd[1]) / 4;
  double ul = 0, vl = 0;
  for (int i = 0; i < 4; ++i) {
    const double x = nd[0] + i * iu, y = nd[1] + i * iv;
    const int su = exact::find_seg(s.bu, s.ns_u, x), sv = exact::find_seg(s.bv, s.ns_v, y);
    const double du = s.bu[su + 1] - s.bu[su], dv = s.bv[sv + 1] - s.bv[sv];
    const double u = (x - s.bu[su]) / du, v = (y - s.bv[sv]) / dv;
    exact::DenseSpan M{s.m64 + (size_t)(su * s.ns_v + sv) * k12 * 4, k2};
    const v4<double> R = exact::point_r(M, p, q, u, v);
    const v3<double> a = exact::der_u(M, p, q, u, v, R, s.range_u / du);
    const v3<double> b = exact::der_v(M, p, q, u, v, R, s.range_v / dv);
    ul += sqrt(a.x * a.x + a.y * a.y + a.z * a.z);
    vl += sqrt(b.x * b.x + b.y * b.y + b.z * b.z);
  }
  ul *= (nd[2] - nd[0]) * 0.25;
  vl *= (nd[3] - nd[1]) * 0.25;
  if (ul < max_edge && vl < max_edge) return 0;
  if (nd[2] - nd[0] > 0.25 || nd[3] - nd[1] > 0.25) return 3;
  if (ul < max_edge) return 1;
  if (vl < max_edge) return 2;
  return 3;
}

// getSplitType decided in FP32 where that is safe: the lengths from the FP32 tables' derivatives,
// used when each differs from max_edge by more than 1 % of max_edge plus 0.1 % of itself and every
// sample falls in the same span as in FP64; otherwise the reference-order FP64 evaluation above.
// Measured against the FP64 lengths over 20,000 nodes (depths 0-8) of six surfaces up to degree 5
// and 256x256 nets, the FP32 lengths err by at most 1.4e-4 of themselves, so both give the same
// decision; the FP32 one costs a fraction of the FP64 work (the FP64 split types took most of a
// launch).
template <class Eval>
__device__ int split_type_fast(const SurfDev& s, const Eval& ev, const double* nd, double max_edge) {
  const double iu = (nd[2] - nd[0]) / 4, iv = (nd[3] - nd[1]) / 4;
  float ul = 0, vl = 0;
  bool exact = false;
  for (int i = 0; i < 4; ++i) {
    const double x = nd[0] + i * iu, y = nd[1] + i * iv;
    const int su = exact::find_seg(s.bu, s.ns_u, x), sv = exact::find_seg(s.bv, s.ns_v, y);
    int hu = su, hv = sv;
    const fast::SDer<float> d = ev.template at<1>((float)x, (float)y, hu, hv);
    exact = exact || hu != su || hv != sv;
    ul += sqrtf(dot3(d.Su, d.Su));
    vl += sqrtf(dot3(d.Sv, d.Sv));
  }
  ul *= (float)((nd[2] - nd[0]) * 0.25);
  vl *= (float)((nd[3] - nd[1]) * 0.25);
  const float me = (float)max_edge;
  exact = exact || !(fabsf(ul - me) > 0.01f * me + 1e-3f * ul) || !(fabsf(vl - me) > 0.01f * me + 1e-3f * vl);
  if (exact) return split_type(s, nd, max_edge);
  const bool us = ul < me, vs = vl < me;
  if (us && vs) return 0;
  if (nd[2] - nd[0] > 0.25 || nd[3] - nd[1] > 0.25) return 3;
  if (us) return 1;
  if (vs) return 2;
  return 3;
}

__device__ __forceinline__ void put_node(double* o, double a, double b, double c, double d) {
  o[0] = a;
  o[1] = b;
  o[2] = c;
  o[3] = d;
}

// Precomputed boxes of the top kQuadtreeDepth levels of square children (depth d, u index a, v index
// b: code = (4^d - 1) / 3 + a 2^d + b), written when the surface is converted.  Deeper nodes, and the
// halves of U / V splits, scan their control points.
__device__ __forceinline__ int child_code(int pc, int hu, int hv) {
  if (pc < 0) return -1;
  int d = 0, base = 0;
  while (pc >= base + (1 << (2 * d))) base += 1 << (2 * d++);
  if (d + 1 >= kQuadtreeDepth) return -1;
  const int a = (pc - base) >> d, b = (pc - base) & ((1 << d) - 1);
  return base + (1 << (2 * d)) + ((2 * a + hu) << (d + 1)) + (2 * b + hv);
}

// Partial box over a node's control points (the rows findSpan(lb.u) - p .. findSpan(rt.u), the
// same in v: BoundingBoxCheck's range), over elements t, t + stride, ..., as order keys.
struct CpRange {
  int i0, j0, nb;
  int64_t cnt;
};
__device__ __forceinline__ CpRange cp_range(const SurfDev& s, const double* nd) {
  const int i0 = knot_span(s.knot_u, s.bu, s.ns_u, nd[0]) - s.p, i1 = knot_span(s.knot_u, s.bu, s.ns_u, nd[2]);
  const int j0 = knot_span(s.knot_v, s.bv, s.ns_v, nd[1]) - s.q, j1 = knot_span(s.knot_v, s.bv, s.ns_v, nd[3]);
  const int nb = j1 - j0 + 1;
  return {i0, j0, nb, (int64_t)(i1 - i0 + 1) * nb};
}
__device__ __forceinline__ void node_box(const SurfDev& s, const CpRange& r, int t, int stride, long long* mn,
                                         long long* mx) {
  for (int c = 0; c < 3; ++c) {
    mn[c] = 0x7fffffffffffffffll;
    mx[c] = -0x7fffffffffffffffll - 1;
  }
  for (int64_t e = t; e < r.cnt; e += stride) {
    const int row = (int)(e / r.nb), col = (int)(e - (int64_t)row * r.nb);
    const double* x = s.cps + 3 * ((size_t)(r.i0 + row) * s.nv + (r.j0 + col));
    for (int c = 0; c < 3; ++c) {
      const long long k = fast::order_key(x[c]);
      mn[c] = k < mn[c] ? k : mn[c];
      mx[c] = k > mx[c] ? k : mx[c];
    }
  }
}
__device__ __forceinline__ double key_value(long long k) {
  return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffll));
}
__device__ __forceinline__ bool box_holds(const double* mn, const double* mx, double px, double py, double pz,
                                          double max_edge) {
  return px >= mn[0] - max_edge && px <= mx[0] + max_edge && py >= mn[1] - max_edge && py <= mx[1] + max_edge &&
         pz >= mn[2] - max_edge && pz <= mx[2] + max_edge;
}
// children of a node split by type t (1 V, 2 U, 3 both), in the reference's order; returns their number
__device__ __forceinline__ int put_children(int type, const double* nd, int pc, double* o, int* oc) {
  if (type == 0) return 0;
  const double lx = nd[0], ly = nd[1], rx = nd[2], ry = nd[3];
  const double mxu = (lx + rx) / 2, myv = (ly + ry) / 2;
  if (type == 3) {
    put_node(o, lx, ly, mxu, myv);
    put_node(o + 4, lx, myv, mxu, ry);
    put_node(o + 8, mxu, myv, rx, ry);
    put_node(o + 12, mxu, ly, rx, myv);
    oc[0] = child_code(pc, 0, 0);
    oc[1] = child_code(pc, 0, 1);
    oc[2] = child_code(pc, 1, 1);
    oc[3] = child_code(pc, 1, 0);
    return 4;
  }
  if (type == 2) {
    put_node(o, lx, ly, mxu, ry);
    put_node(o + 4, mxu, ly, rx, ry);
  } else {
    put_node(o, lx, ly, rx, myv);
    put_node(o + 4, lx, myv, rx, ry);
  }
  oc[0] = oc[1] = -1;
  return 2;
}

__device__ __forceinline__ void far_limits(const Ctx& c, float far[4]) {
  const float eu = 2.0f * (float)(c.dom_u1 - c.dom_u0), ev = 2.0f * (float)(c.dom_v1 - c.dom_v0);
  far[0] = (float)c.dom_u0 - eu;
  far[1] = (float)c.dom_u1 + eu;
  far[2] = (float)c.dom_v0 - ev;
  far[3] = (float)c.dom_v1 + ev;
}
template <typename T>
__device__ __forceinline__ void seed_start(T u, T v, Seed<T>& sd) {
  sd.u = u;
  sd.v = v;
  sd.prev = INFINITY;
  sd.it = 0;
  sd.hu = 0;
  sd.hv = 0;
  sd.newton = false;
}

// One node's trajectory from (u, v): FP64 (the inversion's FP64 iteration), or MIXED (the mixed
// inversion's FP32 iteration, the point relative to the control net's centre, then its FP64
// final steps).  True when it converged inside the domain within max_edge of P; (u, v, rr) the
// result.
template <int P, int Q, int MODE>
__device__ __noinline__ bool node_trajectory(const SurfDev& s, const SpanTables<kSmemSpans>& sm, double px, double py,
                                             double pz, double max_edge, double& u, double& v, double& rr) {
  const Ctx& cx = sm.ctx;
  if constexpr (MODE == kModeMixed) {
    const StagedEval<P, Q, kSmemSpans> ev{sm};
    Seed<float> sd;
    seed_start((float)u, (float)v, sd);
    const float tx = (float)(px - s.org[0]), ty = (float)(py - s.org[1]), tz = (float)(pz - s.org[2]);
    float far[4];
    far_limits(cx, far);
    float dist;
    int r = kContinue;
    while (r == kContinue) {
      r = iterate32(ev, tx, ty, tz, sd, dist);
      if (r == kContinue && !(sd.u >= far[0] && sd.u <= far[1] && sd.v >= far[2] && sd.v <= far[3])) r = kFailed;
    }
    if (r != kConverged) return false;
    u = sd.u;
    v = sd.v;
    return final64<P, Q>(cx, ev, px, py, pz, u, v, rr) && rr < max_edge;
  } else {
    Seed<double> sd;
    seed_start(u, v, sd);
    int r = kContinue;
    double dist2 = 0;
    while (r == kContinue) r = iterate64<P, Q>(cx, px, py, pz, sd, dist2);
    u = sd.u;
    v = sd.v;
    if (r != kConverged || !in_domain64(cx, u, v, dist2)) return false;
    rr = sqrt(dist2);
    return rr < max_edge;
  }
}

// One lane searches one query's tree from the root's children on (the root passed and had no
// result).  Returns the status, or -1 when the search meets a node of more than kLaneCps control
// points (it is then the warp's).
template <int P, int Q, int MODE>
__device__ __noinline__ int quadtree_lane(const SurfDev& s, const SpanTables<kSmemSpans>& sm, const double* __restrict__ qtbox,
                             int root_type, double px, double py, double pz, double max_edge, double& ou, double& ov,
                             double& orr) {
  double node[2][kQtMax][4];
  int code[2][kQtMax];
  double ru[kQtMax], rv[kQtMax], rr[kQtMax];
  const StagedEval<P, Q, kSmemSpans> ev{sm};
  const double root[4] = {s.dom_u0, s.dom_v0, s.dom_u1, s.dom_v1};
  int cur = 0, size = put_children(root_type, root, 0, node[0][0], code[0]);
  for (int layer = 1; layer < kQtLayers && size > 0; ++layer) {
    unsigned long long pass = 0;
    for (int i = 0; i < size; ++i) {
      const double* nd = node[cur][i];
      double mn[3], mx[3];
      if (code[cur][i] >= 0) {  // the top levels' boxes, written with the surface
        const double* b = qtbox + 6 * code[cur][i];
        for (int c = 0; c < 3; ++c) {
          mn[c] = b[c];
          mx[c] = b[3 + c];
        }
      } else {
        const CpRange r = cp_range(s, nd);
        if (r.cnt > kLaneCps) return -1;
        long long kn[3], kx[3];
        node_box(s, r, 0, 1, kn, kx);
        for (int c = 0; c < 3; ++c) {
          mn[c] = key_value(kn[c]);
          mx[c] = key_value(kx[c]);
        }
      }
      if (box_holds(mn, mx, px, py, pz, max_edge)) pass |= 1ull << i;
    }
    int nr = 0;
    for (unsigned long long m = pass; m; m &= m - 1) {
      const double* nd = node[cur][__ffsll((long long)m) - 1];
      double u = (nd[0] + nd[2]) / 2, v = (nd[1] + nd[3]) / 2, r;
      if (node_trajectory<P, Q, MODE>(s, sm, px, py, pz, max_edge, u, v, r)) {
        ru[nr] = u;
        rv[nr] = v;
        rr[nr] = r;
        ++nr;
      }
    }
    if (nr > 0) {  // the layer's closest result (ties: the lower node)
      int best = 0, status = 0;
      for (int i = 1; i < nr; ++i)
        if (rr[i] < rr[best]) best = i;
      for (int i = 0; i < nr; ++i)
        if (i != best && rr[i] <= rr[best] * (1 + 1e-6) + 1e-12 &&
            (fabs(ru[i] - ru[best]) > 1e-7 || fabs(rv[i] - rv[best]) > 1e-7))
          status = 1;
      ou = ru[best];
      ov = rv[best];
      orr = rr[best];
      return status;
    }
    int total = 0;
    for (unsigned long long m = pass; m; m &= m - 1) {
      const int i = __ffsll((long long)m) - 1;
      const int type = split_type_fast(s, ev, node[cur][i], max_edge);
      const int nch = type == 3 ? 4 : (type == 0 ? 0 : 2);
      if (total + nch > kQtMax) return 3;  // layer overflow: unanswered
      put_children(type, node[cur][i], code[cur][i], node[cur ^ 1][total], code[cur ^ 1] + total);
      total += nch;
    }
    cur ^= 1;
    size = total;
  }
  return 3;
}

// The whole warp searches one query's tree from the root's children on (the root passed and had no
// result): a node's control-point box is reduced by the warp, the passing nodes' trajectories and
// splits run one per lane.
template <int P, int Q, int MODE>
__device__ __noinline__ void quadtree_query(const SurfDev& s, const SpanTables<kSmemSpans>& sm, QtWarp& w,
                               const double* __restrict__ qtbox, const double* __restrict__ Pq, int64_t qi,
                               int root_type, double max_edge, double* __restrict__ uv_out, int* __restrict__ st_out, double* __restrict__ res_out) {
  const int lane = threadIdx.x & 31;
  const unsigned FULL = 0xffffffffu;
  const double px = Pq[3 * qi], py = Pq[3 * qi + 1], pz = Pq[3 * qi + 2];
  const StagedEval<P, Q, kSmemSpans> ev{sm};
  int cur = 0, status = 3;
  const double root[4] = {s.dom_u0, s.dom_v0, s.dom_u1, s.dom_v1};
  int size = root_type == 3 ? 4 : (root_type == 0 ? 0 : 2);
  double ou = __longlong_as_double(0x7ff8000000000000ll), ov = ou, orr = ou;
  if (lane == 0) put_children(root_type, root, 0, w.node[0][0], w.code[0]);
  __syncwarp();
  for (int layer = 1; layer < kQtLayers && size > 0; ++layer) {
    // ---- control-point boxes (BoundingBoxCheck), one node at a time, the warp striding over it
    for (int i = 0; i < size; ++i) {
      const double* nd = w.node[cur][i];
      double mn[3], mx[3];
      if (w.code[cur][i] >= 0) {  // the top levels' boxes, written with the surface
        const double* b = qtbox + 6 * w.code[cur][i];
        for (int c = 0; c < 3; ++c) {
          mn[c] = b[c];
          mx[c] = b[3 + c];
        }
      } else {
        long long kn[3], kx[3];
        node_box(s, cp_range(s, nd), lane, 32, kn, kx);
        for (int o = 16; o > 0; o >>= 1)
          for (int c = 0; c < 3; ++c) {
            const long long a = __shfl_xor_sync(FULL, kn[c], o), b = __shfl_xor_sync(FULL, kx[c], o);
            kn[c] = a < kn[c] ? a : kn[c];
            kx[c] = b > kx[c] ? b : kx[c];
          }
        for (int c = 0; c < 3; ++c) {
          mn[c] = key_value(kn[c]);
          mx[c] = key_value(kx[c]);
        }
      }
      if (lane == 0) w.pass[i] = box_holds(mn, mx, px, py, pz, max_edge) ? 1 : 0;
    }
    __syncwarp();
    // ---- trajectories of the passing nodes, one per lane
    for (int i = lane; i < size; i += 32) {
      w.ok[i] = 0;
      if (!w.pass[i]) continue;
      const double* nd = w.node[cur][i];
      double u = (nd[0] + nd[2]) / 2, v = (nd[1] + nd[3]) / 2, rr;
      if (node_trajectory<P, Q, MODE>(s, sm, px, py, pz, max_edge, u, v, rr)) {
        w.ok[i] = 1;
        w.su[i] = u;
        w.sv[i] = v;
        w.sr[i] = rr;
      }
    }
    __syncwarp();
    // ---- the layer's closest result (ties: the lower node), if any
    int best = -1;
    for (int i = 0; i < size; ++i)
      if (w.ok[i] && (best < 0 || w.sr[i] < w.sr[best])) best = i;
    if (best >= 0) {
      status = 0;
      for (int i = 0; i < size; ++i)
        if (w.ok[i] && i != best && w.sr[i] <= w.sr[best] * (1 + 1e-6) + 1e-12 &&
            (fabs(w.su[i] - w.su[best]) > 1e-7 || fabs(w.sv[i] - w.sv[best]) > 1e-7))
          status = 1;
      ou = w.su[best];
      ov = w.sv[best];
      orr = w.sr[best];
      break;
    }
    // ---- split the passing nodes (getSplitType) and compact their children in node order
    int nch[2] = {0, 0}, typ[2] = {0, 0};
    for (int r = 0; r < 2; ++r) {
      const int i = lane + 32 * r;
      if (i < size && w.pass[i]) {
        typ[r] = split_type_fast(s, ev, w.node[cur][i], max_edge);
        nch[r] = typ[r] == 3 ? 4 : (typ[r] == 0 ? 0 : 2);
      }
    }
    int total = 0, off[2];
    for (int r = 0; r < 2; ++r) {
      int incl = nch[r];
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += t;
      }
      off[r] = total + incl - nch[r];
      total += __shfl_sync(FULL, incl, 31);
    }
    if (total > kQtMax) break;  // layer overflow: unanswered
    if (total == 0) break;
    for (int r = 0; r < 2; ++r) {
      const int i = lane + 32 * r;
      if (nch[r] > 0) put_children(typ[r], w.node[cur][i], w.code[cur][i], w.node[cur ^ 1][off[r]], w.code[cur ^ 1] + off[r]);
    }
    __syncwarp();
    cur ^= 1;
    size = total;
  }
  if (lane == 0) {
    uv_out[2 * qi] = ou;
    uv_out[2 * qi + 1] = ov;
    st_out[qi] = status;
    res_out[qi] = orr;
  }
  __syncwarp();
}

// Register budget: 4 CTAs per SM (128 registers); the run-time degrees' variant 2.
template <int P, int Q, int MODE>
__global__ void __launch_bounds__(kThreads, P == 0 ? 2 : 4)
    k_invert_quadtree(SurfDev s, const double* __restrict__ qtbox, const double* __restrict__ Pq, int64_t n,
                      double max_edge, double* __restrict__ uv_out, int* __restrict__ st_out,
                      double* __restrict__ res_out, unsigned long long* __restrict__ counter, float share,
                      int least) {
  __shared__ SpanTables<kSmemSpans> sm;
  __shared__ QtWarp ww[kWarps];
  stage_tables(s, sm, threadIdx.x, blockDim.x);
  __syncthreads();
  const Ctx& cx = sm.ctx;
  const StagedEval<P, Q, kSmemSpans> ev{sm};
  QtWarp& w = ww[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const unsigned FULL = 0xffffffffu, lt_mask = (1u << lane) - 1u;
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  const double cu = (s.dom_u0 + s.dom_u1) / 2, cv = (s.dom_v0 + s.dom_v1) / 2;
  float far[4];
  far_limits(cx, far);
  int nrest = 0, root_type = -1;
  int64_t seen = 0;
  auto answer = [&](int64_t q, int status, double u, double v, double r) {
    uv_out[2 * q] = u;
    uv_out[2 * q + 1] = v;
    st_out[q] = status;
    res_out[q] = r;
  };
  // the last `cnt` queries of the queue
  auto search = [&](int cnt) {
    if (root_type < 0) {
      const double root[4] = {s.dom_u0, s.dom_v0, s.dom_u1, s.dom_v1};
      root_type = split_type_fast(s, ev, root, max_edge);
    }
    nrest -= cnt;
    unsigned byw = cnt <= 2 ? (1u << cnt) - 1u : 0u;  // searched by the whole warp
    if (cnt > 2) {
      bool big = false;
      if (lane < cnt) {
        const int64_t q = w.rest[nrest + lane];
        double u = nan, v = nan, r = nan;
        const int st = quadtree_lane<P, Q, MODE>(s, sm, qtbox, root_type, Pq[3 * q], Pq[3 * q + 1], Pq[3 * q + 2],
                                                 max_edge, u, v, r);
        big = st < 0;
        if (!big) answer(q, st, u, v, r);
      }
      byw = __ballot_sync(FULL, big);
    }
    for (; byw; byw &= byw - 1)
      quadtree_query<P, Q, MODE>(s, sm, w, qtbox, Pq, w.rest[nrest + __ffs(byw) - 1], root_type, max_edge, uv_out,
                                 st_out, res_out);
    __syncwarp();
  };
  // queues the queries of the lanes with `open`, and searches a full warp's worth
  auto queue = [&](bool open, int64_t q) {
    const unsigned m = __ballot_sync(FULL, open);
    if (open) w.rest[nrest + __popc(m & lt_mask)] = q;
    nrest += __popc(m);
    __syncwarp();
    if (nrest >= 32) search(32);
  };
  for (;;) {
    // this warp's share of what is left, a few queries at least
    const float fair = (float)(n - seen) * share;
    const int want = max(fair < (float)kPortion ? (int)fair + 1 : kPortion, least);
    unsigned long long a = 0;
    if (lane == 0) a = atomicAdd(counter, (unsigned long long)want);
    const int64_t q0 = (int64_t)__shfl_sync(FULL, a, 0);
    if (q0 >= n) break;
    seen = q0 + want;
    const int cnt = (int)(n - q0 < want ? n - q0 : want);
    // ---- the root's box: queries outside it have no candidate
    int total = 0;
    for (int base = 0; base < cnt; base += 32) {
      const int k = base + lane;
      bool pass = false;
      if (k < cnt) {
        const int64_t q = q0 + k;
        pass = box_holds(qtbox, qtbox + 3, Pq[3 * q], Pq[3 * q + 1], Pq[3 * q + 2], max_edge);
        if (!pass) answer(q, 2, nan, nan, nan);  // no node ever passes
      }
      const unsigned m = __ballot_sync(FULL, pass);
      if (pass) w.list[total + __popc(m & lt_mask)] = (unsigned char)k;
      total += __popc(m);
    }
    __syncwarp();
    // ---- trajectories from the domain's centre
    int next = 0, slot = 0;
    bool waiting = true;
    int end = kContinue;
    typedef typename std::conditional<MODE == kModeMixed, float, double>::type T;
    Seed<T> sd;
    T tx = 0, ty = 0, tz = 0, dist = 0;
    for (;;) {
      const unsigned wm = __ballot_sync(FULL, waiting);
      if (__popc(wm) >= (MODE == kModeMixed ? kStartBatch : kStartBatch64) || wm == FULL) {
        if constexpr (MODE == kModeMixed) {
          if (end != kContinue) {
            w.end[slot] = (unsigned char)end;
            w.ru[slot] = sd.u;
            w.rv[slot] = sd.v;
          }
        } else {
          bool open = false;
          const int64_t q = q0 + w.list[slot];
          if (end != kContinue) {
            const double r = sqrt(dist);
            if (end == kConverged && in_domain64(cx, sd.u, sd.v, dist) && r < max_edge) answer(q, 0, sd.u, sd.v, r);
            else open = true;
          }
          queue(open, q);
        }
        end = kContinue;
        if (next >= total && wm == FULL) break;
        const int t = next + __popc(wm & lt_mask);
        if (waiting && t < total) {
          waiting = false;
          slot = t;
          const int64_t q = q0 + w.list[t];
          if constexpr (MODE == kModeMixed) {
            tx = (float)(Pq[3 * q] - s.org[0]);
            ty = (float)(Pq[3 * q + 1] - s.org[1]);
            tz = (float)(Pq[3 * q + 2] - s.org[2]);
          } else {
            tx = Pq[3 * q];
            ty = Pq[3 * q + 1];
            tz = Pq[3 * q + 2];
          }
          seed_start((T)cu, (T)cv, sd);
        }
        next = min(next + __popc(wm), total);
      }
      if (!waiting) {
        if constexpr (MODE == kModeMixed) {
          end = iterate32(ev, tx, ty, tz, sd, dist);
          if (end == kContinue && !(sd.u >= far[0] && sd.u <= far[1] && sd.v >= far[2] && sd.v <= far[3])) end = kFailed;
        } else {
          end = iterate64<P, Q>(cx, tx, ty, tz, sd, dist);
        }
        waiting = end != kContinue;
      }
      __syncwarp();
    }
    __syncwarp();
    // ---- MIXED: the final FP64 steps of their ends
    if constexpr (MODE == kModeMixed) {
      for (int base = 0; base < total; base += 32) {
        const int k = base + lane;
        bool open = false;
        int64_t q = 0;
        if (k < total) {
          q = q0 + w.list[k];
          open = true;
          if (w.end[k] == kConverged) {
            double u = w.ru[k], v = w.rv[k], r;
            if (final64<P, Q>(cx, ev, Pq[3 * q], Pq[3 * q + 1], Pq[3 * q + 2], u, v, r) && r < max_edge) {
              answer(q, 0, u, v, r);
              open = false;
            }
          }
        }
        queue(open, q);
      }
    }
  }
  if (nrest > 0) search(nrest);
}

template <int P, int Q, int MODE>
cudaError_t launch_quadtree_mode(const SurfDev& s, const double* P_, int64_t n, double max_edge, double* uv, int* st_,
                                 double* res, unsigned long long* counter, cudaStream_t st) {
  if ((n + 31) / 32 > 0xffffffffLL) return cudaErrorInvalidValue;  // far beyond any device's memory
  static int cached[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (!cached[dev]) {
    int sms = 0, per_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_invert_quadtree<P, Q, MODE>, kThreads, 0);
    cached[dev] = (sms > 0 ? sms : 1) * (per_sm > 0 ? per_sm : 1);
  }
  // as many warps as take at least one query per scheduler of the launch (up to 32: a pass of the
  // final steps costs as much for one), at most the resident ones
  const int64_t spread = n / kSchedulers;
  const int least = (int)(spread < 1 ? 1 : (spread < 32 ? spread : 32));
  int64_t blocks = ((n + least - 1) / least + kWarps - 1) / kWarps;
  if (blocks > cached[dev]) blocks = cached[dev];
  k_invert_quadtree<P, Q, MODE><<<(unsigned)blocks, kThreads, 0, st>>>(s, s.qtbox, P_, n, max_edge, uv, st_, res,
                                                                       counter, 1.0f / (float)(blocks * kWarps), least);
  return cudaGetLastError();
}

template <int P, int Q>
cudaError_t launch_quadtree_pq(const SurfDev& s, const double* P_, int64_t n, double max_edge, double* uv, int* st_,
                               double* res, int precision, unsigned long long* counter, cudaStream_t st) {
  if (precision == kModeMixed)
    return launch_quadtree_mode<P, Q, kModeMixed>(s, P_, n, max_edge, uv, st_, res, counter, st);
  return launch_quadtree_mode<P, Q, kModeFP64>(s, P_, n, max_edge, uv, st_, res, counter, st);
}

}  // namespace

cudaError_t launch_invert_quadtree(const SurfDev& s, const double* P, int64_t n, double max_edge, double* uv,
                                   int* status, double* residual, int precision, unsigned long long* counter, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if (s.p == 3 && s.q == 3)
    return launch_quadtree_pq<3, 3>(s, P, n, max_edge, uv, status, residual, precision, counter, st);
  return launch_quadtree_pq<0, 0>(s, P, n, max_edge, uv, status, residual, precision, counter, st);
}

}  // namespace gnurbs
