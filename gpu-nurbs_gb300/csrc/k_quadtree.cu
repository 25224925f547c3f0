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
//   2. the others collect in a queue; 32 at a time they are searched layer by layer from the root's
//      children on, a query per lane (the root's split does not depend on the query and is decided once
//      per warp).  Layers hold about one passing node, so a warp that searched one query at a time kept
//      1 lane in 32 busy.  The trajectories and splits of the layer's passing nodes are one list of
//      tasks for all lanes, and a node of many control points is scanned by the whole warp, so neither
//      makes one lane the last.
//   3. a query whose layer outgrows what a lane keeps is searched on by the whole warp, a node per lane.
// Measured with a warp per query / a lane per query, its trajectories one after the other / now:
//   64x64 surface, mixed, 2^18 points within 5e-5      3,236 / 1,548 / 1,270 us  (max_edge 1e-4)
//   64x64 surface, mixed, 20,000 points off by ~3e-5   1,339 / 3,204 /   729 us  (max_edge 1e-4)
//   8x8 rough surface, FP64, 20,000 off by ~3e-2       5,172 / 52,467 / 4,103 us (max_edge 0.1: wide layers)
//   degrees 7 and 4, mixed, 6,000 off by ~3e-3         3,457 / 6,963 / 2,156 us  (max_edge 1e-2)
// The stack is what a lane keeps (576 bytes of layers, 1.6 KB with the calls' frames; 7.4 KB with whole
// layers per lane): the context reserves it for every resident thread, 156 MiB (1,866 MiB).
#include "invert_core.cuh"

namespace gnurbs {
namespace {

using namespace inv;

constexpr int kQtMax = 64;     // nodes per layer (NODE_MAX_SIZE)
constexpr int kQtLayers = 60;
constexpr int kPortion = 128;   // queries a warp takes at a time, at most
// Nodes of a layer that a lane keeps.  4 / 8 / 16: 26.5 / 23.6 / 20.0 ms on 200,000 points off the 64x64
// surface, 128 / 109 / 90 ms on a biquadratic one, but 16 reserve 352 MiB of local memory instead of 156.
constexpr int kLaneNodes = 8;
// Cost of a warp's scan of a node besides its control points, in control points of a lane's scan.  700x700
// net, 500 points off by ~2e-3: 2,854 / 2,766 / 2,750 / 2,847 us with 0 / 2 / 8 / 32, 4,416 with the lanes
// alone.
constexpr int kWarpScan = 8;

struct QtWarp {
  float ru[kPortion], rv[kPortion];   // mixed: ends of the root trajectories
  unsigned char list[kPortion], end[kPortion];
  unsigned char open[kPortion];       // the portion's queries that the root did not answer
  long long rest[32];                 // queries to be searched
  double node[2][kQtMax + 4][4];  // two layers: lb.u, lb.v, rt.u, rt.v
  int code[2][kQtMax + 4];        // index of the node's precomputed box, -1 when it has none
  double su[kQtMax], sv[kQtMax], sr[kQtMax];
  unsigned char pass[kQtMax], ok[kQtMax], owner[32];
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
template <int MODE, class Eval>
__device__ __noinline__ int split_type_fast(const SurfDev& s, const Eval& ev, const double* nd, double max_edge) {
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
// The same by the whole warp: every lane's result is the node's box.
__device__ __forceinline__ void warp_box(const SurfDev& s, const CpRange& r, long long* mn, long long* mx) {
  node_box(s, r, threadIdx.x & 31, 32, mn, mx);
  for (int o = 16; o > 0; o >>= 1)
    for (int c = 0; c < 3; ++c) {
      const long long a = __shfl_xor_sync(0xffffffffu, mn[c], o), b = __shfl_xor_sync(0xffffffffu, mx[c], o);
      mn[c] = a < mn[c] ? a : mn[c];
      mx[c] = b > mx[c] ? b : mx[c];
    }
}
__device__ __forceinline__ bool box_holds(const double* mn, const double* mx, double px, double py, double pz,
                                          double max_edge) {
  return px >= mn[0] - max_edge && px <= mx[0] + max_edge && py >= mn[1] - max_edge && py <= mx[1] + max_edge &&
         pz >= mn[2] - max_edge && pz <= mx[2] + max_edge;
}
// Whether the box of each lane's node (of the lanes with `have`) holds the lane's point.  The nodes
// without a precomputed box are scanned by their lanes, or one after the other by the whole warp where
// that is less work.
__device__ __forceinline__ bool lane_box_holds(const SurfDev& s, const double* __restrict__ qtbox, bool have,
                                               const double* nd, int code, double px, double py, double pz,
                                               double max_edge) {
  const unsigned FULL = 0xffffffffu;
  const bool scan = have && code < 0;
  double mn[3], mx[3];
  if (have && !scan) {  // the top levels' boxes, written with the surface
    const double* b = qtbox + 6 * code;
    for (int c = 0; c < 3; ++c) {
      mn[c] = b[c];
      mx[c] = b[3 + c];
    }
  }
  unsigned left = __ballot_sync(FULL, scan);
  if (left) {
    CpRange r = {0, 0, 1, 0};
    if (scan) r = cp_range(s, nd);
    const unsigned c = (unsigned)(r.cnt < 0x100000 ? r.cnt : 0x100000);
    const unsigned longest = __reduce_max_sync(FULL, c);
    const unsigned together = __reduce_add_sync(FULL, scan ? c / 32 + kWarpScan : 0u);
    long long kn[3], kx[3];
    if (longest <= together) {
      if (scan) node_box(s, r, 0, 1, kn, kx);
    } else {
      for (; left; left &= left - 1) {
        const int j = __ffs(left) - 1;
        const CpRange rj = {__shfl_sync(FULL, r.i0, j), __shfl_sync(FULL, r.j0, j), __shfl_sync(FULL, r.nb, j),
                            __shfl_sync(FULL, r.cnt, j)};
        long long an[3], ax[3];
        warp_box(s, rj, an, ax);
        if ((threadIdx.x & 31) == j)
          for (int k = 0; k < 3; ++k) {
            kn[k] = an[k];
            kx[k] = ax[k];
          }
      }
    }
    if (scan)
      for (int k = 0; k < 3; ++k) {
        mn[k] = fast::key_value(kn[k]);
        mx[k] = fast::key_value(kx[k]);
      }
  }
  return have && box_holds(mn, mx, px, py, pz, max_edge);
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
    if (r != kConverged) return false;
    evaluate_dist2<P, Q>(cx, px, py, pz, u, v, sd.hu, sd.hv, dist2);
    if (!in_domain64(cx, u, v, dist2)) return false;
    rr = sqrt(dist2);
    return rr < max_edge;
  }
}

// The whole warp searches one query's tree from layer `layer` on, whose `size` nodes are in w.node[0] and
// w.code[0] (no layer before had a result): a node's control-point box is reduced by the warp, the
// passing nodes' trajectories and splits run one per lane.
template <int P, int Q, int MODE>
__device__ __noinline__ void quadtree_query(const SurfDev& s, const SpanTables<kSmemSpans>& sm, QtWarp& w,
                                            const double* __restrict__ qtbox, const double* __restrict__ Pq,
                                            int64_t qi, int layer, int size, double max_edge,
                                            double* __restrict__ uv_out, int* __restrict__ st_out,
                                            double* __restrict__ res_out) {
  const int lane = threadIdx.x & 31;
  const unsigned FULL = 0xffffffffu;
  const double px = Pq[3 * qi], py = Pq[3 * qi + 1], pz = Pq[3 * qi + 2];
  const StagedEval<P, Q, kSmemSpans> ev{sm};
  int cur = 0, status = 3;
  double ou = __longlong_as_double(0x7ff8000000000000ll), ov = ou, orr = ou;
  for (; layer < kQtLayers && size > 0; ++layer) {
    // ---- control-point boxes (BoundingBoxCheck), a node per lane
    for (int base = 0; base < size; base += 32) {
      const int i = base + lane;
      const int k = i < size ? i : 0;
      const bool held = lane_box_holds(s, qtbox, i < size, w.node[cur][k], w.code[cur][k], px, py, pz, max_edge);
      if (i < size) w.pass[i] = held ? 1 : 0;
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
        typ[r] = split_type_fast<MODE>(s, ev, w.node[cur][i], max_edge);
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

// The warp searches up to 32 queries' trees, a query per lane, from the root's children on (the root
// passed and had no result), layer by layer.  A lane keeps its query's layer (kLaneNodes nodes) and scans
// the control points of its nodes; the trajectories and the splits of all the lanes' passing nodes are
// one list of tasks, which the lanes take 32 at a time, so a query with several passing nodes does not
// run them one after the other on its lane.  A query whose layer is wider is searched on by the whole
// warp (quadtree_query).  rest: the queries; cnt: their number.
template <int P, int Q, int MODE>
__device__ __forceinline__ void quadtree_search(const SurfDev& s, const SpanTables<kSmemSpans>& sm, QtWarp& w,
                                                const double* __restrict__ qtbox, const double* __restrict__ Pq,
                                                const long long* rest, int cnt, int root_type, double max_edge,
                                                double* __restrict__ uv_out, int* __restrict__ st_out,
                                                double* __restrict__ res_out) {
  const int lane = threadIdx.x & 31;
  const unsigned FULL = 0xffffffffu;
  const StagedEval<P, Q, kSmemSpans> ev{sm};
  double node[2][kLaneNodes][4];
  int code[2][kLaneNodes];
  const long long q = lane < cnt ? rest[lane] : 0;
  bool open = lane < cnt;  // not answered yet
  int cur = 0, size = 0;
  if (open) {
    const double root[4] = {s.dom_u0, s.dom_v0, s.dom_u1, s.dom_v1};
    size = put_children(root_type, root, 0, node[0][0], code[0]);
  }
  auto answer = [&](int status, double u, double v, double r) {
    uv_out[2 * q] = u;
    uv_out[2 * q + 1] = v;
    st_out[q] = status;
    res_out[q] = r;
    open = false;
  };
  // the position of this lane's first task when each lane has as many as `mask` has bits, and the total
  auto place = [&](unsigned mask, int& total) {
    const int k = __popc(mask);
    int incl = k;
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += t;
    }
    total = __shfl_sync(FULL, incl, 31);
    return incl - k;
  };
  for (int layer = 1; layer < kQtLayers && __any_sync(FULL, size > 0); ++layer) {
    // ---- control-point boxes (BoundingBoxCheck)
    unsigned pass = 0;
    for (int i = 0; __any_sync(FULL, i < size); ++i) {
      const int k = i < size ? i : 0;
      if (lane_box_holds(s, qtbox, i < size, node[cur][k], code[cur][k], Pq[3 * q], Pq[3 * q + 1], Pq[3 * q + 2],
                         max_edge))
        pass |= 1u << i;
    }
    // ---- trajectories of the passing nodes; the converged ones' (u, v, residual) in node order replace
    // the layer before this one
    int total, nr = 0;
    int first = place(pass, total);
    for (int base = 0; base < total; base += 32) {
      int t = first - base;
      for (unsigned m = pass; m; m &= m - 1, ++t)
        if (t >= 0 && t < 32) {
          const double* nd = node[cur][__ffs(m) - 1];
          w.owner[t] = (unsigned char)lane;
          w.su[t] = (nd[0] + nd[2]) / 2;
          w.sv[t] = (nd[1] + nd[3]) / 2;
        }
      __syncwarp();
      const bool task = base + lane < total;
      const long long qo = __shfl_sync(FULL, q, task ? w.owner[lane] : 0);
      if (task) {
        double u = w.su[lane], v = w.sv[lane], rr = 0;
        w.ok[lane] = node_trajectory<P, Q, MODE>(s, sm, Pq[3 * qo], Pq[3 * qo + 1], Pq[3 * qo + 2], max_edge, u, v, rr);
        w.su[lane] = u;
        w.sv[lane] = v;
        w.sr[lane] = rr;
      }
      __syncwarp();
      t = first - base;
      for (unsigned m = pass; m; m &= m - 1, ++t)
        if (t >= 0 && t < 32 && w.ok[t]) {
          double* o = node[cur ^ 1][nr++];
          o[0] = w.su[t];
          o[1] = w.sv[t];
          o[2] = w.sr[t];
        }
      __syncwarp();
    }
    // ---- the layer's closest result (ties: the lower node), if any
    if (nr > 0) {
      const double(*o)[4] = node[cur ^ 1];
      int best = 0, status = 0;
      for (int i = 1; i < nr; ++i)
        if (o[i][2] < o[best][2]) best = i;
      for (int i = 0; i < nr; ++i)
        if (i != best && o[i][2] <= o[best][2] * (1 + 1e-6) + 1e-12 &&
            (fabs(o[i][0] - o[best][0]) > 1e-7 || fabs(o[i][1] - o[best][1]) > 1e-7))
          status = 1;
      answer(status, o[best][0], o[best][1], o[best][2]);
      pass = 0;
    }
    // ---- the passing nodes' split types (getSplitType), two bits each
    unsigned types = 0;
    first = place(pass, total);
    for (int base = 0; base < total; base += 32) {
      int t = first - base;
      for (unsigned m = pass; m; m &= m - 1, ++t)
        if (t >= 0 && t < 32) {
          const double* nd = node[cur][__ffs(m) - 1];
          put_node(w.node[0][t], nd[0], nd[1], nd[2], nd[3]);
        }
      __syncwarp();
      if (base + lane < total) w.ok[lane] = (unsigned char)split_type_fast<MODE>(s, ev, w.node[0][lane], max_edge);
      __syncwarp();
      t = first - base;
      for (unsigned m = pass; m; m &= m - 1, ++t)
        if (t >= 0 && t < 32) types |= (unsigned)w.ok[t] << (2 * (__ffs(m) - 1));
      __syncwarp();
    }
    // ---- their children, in node order
    auto children = [&](int i) {
      const unsigned type = types >> (2 * i) & 3u;
      return type == 3 ? 4 : (type == 0 ? 0 : 2);
    };
    int many = 0;
    for (unsigned m = pass; m; m &= m - 1) many += children(__ffs(m) - 1);
    if (many > kQtMax) many = 0;  // layer overflow: unanswered
    auto put_layer = [&](double (*o)[4], int* oc) {
      int at = 0;
      for (unsigned m = pass; m; m &= m - 1) {
        const int i = __ffs(m) - 1;
        at += put_children((int)(types >> (2 * i) & 3u), node[cur][i], code[cur][i], o[at], oc + at);
      }
    };
    const bool wide = many > kLaneNodes;
    if (many > 0 && !wide) put_layer(node[cur ^ 1], code[cur ^ 1]);
    for (unsigned wm = __ballot_sync(FULL, wide); wm; wm &= wm - 1) {
      const int j = __ffs(wm) - 1;
      if (lane == j) {
        put_layer(w.node[0], w.code[0]);
        open = false;
      }
      __syncwarp();
      quadtree_query<P, Q, MODE>(s, sm, w, qtbox, Pq, __shfl_sync(FULL, q, j), layer + 1, __shfl_sync(FULL, many, j),
                                 max_edge, uv_out, st_out, res_out);
    }
    size = wide ? 0 : many;
    cur ^= 1;
  }
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  if (open) answer(3, nan, nan, nan);
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
  int nrest = 0, nopen = 0, root_type = -1;
  int64_t seen = 0;
  auto answer = [&](int64_t q, int status, double u, double v, double r) {
    uv_out[2 * q] = u;
    uv_out[2 * q + 1] = v;
    st_out[q] = status;
    res_out[q] = r;
  };
  // the lanes' queries k of the portion that the root did not answer
  auto queue = [&](bool open, int k) {
    const unsigned m = __ballot_sync(FULL, open);
    if (open) w.open[nopen + __popc(m & lt_mask)] = (unsigned char)k;
    nopen += __popc(m);
  };
  for (bool last = false; !last;) {
    // this warp's share of what is left, a few queries at least
    const float fair = (float)(n - seen) * share;
    const int want = max(fair < (float)kPortion ? (int)fair + 1 : kPortion, least);
    unsigned long long a = 0;
    if (lane == 0) a = atomicAdd(counter, (unsigned long long)want);
    const int64_t q0 = (int64_t)__shfl_sync(FULL, a, 0);
    last = q0 >= n;
    seen = q0 + want;
    const int cnt = last ? 0 : (int)(n - q0 < want ? n - q0 : want);
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
          const int k = w.list[slot];
          if (end != kContinue) {
            if (end == kConverged) evaluate_dist2<P, Q>(cx, tx, ty, tz, sd.u, sd.v, sd.hu, sd.hv, dist);
            const double r = sqrt(dist);
            if (end == kConverged && in_domain64(cx, sd.u, sd.v, dist) && r < max_edge) answer(q0 + k, 0, sd.u, sd.v, r);
            else open = true;
          }
          queue(open, k);
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
        if (k < total) {
          const int64_t q = q0 + w.list[k];
          open = true;
          if (w.end[k] == kConverged) {
            double u = w.ru[k], v = w.rv[k], r;
            if (final64<P, Q>(cx, ev, Pq[3 * q], Pq[3 * q + 1], Pq[3 * q + 2], u, v, r) && r < max_edge) {
              answer(q, 0, u, v, r);
              open = false;
            }
          }
        }
        queue(open, k < total ? w.list[k] : 0);
      }
    }
    __syncwarp();
    // ---- the open queries' trees, a full warp's worth at a time
    for (;;) {
      const int more = min(nopen, 32 - nrest);
      nopen -= more;
      if (lane < more) w.rest[nrest + lane] = q0 + w.open[nopen + lane];
      nrest += more;
      __syncwarp();
      if (nrest < 32 && !(last && nrest > 0)) break;
      if (root_type < 0) {
        const double root[4] = {s.dom_u0, s.dom_v0, s.dom_u1, s.dom_v1};
        root_type = split_type_fast<MODE>(s, ev, root, max_edge);
      }
      quadtree_search<P, Q, MODE>(s, sm, w, qtbox, Pq, w.rest, nrest, root_type, max_edge, uv_out, st_out, res_out);
      nrest = 0;
    }
  }
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
  // final steps costs as much for one), at most the resident ones (8 / 16 / 32 / 64: 30,000 points, mixed,
  // 8x8 surface 323 / 320 / 292 / 384 us, 64x64 735 / 749 / 730 / 966; the same on 9,000 and on 262,147)
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
