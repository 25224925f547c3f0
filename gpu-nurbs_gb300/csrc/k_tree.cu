// Stage c: 2-level subdivision tree of AABBs and candidate selection (K3 tree_build), and the
// projection's and the quadtree inversion's culling data.
//
// Replaces, per level, the reference's chain GetPoints -> 3x GetSecondDerivatives ->
// 3x Max_Sequential_Addressing_Shared -> TightBoundingBox (src/kernel/kernel.cu:375-431,
// 544-621, 707-733; driven by src/main.cu:280-309): 9x9 samples per node, second-derivative maxima,
// box inflation K = (M1 + 2 M2 + M3) sqrt(3) / (8 (8g)^2), clip to the parent box, flatness test
// NeedDivide (kernel.cu:859-878).
//
// Two launches.  k_nodes: one CTA per node evaluates the node's samples and reduces them to the
// unclipped box, the unclipped normal box and the control-point box, in nodebox; a node's samples do
// not depend on its parent, so both levels run at once (the quadtree boxes are further CTAs of the same
// launch).  k_nodes_finish: a warp per node clips to the root and writes the records.  Only final values
// are written to what the queries read, so a rebuild, which repeats them, does not disturb queries on
// other streams.
//
// What bounds it: FP64 arithmetic in the reference's order.  An FP64 instruction of a warp takes 64
// clocks here whatever its active lanes, so the build is a question of how few of them follow one
// another on one scheduler.  Hence four lanes per sample, one per homogeneous component; the
// matrix-vector products are shared by all derivatives (4 v-contractions and one u-contraction
// instead of 15) and nothing else is done twice; the components meet by shuffles in the quotient
// rule and the cross products; minima and maxima of control points compare integers.
// Measured on a bicubic 64x64 net: 102 + 10 us, against 817 us in five launches of one thread per
// sample with 9-thread reductions (and a serial scan of the control points' boxes); the whole
// conversion through the Python binding with all results read back 1352 -> 683 us (515
// since the host side's copies are fewer).
//
// Compiled with --fmad=false and evaluated in the order of operations of gnurbs::exact (power
// vectors by running product, sums from 0 in ascending order), so boxes and Divided flags are
// bit-identical to the reference's FP64 math, and the cones to the oracle's.
#include "nurbs_internal.h"
#include "nurbs_math.cuh"

namespace gnurbs {

__device__ __forceinline__ bool need_divide(const TreeNodeDev& n) {  // kernel.cu:859-878
  double dx = n.rt[0] - n.lb[0], dy = n.rt[1] - n.lb[1], dz = n.rt[2] - n.lb[2], t;
  if (dx > dy) { t = dx; dx = dy; dy = t; }
  if (dx > dz) { t = dx; dx = dz; dz = t; }
  if ((dx < 0.5 * dy) && (dx < 0.5 * dz)) return false;
  return true;
}

constexpr int kSamples = kPts * kPts;
constexpr int kNodeThreads = 352;  // 4 lanes per sample, whole warps
constexpr int kNodeWarps = kNodeThreads / 32;

struct NodeSmem {
  double U[kSamples][4][kMaxDegree + 1], V[kSamples][4][kMaxDegree + 1];  // power vectors and derivatives
  double spanU[kSamples], spanV[kSamples];
  int span[kSamples];
};
struct NodeReduce {  // per warp, by component lane: maxima and minima of S and N; M and N_uu.. maxima
  double smax[3], smin[3], m[3], nmax[3], nmin[3], nm[3];
  long long hull[6];
};

// Maximum (or minimum) over the warp's samples of lanes of one component (lanes 4 apart), with the
// sequential scan's result: a NaN is skipped, and of equal values the first sample's stays.
template <bool MAX>
__device__ __forceinline__ double pick(double first, double later) {
  if (isnan(first)) return later;
  return MAX ? (first < later ? later : first) : (first > later ? later : first);
}
template <bool MAX>
__device__ __forceinline__ double warp_pick(double x) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) {
    const double y = __shfl_xor_sync(0xffffffffu, x, o);
    x = (lane & o) ? pick<MAX>(y, x) : pick<MAX>(x, y);
  }
  return x;
}
__device__ __forceinline__ double shfl(double x, int src) { return __shfl_sync(0xffffffffu, x, src); }

// Control points a0..a1 x b0..b1: total keys of their minima (0..2) and maxima (3..5) over the
// elements t, t + stride, ..., reduced over the warp.
__device__ __forceinline__ void hull_of(const SurfDev& s, int a0, int a1, int b0, int b1, int t, int stride,
                                        long long h[6]) {
  const int nb = b1 - b0 + 1;
  const int64_t cnt = (int64_t)(a1 - a0 + 1) * nb;
  for (int c = 0; c < 3; ++c) {
    h[c] = 0x7fffffffffffffffll;
    h[3 + c] = -0x7fffffffffffffffll - 1;
  }
  for (int64_t e = t; e < cnt; e += stride) {
    const int row = (int)(e / nb), col = (int)(e - (int64_t)row * nb);
    const double* x = s.cps + 3 * ((size_t)(a0 + row) * s.nv + (b0 + col));
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const long long k = fast::total_key(x[c]);
      h[c] = k < h[c] ? k : h[c];
      h[3 + c] = k > h[3 + c] ? k : h[3 + c];
    }
  }
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const long long lo = __shfl_xor_sync(0xffffffffu, h[c], o), hi = __shfl_xor_sync(0xffffffffu, h[3 + c], o);
      h[c] = lo < h[c] ? lo : h[c];
      h[3 + c] = hi > h[3 + c] ? hi : h[3 + c];
    }
}

// The samples of node k (0: root, 1 + bx*8 + by: its children): its unclipped box into nodebox; CONES:
// also its unclipped normal box and control-point box there, and the lattice points.
//
// Normal cones (the projection's culling data): the normal N = Su x Sv and its second derivatives at
// the same samples, the normal box widened by the box tree's bound K applied to N.
template <bool CONES>
__device__ __forceinline__ void node_samples(const SurfDev& s, int k) {
  __shared__ NodeSmem sm;
  __shared__ NodeReduce red[kNodeWarps];
  __shared__ double first_m[6];  // sample 0's M1..M3 and N_uu, N_uv, N_vv maxima (a NaN there stays)
  __shared__ double first_s[3], first_n[3];
  const unsigned g = k == 0 ? 1u : (unsigned)kGap;
  const unsigned bx = k == 0 ? 0u : (unsigned)(k - 1) / kGap, by = k == 0 ? 0u : (unsigned)(k - 1) % kGap;
  const double uunit = k == 0 ? 1.0 : 1.0 / kGap;  // 1/g: kernel.cu:604-605
  const int p = s.p, q = s.q, k1 = p + 1, k2 = q + 1, k12 = k1 * k2;
  if (threadIdx.x < kSamples) {
    const int t = threadIdx.x, tx = t / kPts, ty = t % kPts;
    // GetPoints / GetSecondDerivatives sample (kernel.cu:383-388, 412-417)
    const double base_unit = uunit;
    const double unit = base_unit * (1.0 / kGap);  // exact: kGap is a power of two
    const double base_u = base_unit * bx, base_v = base_unit * by;
    const double p1 = base_u + tx * unit, p2 = base_v + ty * unit;
    const int su = exact::find_seg(s.bu, s.ns_u, p1);
    const int sv = exact::find_seg(s.bv, s.ns_v, p2);
    const double du = s.bu[su + 1] - s.bu[su], dv = s.bv[sv + 1] - s.bv[sv];
    const double u = (p1 - s.bu[su]) / du;
    const double v = (p2 - s.bv[sv]) / dv;
    sm.spanU[t] = s.range_u / du;
    sm.spanV[t] = s.range_v / dv;
    sm.span[t] = su * s.ns_v + sv;
    exact::vectors_k(u, k1, sm.U[t][0], sm.U[t][1], sm.U[t][2], sm.U[t][3]);
    exact::vectors_k(v, k2, sm.V[t][0], sm.V[t][1], sm.V[t][2], sm.V[t][3]);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = min((int)(threadIdx.x >> 2), kSamples - 1), c = lane & 3, w0 = lane & ~3;
  const bool real = (int)(threadIdx.x >> 2) < kSamples;
  // ---- this lane's component of R and its local derivatives
  const double* M = s.m64 + (size_t)sm.span[t] * k12 * 4 + c;
  double R = 0, Ru = 0, Ruu = 0, Ruuu = 0, Rv = 0, Ruv = 0, Ruuv = 0, Ruvv = 0, Rvvv = 0;
  double ucol[kMaxDegree + 1];  // u-contraction, per power of v
#pragma unroll
  for (int b = 0; b <= kMaxDegree; ++b) ucol[b] = 0;
  for (int a = 0; a < k1; ++a) {
    double t0 = 0, t1 = 0, t2 = 0, t3 = 0;
    const double U0 = sm.U[t][0][a], U1 = sm.U[t][1][a], U2 = sm.U[t][2][a];
#pragma unroll
    for (int b = 0; b <= kMaxDegree; ++b) {
      if (b < k2) {
        const double m = M[(a * k2 + b) * 4];
        t0 += m * sm.V[t][0][b];
        t1 += m * sm.V[t][1][b];
        if (CONES) {
          t2 += m * sm.V[t][2][b];
          t3 += m * sm.V[t][3][b];
        }
        ucol[b] += U0 * m;
      }
    }
    R += U0 * t0;
    Ru += U1 * t0;
    Ruu += U2 * t0;
    Rv += U0 * t1;
    Ruv += U1 * t1;
    if (CONES) {
      Ruuu += sm.U[t][3][a] * t0;
      Ruuv += U2 * t1;
      Ruvv += U1 * t2;
      Rvvv += U0 * t3;
    }
  }
  double Rv2 = 0, Rvv = 0;  // contracting u first (MatrixSurfaceDerivativeVV, Evaluate.cu:849-930)
#pragma unroll
  for (int b = 0; b <= kMaxDegree; ++b)
    if (b < k2) {
      Rv2 += sm.V[t][1][b] * ucol[b];
      Rvv += sm.V[t][2][b] * ucol[b];
    }
  const double su = sm.spanU[t], sv = sm.spanV[t];
  const double h = shfl(R, w0 + 3);
  // ---- old-style second derivatives (exact::der_uu, der_uv, der_vv), this lane's coordinate
  {
    const double hu = shfl(Ru, w0 + 3), huu = shfl(Ruu, w0 + 3), hv = shfl(Rv, w0 + 3), huv = shfl(Ruv, w0 + 3);
    const double hv2 = shfl(Rv2, w0 + 3), hvv = shfl(Rvv, w0 + 3);
    const double h2 = exact::sq(h), h3 = exact::cube(h);
    const double u1 = (2 * exact::sq(hu) / h3) - (huu / h2), u2 = -hu / h2;
    const double uu = ((R * u1 + (2 * Ru) * u2) + Ruu / h) * su * su;
    const double uv = ((((Ruv * h - hv * Ru) - Rv * hu) - R * huv) / h2 + ((2 * R) * hu * hv) / h3) * su * sv;
    const double v1 = (2 * exact::sq(hv2) / h3) - (hvv / h2), v2 = -hv2 / h2;
    const double vv = ((R * v1 + (2 * Rv2) * v2) + Rvv / h) * sv * sv;
    const double S = R / h;
    const double none = __longlong_as_double(0x7ff8000000000000ll);
    double m1 = fmax(fabs(uu), fmax(fabs(shfl(uu, w0 + 1)), fabs(shfl(uu, w0 + 2))));  // kernel.cu:399
    double m2 = fmax(fabs(uv), fmax(fabs(shfl(uv, w0 + 1)), fabs(shfl(uv, w0 + 2))));
    double m3 = fmax(fabs(vv), fmax(fabs(shfl(vv, w0 + 1)), fabs(shfl(vv, w0 + 2))));
    if (threadIdx.x == 0) {
      first_m[0] = m1;
      first_m[1] = m2;
      first_m[2] = m3;
    }
    if (threadIdx.x < 3) first_s[c] = S;
    const double x = real ? S : none;
    const double hi = warp_pick<true>(x), lo = warp_pick<false>(x);
    m1 = warp_pick<true>(real ? m1 : none);
    m2 = warp_pick<true>(real ? m2 : none);
    m3 = warp_pick<true>(real ? m3 : none);
    if (lane < 3) {
      red[warp].smax[c] = hi;
      red[warp].smin[c] = lo;
    }
    if (lane == 0) {
      red[warp].m[0] = m1;
      red[warp].m[1] = m2;
      red[warp].m[2] = m3;
    }
  }
  if (CONES) {
    // ---- derivatives to third order by the new-style quotient rule (exact::ders3), then N and its
    // second derivatives (exact::normal_ders2), this lane's coordinate
    const double r1 = Ru * su, r2 = Rv * sv, r3 = (Ruu * su) * su, r4 = (Ruv * su) * sv, r5 = (Rvv * sv) * sv;
    const double r6 = ((Ruuu * su) * su) * su, r7 = ((Ruuv * su) * su) * sv, r8 = ((Ruvv * su) * sv) * sv,
                 r9 = ((Rvvv * sv) * sv) * sv;
    const double hu = shfl(r1, w0 + 3), hv = shfl(r2, w0 + 3), huu = shfl(r3, w0 + 3), huv = shfl(r4, w0 + 3),
                 hvv = shfl(r5, w0 + 3), huuu = shfl(r6, w0 + 3), huuv = shfl(r7, w0 + 3), huvv = shfl(r8, w0 + 3),
                 hvvv = shfl(r9, w0 + 3);
    const double o0 = R / h;
    const double o1 = (r1 - hu * o0) / h;
    const double o2 = (r2 - hv * o0) / h;
    const double o3 = ((r3 - 2 * hu * o1) - huu * o0) / h;
    const double o4 = (((r4 - hv * o1) - hu * o2) - huv * o0) / h;
    const double o5 = ((r5 - 2 * hv * o2) - hvv * o0) / h;
    const double o6 = (((r6 - 3 * hu * o3) - 3 * huu * o1) - huuu * o0) / h;
    const double o7 = (((((r7 - hv * o3) - 2 * hu * o4) - 2 * huv * o1) - huu * o2) - huuv * o0) / h;
    const double o8 = (((((r8 - hu * o5) - 2 * hv * o4) - 2 * huv * o2) - hvv * o1) - huvv * o0) / h;
    const double o9 = (((r9 - 3 * hv * o5) - 3 * hvv * o2) - hvvv * o0) / h;
    if (real && c < 3) s.lattice[(size_t)(k * kSamples + t) * 3 + c] = (float)(o0 - s.org[c]);
    // coordinates (c+1)%3 and (c+2)%3 of a vector from the neighbouring lanes
    const int l1 = w0 + (c + 1) % 3, l2 = w0 + (c + 2) % 3;
    const double a1 = shfl(o1, l1), a2 = shfl(o2, l1), a3 = shfl(o3, l1), a4 = shfl(o4, l1), a5 = shfl(o5, l1),
                 a6 = shfl(o6, l1), a7 = shfl(o7, l1), a8 = shfl(o8, l1), a9 = shfl(o9, l1);
    const double b1 = shfl(o1, l2), b2 = shfl(o2, l2), b3 = shfl(o3, l2), b4 = shfl(o4, l2), b5 = shfl(o5, l2),
                 b6 = shfl(o6, l2), b7 = shfl(o7, l2), b8 = shfl(o8, l2), b9 = shfl(o9, l2);
    const double n0 = a1 * b2 - b1 * a2;
    const double n1 = ((a6 * b2 - b6 * a2) + 2 * (a3 * b4 - b3 * a4)) + (a1 * b7 - b1 * a7);
    const double n2 = (((a7 * b2 - b7 * a2) + (a3 * b5 - b3 * a5)) + (a4 * b4 - b4 * a4)) + (a1 * b8 - b1 * a8);
    const double n3 = ((a8 * b2 - b8 * a2) + 2 * (a4 * b5 - b4 * a5)) + (a1 * b9 - b1 * a9);
    const double none = __longlong_as_double(0x7ff8000000000000ll);
    double m1 = fmax(fabs(n1), fmax(fabs(shfl(n1, w0 + 1)), fabs(shfl(n1, w0 + 2))));
    double m2 = fmax(fabs(n2), fmax(fabs(shfl(n2, w0 + 1)), fabs(shfl(n2, w0 + 2))));
    double m3 = fmax(fabs(n3), fmax(fabs(shfl(n3, w0 + 1)), fabs(shfl(n3, w0 + 2))));
    if (threadIdx.x == 0) {
      first_m[3] = m1;
      first_m[4] = m2;
      first_m[5] = m3;
    }
    if (threadIdx.x < 3) first_n[c] = n0;
    const double x = real ? n0 : none;
    const double hi = warp_pick<true>(x), lo = warp_pick<false>(x);
    m1 = warp_pick<true>(real ? m1 : none);
    m2 = warp_pick<true>(real ? m2 : none);
    m3 = warp_pick<true>(real ? m3 : none);
    // control points acting on the node's parameter rectangle (uv_lb, uv_rt of the tree node)
    const double ul = bx * uunit, ur = (bx + 1) * uunit, vl = by * uunit, vr = (by + 1) * uunit;
    int i0 = exact::find_seg(s.bu, s.ns_u, ul), i1 = exact::find_seg(s.bu, s.ns_u, ur);
    int j0 = exact::find_seg(s.bv, s.ns_v, vl), j1 = exact::find_seg(s.bv, s.ns_v, vr);
    if (i1 > i0 && s.bu[i1] >= ur) --i1;  // the span starting at the right end
    if (j1 > j0 && s.bv[j1] >= vr) --j1;
    long long hull[6];
    hull_of(s, s.knot_u[i0] - p, s.knot_u[i1], s.knot_v[j0] - q, s.knot_v[j1], threadIdx.x, blockDim.x,
            hull);
    if (lane < 3) {
      red[warp].nmax[c] = hi;
      red[warp].nmin[c] = lo;
    }
    if (lane == 0) {
      red[warp].nm[0] = m1;
      red[warp].nm[1] = m2;
      red[warp].nm[2] = m3;
      for (int j = 0; j < 6; ++j) red[warp].hull[j] = hull[j];
    }
  }
  __syncthreads();
  // ---- across the warps, in sample order: lanes 0..5 the M maxima, 6..8 / 9..11 max / min of S,
  // 12..17 the same of N, 18..23 the control-point box
  if (warp == 0) {
    double acc = 0;
    const int j = lane % 3;
    if (lane < 18) {
      auto val = [&](int w) {
        if (lane < 3) return red[w].m[j];
        if (lane < 6) return red[w].nm[j];
        if (lane < 9) return red[w].smax[j];
        if (lane < 12) return red[w].smin[j];
        return lane < 15 ? red[w].nmax[j] : red[w].nmin[j];
      };
      const bool mn = (lane >= 9 && lane < 12) || lane >= 15;
      if (CONES || lane < 3 || (lane >= 6 && lane < 12)) {
        acc = val(0);
        for (int w = 1; w < kNodeWarps; ++w) acc = mn ? pick<false>(acc, val(w)) : pick<true>(acc, val(w));
        const double f = lane < 6 ? first_m[lane] : (lane < 12 ? first_s[j] : first_n[j]);
        if (isnan(f)) acc = f;  // the scan starts from sample 0 and a comparison with NaN never replaces it
      }
    } else if (CONES && lane < 24) {
      long long hk = red[0].hull[lane - 18];
      for (int w = 1; w < kNodeWarps; ++w) {
        const long long o = red[w].hull[lane - 18];
        hk = lane < 21 ? (o < hk ? o : hk) : (o > hk ? o : hk);
      }
      acc = fast::key_value(hk);
    }
    const unsigned den = 8u * kGap * g * kGap * g;
    // sqrt(3): kernel.cu:574
    const double K = (shfl(acc, 0) + 2 * shfl(acc, 1) + shfl(acc, 2)) * 1.7320508075688772 / den;
    const double KN = (shfl(acc, 3) + 2 * shfl(acc, 4) + shfl(acc, 5)) * 1.7320508075688772 / den;
    double* box = s.nodebox + 6 * k;
    if (lane >= 6 && lane < 9) box[3 + j] = acc + K;
    if (lane >= 9 && lane < 12) box[j] = acc - K;
    if (CONES) {
      double *nbox = box + 6 * kTreeNodes, *hull = nbox + 6 * kTreeNodes;
      if (lane >= 12 && lane < 15) nbox[3 + j] = acc + KN;
      if (lane >= 15 && lane < 18) nbox[j] = acc - KN;
      if (lane >= 18 && lane < 24) hull[lane - 18] = acc;
    }
  }
}

__device__ __forceinline__ float round_down(double x) { return __double2float_rd(x); }
__device__ __forceinline__ float round_up(double x) { return __double2float_ru(x); }

// One warp per node: the box clipped to the root's, the flags, and with CONES the culling record:
// the node's bound box (its box intersected with the box of the control points acting on its
// parameter rectangle) and the cone around the centre of the clipped normal box, in the oracle's
// order of operations (record layout: nurbs_internal.h).
template <bool CONES>
__device__ __forceinline__ void node_finish(const SurfDev& s, int k) {
  const int lane = threadIdx.x & 31;
  const unsigned bx = k == 0 ? 0u : (unsigned)(k - 1) / kGap, by = k == 0 ? 0u : (unsigned)(k - 1) % kGap;
  const double uunit = k == 0 ? 1.0 : 1.0 / kGap;
  const double *box0 = s.nodebox, *nbox0 = box0 + 6 * kTreeNodes, *hull0 = nbox0 + 6 * kTreeNodes;  // the root's
  TreeNodeDev root, n;
  for (int c = 0; c < 3; ++c) {
    root.lb[c] = box0[c];
    root.rt[c] = box0[3 + c];
    n.lb[c] = box0[6 * k + c];
    n.rt[c] = box0[6 * k + 3 + c];
  }
  n.uv_lb[0] = bx * uunit;
  n.uv_lb[1] = by * uunit;
  n.uv_rt[0] = (bx + 1) * uunit;
  n.uv_rt[1] = (by + 1) * uunit;
  const bool built = k == 0 || need_divide(root);  // children of a flat root are not built
  double nb[6] = {0, 0, 0, 0, 0, 0}, hb[6] = {0, 0, 0, 0, 0, 0};
  if (CONES)
    for (int c = 0; c < 6; ++c) {
      nb[c] = nbox0[6 * k + c];
      hb[c] = hull0[6 * k + c];
    }
  if (k > 0)
    for (int c = 0; c < 3; ++c) {  // min/max(TreeNode) against the parent (kernel.cu:606-611, 885-901)
      n.rt[c] = fmin(n.rt[c], root.rt[c]);
      n.lb[c] = fmax(n.lb[c], root.lb[c]);
      if (CONES) {
        nb[c] = fmax(nb[c], nbox0[c]);
        nb[3 + c] = fmin(nb[3 + c], nbox0[3 + c]);
      }
    }
  if (lane == 0) {
    if (!built) n = TreeNodeDev{};
    s.tree[k] = n;
    s.divided[k] = built && need_divide(n) ? 1 : 0;
    s.built[k] = built ? 1 : 0;
  }
  if (!CONES) return;
  float* rec = s.cone + kConeStride * k;
  if (!built) {
    if (lane < 6) s.nbox[6 * k + lane] = 0;
    if (lane < kConeStride) rec[lane] = 0;
    return;
  }
  if (lane == 0)
    for (int c = 0; c < 6; ++c) s.nbox[6 * k + c] = nb[c];
  // the node's own box where it is narrower
  double xb[6];
  bool empty = false;
  for (int c = 0; c < 3; ++c) {
    xb[c] = hb[c] > n.lb[c] ? hb[c] : n.lb[c];
    xb[3 + c] = hb[3 + c] < n.rt[c] ? hb[3 + c] : n.rt[c];
    empty = empty || xb[c] > xb[3 + c];
  }
  double bb[6];
  for (int c = 0; c < 6; ++c) bb[c] = empty ? hb[c] : xb[c];
  // cosine between the normal box's centre and its corner `lane`
  const double m[3] = {(nb[0] + nb[3]) / 2, (nb[1] + nb[4]) / 2, (nb[2] + nb[5]) / 2};
  const double mm = sqrt(m[0] * m[0] + m[1] * m[1] + m[2] * m[2]);
  const int i = lane >> 2 & 1, j = lane >> 1 & 1, l = lane & 1;
  const double co[3] = {i ? nb[3] : nb[0], j ? nb[4] : nb[1], l ? nb[5] : nb[2]};
  const double cc = (m[0] * co[0] + m[1] * co[1] + m[2] * co[2]) /
                    (mm * sqrt(co[0] * co[0] + co[1] * co[1] + co[2] * co[2]));
  double cmin = 1;
  for (int e = 0; e < 8; ++e) {
    const double x = shfl(cc, e);
    cmin = cmin < x ? cmin : x;
  }
  if (lane != 0) return;
  double ctr[3], hh[3];
  for (int c = 0; c < 3; ++c) {
    ctr[c] = (bb[c] + bb[3 + c]) / 2;
    hh[c] = (bb[3 + c] - bb[c]) / 2;
  }
  const double r = sqrt(hh[0] * hh[0] + hh[1] * hh[1] + hh[2] * hh[2]);
  const double cm = fmax(fabs(ctr[0] - s.org[0]), fmax(fabs(ctr[1] - s.org[1]), fabs(ctr[2] - s.org[2])));
  for (int c = 0; c < 3; ++c) rec[c] = (float)(ctr[c] - s.org[c]);
  rec[3] = (float)(r * (1 + 0x1p-20) + cm * 0x1p-20);
  bool all = nb[0] > nb[3] || nb[1] > nb[4] || nb[2] > nb[5];
  all = all || (nb[0] <= 0 && nb[3] >= 0 && nb[1] <= 0 && nb[4] >= 0 && nb[2] <= 0 && nb[5] >= 0);
  double cosA = 0, sinA = 1, ax[3] = {0, 0, 1};
  if (!all && cmin > 0) {
    const double sn = sqrt(fmax(0.0, 1 - cmin * cmin));
    const double tt = 0x1p-11, cd = (1 - tt * tt) / (1 + tt * tt), sd = (2 * tt) / (1 + tt * tt);
    const double ca = cmin * cd - sn * sd, sa = sn * cd + cmin * sd;
    if (ca > 0) {
      cosA = ca;
      sinA = sa;
      ax[0] = m[0] / mm;
      ax[1] = m[1] / mm;
      ax[2] = m[2] / mm;
    }
  }
  for (int c = 0; c < 3; ++c) rec[4 + c] = (float)ax[c];
  rec[7] = (float)cosA;
  rec[8] = (float)sinA;
  for (int c = 0; c < 3; ++c) {
    rec[9 + c] = round_down(bb[c] - s.org[c]);
    rec[12 + c] = round_up(bb[3 + c] - s.org[c]);
  }
  for (int c = 15; c < kConeStride; ++c) rec[c] = 0;
}

// Control-point box of one of the quadtree inversion's precomputed nodes (kQuadtreeDepth levels of
// square children: depth d, u index a, v index b, code = (4^d - 1) / 3 + a 2^d + b), the node's
// rectangle by the search's own midpoint splits, the control points of BoundingBoxCheck's range: the
// part of threads t, t + stride, ..., reduced over the warp.
__device__ __forceinline__ void quadtree_box(const SurfDev& s, int code, int t, int stride, long long h[6]) {
  int d = 0, base = 0;
  while (code >= base + (1 << (2 * d))) base += 1 << (2 * d++);
  const int a = (code - base) >> d, b = (code - base) & ((1 << d) - 1);
  double nd[4] = {s.dom_u0, s.dom_v0, s.dom_u1, s.dom_v1};
  for (int l = d - 1; l >= 0; --l) {
    const double mu = (nd[0] + nd[2]) / 2, mv = (nd[1] + nd[3]) / 2;
    if ((a >> l) & 1) nd[0] = mu; else nd[2] = mu;
    if ((b >> l) & 1) nd[1] = mv; else nd[3] = mv;
  }
  auto knot = [](const int* idx_of, const double* br, int ns, double x) { return idx_of[exact::find_seg(br, ns, x)]; };
  hull_of(s, knot(s.knot_u, s.bu, s.ns_u, nd[0]) - s.p, knot(s.knot_u, s.bu, s.ns_u, nd[2]),
          knot(s.knot_v, s.bv, s.ns_v, nd[1]) - s.q, knot(s.knot_v, s.bv, s.ns_v, nd[3]), t, stride, h);
}

constexpr int kQuadtreeLarge = 1 + 4 + 16;  // boxes of depth 0..2: a CTA each; the deeper ones a warp each
__device__ __forceinline__ void quadtree_box_cta(const SurfDev& s, int code) {
  long long h[6];
  quadtree_box(s, code, threadIdx.x, blockDim.x, h);
  __shared__ long long red[kNodeWarps][6];
  if ((threadIdx.x & 31) == 0)
    for (int c = 0; c < 6; ++c) red[threadIdx.x >> 5][c] = h[c];
  __syncthreads();
  if (threadIdx.x < 6) {
    const int c = threadIdx.x;
    long long k = red[0][c];
    for (int w = 1; w < kNodeWarps; ++w) k = c < 3 ? min(k, red[w][c]) : max(k, red[w][c]);
    s.qtbox[6 * code + c] = fast::key_value(k);
  }
}
__device__ __forceinline__ void quadtree_box_warp(const SurfDev& s, int code) {
  if (code >= kQuadtreeBoxes) return;
  long long h[6];
  quadtree_box(s, code, threadIdx.x & 31, 32, h);
  if ((threadIdx.x & 31) == 0)
    for (int c = 0; c < 6; ++c) s.qtbox[6 * code + c] = fast::key_value(h[c]);
}

__global__ void __launch_bounds__(kNodeThreads) k_nodes(SurfDev s) {
  const int b = blockIdx.x;
  if (b < kTreeNodes) node_samples<true>(s, b);
  else if (b < kTreeNodes + kQuadtreeLarge) quadtree_box_cta(s, b - kTreeNodes);
  else quadtree_box_warp(s, kQuadtreeLarge + (b - kTreeNodes - kQuadtreeLarge) * kNodeWarps + (threadIdx.x >> 5));
}
__global__ void __launch_bounds__(32) k_nodes_finish(SurfDev s) { node_finish<true>(s, blockIdx.x); }

// Many surfaces (boxes only): blockIdx.y selects the surface of ids[] in the device table.
__global__ void __launch_bounds__(kNodeThreads) k_nodes_batched(const SurfDev* __restrict__ table,
                                                                const int* __restrict__ ids) {
  const SurfDev s = table[ids[blockIdx.y]];
  node_samples<false>(s, blockIdx.x);
}
__global__ void __launch_bounds__(32) k_nodes_finish_batched(const SurfDev* __restrict__ table,
                                                             const int* __restrict__ ids) {
  const SurfDev s = table[ids[blockIdx.y]];
  node_finish<false>(s, blockIdx.x);
}

// NewInverse's scan (kernel.cu:456-457) over built nodes, NewBoundingBoxCheck (:466-469).
__global__ void k_candidates(SurfDev s, const double* __restrict__ P, int64_t n, int* __restrict__ list,
                             int* __restrict__ counts) {
  __shared__ double box[kTreeNodes][6];
  __shared__ unsigned char built[kTreeNodes];
  for (int k = threadIdx.x; k < kTreeNodes; k += blockDim.x) {
    built[k] = s.built[k];
    for (int c = 0; c < 3; ++c) {
      box[k][c] = s.tree[k].lb[c];
      box[k][3 + c] = s.tree[k].rt[c];
    }
  }
  __syncthreads();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double x = P[3 * i], y = P[3 * i + 1], z = P[3 * i + 2];
    int cnt = 0;
    for (int k = 0; k < kTreeNodes; ++k) {
      if (!built[k]) continue;
      if ((x >= box[k][0]) && (y >= box[k][1]) && (z >= box[k][2]) && (x <= box[k][3]) && (y <= box[k][4]) &&
          (z <= box[k][5]))
        list[i * kTreeNodes + cnt++] = k;
    }
    counts[i] = cnt;
  }
}

cudaError_t launch_nodes(const SurfDev& s, cudaStream_t st) {
  constexpr int small = (kQuadtreeBoxes - kQuadtreeLarge + kNodeWarps - 1) / kNodeWarps;
  k_nodes<<<kTreeNodes + kQuadtreeLarge + small, kNodeThreads, 0, st>>>(s);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_nodes_finish<<<kTreeNodes, 32, 0, st>>>(s);
  return cudaGetLastError();
}

cudaError_t launch_nodes_batched(const SurfDev* table, const int* ids, int count, cudaStream_t st) {
  for (int off = 0; off < count; off += 65535) {
    const int c = count - off < 65535 ? count - off : 65535;
    k_nodes_batched<<<dim3(kTreeNodes, c), kNodeThreads, 0, st>>>(table, ids + off);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_nodes_finish_batched<<<dim3(kTreeNodes, c), 32, 0, st>>>(table, ids + off);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_candidates(const SurfDev& s, const double* P, int64_t n, int* list, int* counts,
                              cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  int64_t blocks = (n + 255) / 256;
  if (blocks > 152 * 32) blocks = 152 * 32;
  k_candidates<<<(unsigned)blocks, 256, 0, st>>>(s, P, n, list, counts);
  return cudaGetLastError();
}

}  // namespace gnurbs
