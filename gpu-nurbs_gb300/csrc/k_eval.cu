// Stage b: batched evaluation of points and derivatives up to second order (K2 eval).
//
// Replaces MatrixSurfacePoint / MatrixSurfaceDerivative{U,V,UU,UV,VV}
// (src/NURBS/Evaluate.cu:159-227, 535-930) driven per point as EvaluateRandom does
// (:1023-1038).  The reference recontracts the span matrix once per requested quantity from
// local-memory arrays; here one thread per point (few FP64 points: four lanes, k_eval_few) streams
// the span's (p+1)(q+1) 4-vectors of coefficients once (256-bit loads, L1/L2-resident span table)
// through a Horner scheme that yields R and all its derivatives to the requested order together,
// then applies the quotient rule once.  Output is SoA, one coalesced streaming store per value.
//
// FP64 cost per point for p = q = 3: 60 / 112 / 152 FMAs for order 0 / 1 / 2 (the
// reference's formulation spends 80 / 176 / 288), plus one reciprocal.  FP64 is bound by that pipe,
// so the span search compares the breakpoints as integers (64x64 surface, S..Svv, 2^22 points 1768 ->
// 1675 us, S alone 599 -> 509).  FP32 on a parameter grid is bound by the latency of the chain (u, v) ->
// span -> coefficients, so the search starts from a lookup grid (3001x2001 points: 137 -> 123 us).
#include "nurbs_internal.h"
#include "nurbs_math.cuh"

namespace gnurbs {

template <typename T>
__device__ __forceinline__ void st_stream(T* p, T v) {
  __stcs(p, v);
}

template <typename T, int P, int Q, int ORDER>
__global__ void __launch_bounds__(256) k_eval(SurfDev s, const T* __restrict__ uv, int64_t n, unsigned mask,
                                              T* __restrict__ out) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    T u = uv[2 * i], v = uv[2 * i + 1];
    fast::SDer<T> d = fast::eval_point<T, P, Q, ORDER>(s, u, v);
    if constexpr (sizeof(T) == 4) {  // FP32 tables hold the surface relative to org
      d.S.x += s.org32[0];
      d.S.y += s.org32[1];
      d.S.z += s.org32[2];
    }
    int o = 0;
    auto put = [&](const v3<T>& a) {
      st_stream(out + (int64_t)(3 * o + 0) * n + i, a.x);
      st_stream(out + (int64_t)(3 * o + 1) * n + i, a.y);
      st_stream(out + (int64_t)(3 * o + 2) * n + i, a.z);
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
    if (ORDER >= 3) {
      if (mask & 64u) put(d.Suuu);
      if (mask & 128u) put(d.Suuv);
      if (mask & 256u) put(d.Suvv);
      if (mask & 512u) put(d.Svvv);
    }
  }
}

// FP64 evaluation of a few points: four lanes per point, one per homogeneous component, a warp of 8
// points per CTA.  An FP64 instruction takes a warp 64 clocks whatever its active lanes, so with fewer
// points than the GPU's FP64 pipes can take at once the time is the number of FP64 instructions one
// after the other in a warp: a quarter of the contraction's and a third of the quotient rule's this
// way.  Per component the same operations as k_eval's, so the same bits.
// (1,003 points, S, Su, Sv on the 8x8 surface: 12.0 -> 4.2 us of GPU time, 4,800 points 12.1 -> 4.9.)
template <int P, int Q, int ORDER>
__global__ void __launch_bounds__(32) k_eval_few(SurfDev s, const double* __restrict__ uv, int64_t n, unsigned mask,
                                                 double* __restrict__ out) {
  const int lane = threadIdx.x, c = lane & 3, w3 = lane | 3;
  const int64_t at = (int64_t)blockIdx.x * 8 + (lane >> 2);
  const int64_t i = at < n ? at : n - 1;
  const double u = uv[2 * i], v = uv[2 * i + 1];
  const int su = fast::find_seg(s.bu, s.ns_u, u), sv = fast::find_seg(s.bv, s.ns_v, v);
  const double idu = __ldg(s.inv_du + su), idv = __ldg(s.inv_dv + sv);
  const double lu = (u - __ldg(s.bu + su)) * idu, lv = (v - __ldg(s.bv + sv)) * idv;
  const int pp = P > 0 ? P : s.p, qq = Q > 0 ? Q : s.q, k2 = qq + 1;
  const double* m = s.m64 + (size_t)(su * s.ns_v + sv) * (pp + 1) * k2 * 4 + c;
  fast::HornerOne<ORDER> colR;
  fast::HornerOne<(ORDER >= 1 ? ORDER - 1 : 0)> colV;
  fast::HornerOne<(ORDER >= 2 ? ORDER - 2 : 0)> colVV;
#pragma unroll
  for (int a = P > 0 ? P : kMaxDegree; a >= 0; --a) {
    if (P == 0 && a > pp) continue;
    fast::HornerOne<ORDER> row;
#pragma unroll
    for (int b = Q > 0 ? Q : kMaxDegree; b >= 0; --b) {
      if (Q == 0 && b > qq) continue;
      row.push(__ldg(m + 4 * (a * k2 + b)), lv);
    }
    colR.push(row.p, lu);
    if (ORDER >= 1) colV.push(row.dp, lu);
    if (ORDER >= 2) colVV.push(row.ddp, lu);
  }
  auto w_of = [&](double x) { return __shfl_sync(0xffffffffu, x, w3); };
  const double ih = fast::rcp<false>(w_of(colR.p));
  const double S = colR.p * ih;
  int o = 0;
  auto put = [&](double x) {
    if (c < 3 && at < n) st_stream(out + (int64_t)(3 * o + c) * n + i, x);
    ++o;
  };
  if (mask & 1u) put(S);
  if constexpr (ORDER >= 1) {
    const double scu = s.range_u * idu, scv = s.range_v * idv;
    const double hu = w_of(colR.dp), hv = w_of(colV.p);
    const double Au = fast::mad(-hu, S, colR.dp) * ih, Av = fast::mad(-hv, S, colV.p) * ih;
    if (mask & 2u) put(Au * scu);
    if (mask & 4u) put(Av * scv);
    if constexpr (ORDER >= 2) {
      const double Ruu = 2.0 * colR.ddp, Ruv = colV.dp, Rvv = 2.0 * colVV.p;
      const double huu = w_of(Ruu), huv = w_of(Ruv), hvv = w_of(Rvv), hu2 = 2.0 * hu, hv2 = 2.0 * hv;
      const double Auu = fast::mad(-huu, S, fast::mad(-hu2, Au, Ruu)) * ih;
      const double Auv = fast::mad(-huv, S, fast::mad(-hv, Au, fast::mad(-hu, Av, Ruv))) * ih;
      const double Avv = fast::mad(-hvv, S, fast::mad(-hv2, Av, Rvv)) * ih;
      if (mask & 8u) put(Auu * (scu * scu));
      if (mask & 16u) put(Auv * (scu * scv));
      if (mask & 32u) put(Avv * (scv * scv));
    }
  }
}

// Surface normal N = Su x Sv (not normalised, as the reference's TrueNormal, Evaluate.cu:
// 1111-1117) and its first and second derivatives, the latter as the reference's
// SurfaceNormalDerivative{UU,UV,VV} (Evaluate.cu:1125-1135) with correct third derivatives:
//   Nu = Suu x Sv + Su x Suv,  Nv = Suv x Sv + Su x Svv,
//   Nuu = Suuu x Sv + 2 Suu x Suv + Su x Suuv,  Nuv = Suuv x Sv + Suu x Svv + Su x Suvv,
//   Nvv = Suvv x Sv + 2 Suv x Svv + Su x Svvv.
__device__ __forceinline__ v3<double> cross(const v3<double>& a, const v3<double>& b) {
  return {fast::mad(a.y, b.z, -(a.z * b.y)), fast::mad(a.z, b.x, -(a.x * b.z)), fast::mad(a.x, b.y, -(a.y * b.x))};
}
__device__ __forceinline__ v3<double> add3(const v3<double>& a, const v3<double>& b, double sb, const v3<double>& c) {
  return {fast::mad(sb, b.x, a.x) + c.x, fast::mad(sb, b.y, a.y) + c.y, fast::mad(sb, b.z, a.z) + c.z};
}

template <int P, int Q, int ORDER>
__global__ void __launch_bounds__(256) k_eval_normal(SurfDev s, const double* __restrict__ uv, int64_t n,
                                                     unsigned mask, double* __restrict__ out) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const fast::SDer<double> d = fast::eval_point<double, P, Q, ORDER>(s, uv[2 * i], uv[2 * i + 1]);
    int o = 0;
    auto put = [&](const v3<double>& a) {
      st_stream(out + (int64_t)(3 * o + 0) * n + i, a.x);
      st_stream(out + (int64_t)(3 * o + 1) * n + i, a.y);
      st_stream(out + (int64_t)(3 * o + 2) * n + i, a.z);
      ++o;
    };
    if (mask & 1u) put(cross(d.Su, d.Sv));
    if (ORDER >= 2) {
      if (mask & 2u) put(add3(cross(d.Suu, d.Sv), cross(d.Su, d.Suv), 1.0, {0, 0, 0}));
      if (mask & 4u) put(add3(cross(d.Suv, d.Sv), cross(d.Su, d.Svv), 1.0, {0, 0, 0}));
    }
    if (ORDER >= 3) {
      if (mask & 8u) put(add3(cross(d.Suuu, d.Sv), cross(d.Suu, d.Suv), 2.0, cross(d.Su, d.Suuv)));
      if (mask & 16u) put(add3(cross(d.Suuv, d.Sv), cross(d.Suu, d.Svv), 1.0, cross(d.Su, d.Suvv)));
      if (mask & 32u) put(add3(cross(d.Suvv, d.Sv), cross(d.Suv, d.Svv), 2.0, cross(d.Su, d.Svvv)));
    }
  }
}

static int order_of(unsigned mask) {
  if (mask & (64u | 128u | 256u | 512u)) return 3;
  if (mask & (8u | 16u | 32u)) return 2;
  if (mask & (2u | 4u)) return 1;
  return 0;
}

template <typename T, int P, int Q>
static cudaError_t launch_pq(const SurfDev& s, const T* uv, int64_t n, unsigned mask, T* out, cudaStream_t st) {
  int threads = 256;
  if constexpr (sizeof(T) == 8) {
    // four lanes per point while that leaves at most one warp per scheduler, then warps of their own
    // while there are few of them (CTAs of 8 warps would put two on each scheduler of a few SMs)
    if (n <= 8 * kSchedulers && order_of(mask) <= 2) {
      const unsigned blocks = (unsigned)((n + 7) / 8);
      switch (order_of(mask)) {
        case 0: k_eval_few<P, Q, 0><<<blocks, 32, 0, st>>>(s, uv, n, mask, out); break;
        case 1: k_eval_few<P, Q, 1><<<blocks, 32, 0, st>>>(s, uv, n, mask, out); break;
        default: k_eval_few<P, Q, 2><<<blocks, 32, 0, st>>>(s, uv, n, mask, out); break;
      }
      return cudaGetLastError();
    }
    if (n <= 32 * 4 * kSchedulers) threads = 32;
  }
  int64_t blocks = (n + threads - 1) / threads;
  const int64_t cap = 152 * 64;
  if (blocks > cap) blocks = cap;
  switch (order_of(mask)) {
    case 0: k_eval<T, P, Q, 0><<<(unsigned)blocks, threads, 0, st>>>(s, uv, n, mask, out); break;
    case 1: k_eval<T, P, Q, 1><<<(unsigned)blocks, threads, 0, st>>>(s, uv, n, mask, out); break;
    case 2: k_eval<T, P, Q, 2><<<(unsigned)blocks, threads, 0, st>>>(s, uv, n, mask, out); break;
    default: k_eval<T, P, Q, 3><<<(unsigned)blocks, threads, 0, st>>>(s, uv, n, mask, out); break;
  }
  return cudaGetLastError();
}

template <int P, int Q>
static cudaError_t launch_normal_pq(const SurfDev& s, const double* uv, int64_t n, unsigned mask, double* out,
                                    cudaStream_t st) {
  int64_t blocks = (n + 255) / 256;
  const int64_t cap = 152 * 64;
  if (blocks > cap) blocks = cap;
  if (mask & (8u | 16u | 32u)) k_eval_normal<P, Q, 3><<<(unsigned)blocks, 256, 0, st>>>(s, uv, n, mask, out);
  else if (mask & (2u | 4u)) k_eval_normal<P, Q, 2><<<(unsigned)blocks, 256, 0, st>>>(s, uv, n, mask, out);
  else k_eval_normal<P, Q, 1><<<(unsigned)blocks, 256, 0, st>>>(s, uv, n, mask, out);
  return cudaGetLastError();
}

template <typename T>
static cudaError_t dispatch(const SurfDev& s, const T* uv, int64_t n, unsigned mask, T* out, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if (s.p == 3 && s.q == 3) return launch_pq<T, 3, 3>(s, uv, n, mask, out, st);
  if (s.p == 5 && s.q == 5) return launch_pq<T, 5, 5>(s, uv, n, mask, out, st);
  if (s.p == 2 && s.q == 2) return launch_pq<T, 2, 2>(s, uv, n, mask, out, st);
  return launch_pq<T, 0, 0>(s, uv, n, mask, out, st);
}

cudaError_t launch_eval_f64(const SurfDev& s, const double* uv, int64_t n, unsigned mask, double* out,
                            cudaStream_t st) {
  return dispatch<double>(s, uv, n, mask, out, st);
}
cudaError_t launch_eval_f32(const SurfDev& s, const float* uv, int64_t n, unsigned mask, float* out,
                            cudaStream_t st) {
  return dispatch<float>(s, uv, n, mask, out, st);
}
cudaError_t launch_eval_normal(const SurfDev& s, const double* uv, int64_t n, unsigned mask, double* out,
                               cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if (s.p == 3 && s.q == 3) return launch_normal_pq<3, 3>(s, uv, n, mask, out, st);
  if (s.p == 5 && s.q == 5) return launch_normal_pq<5, 5>(s, uv, n, mask, out, st);
  return launch_normal_pq<0, 0>(s, uv, n, mask, out, st);
}

}  // namespace gnurbs
