// Stage a: knot vectors -> per-span rational power-basis matrices (K1 span_convert).
//
// Replaces GetMatrixN (src/NURBS/Evaluate.cu:3-88).  The reference launches one thread per
// knot pair (i,j), recomputes both basis-to-power matrices per thread with the 4^p-way Nrc
// recursion (:90-103), allocates temporaries on the device heap and multiplies through eight
// dynamic-parallelism child grids.  Here:
//   1. k_basis: one CTA per (direction, span) evaluates the Nrc recurrence of all its columns level
//      by level (each state once, one thread per state), the level's knot quotients once for all;
//      each direction's spans are done once, not once per (i,j).
//   2. k_span_matrices: one thread per (span, column of the product, homogeneous component) forms
//      N_u . (W.P_c) . N_v^T with the reference's summation order, the weighted control net of the
//      CTA's spans in shared memory.
// Both are bound by FP64 issue (64 clocks per warp instruction): the threads are laid out so that
// few FP64 instructions follow one another in one warp and all schedulers have some.
// This translation unit is compiled with --fmad=false: every product and sum rounds as in
// the reference's unfused FP64 arithmetic, so the matrices are bit-identical to GetMatrixN's.
#include "nurbs_internal.h"
#include "nurbs_math.cuh"

namespace gnurbs {

// Nrc table of one span, by one CTA: the reference's recurrence (src/NURBS/Evaluate.cu:90-103)
// evaluated bottom-up, each (column, r, j) entry once, in the reference's expression order.
// out[(r-1)*k + (c-1)] = Nrc(knot, d, r, c, I, I, d), I = span - (d-1).
constexpr int kBasisThreads = 128;
__device__ __forceinline__ void basis_span(const double* __restrict__ knot, int d, int span, double* __restrict__ out) {
  constexpr int kMaxR = 2 * kMaxDegree + 1, kMaxJ = kMaxDegree + 1;
  __shared__ double tab[2][kMaxJ][kMaxR * kMaxJ];
  __shared__ double quo[kMaxJ][4];
  const int k = d + 1;
  const int I = span - (d - 1);
  const int R0 = 1 - d, RN = 2 * d + 1;
  const int J0 = I - d, JN = d + 1;
  for (int e = threadIdx.x; e < k * RN * JN; e += kBasisThreads) {
    const int c = e / (RN * JN) + 1, x = e % (RN * JN), r = R0 + x / JN, j = J0 + x % JN;
    tab[0][c - 1][x] = (((I + c - 1) == (j + d)) && (r == 1)) ? 1.0 : 0.0;  // Evaluate.cu:91-95
  }
  // A = Nabla(knot, d, I, 1) = knot[I+d] - knot[I+d-1] (the span length)
  const double A = knot[I + d] - knot[I + d - 1];
  for (int m = 1; m <= d; ++m) {
    const int r0 = 1 - (d - m), nr = d + 1 - r0 + 1, j0 = I - (d - m), nj = d - m + 1;
    if ((int)threadIdx.x < nj) {
      const int j = j0 + threadIdx.x;
      // B = Nabla(knot, d, j, d-m+1), C = Nabla(knot, d, j, I-j)   (Evaluate.cu:105-108)
      const double B = knot[j + d - 1 + (d - m + 1)] - knot[j + d - 1];
      const double C = knot[j + d - 1 + (I - j)] - knot[j + d - 1];
      const double ab = A / B, cb = C / B;
      quo[threadIdx.x][0] = ab;
      quo[threadIdx.x][1] = cb;
      quo[threadIdx.x][2] = 1 - cb;
      quo[threadIdx.x][3] = -ab;
    }
    __syncthreads();
    const double(*prev)[kMaxR * kMaxJ] = tab[(m - 1) & 1];
    double(*cur)[kMaxR * kMaxJ] = tab[m & 1];
    for (int e = threadIdx.x; e < k * nr * nj; e += kBasisThreads) {
      const int c = e / (nr * nj), x = e % (nr * nj), jj = x % nj;
      const int ri = r0 + x / nj - R0, ji = j0 + jj - J0;
      const double n1 = prev[c][(ri - 1) * JN + ji];
      const double n2 = prev[c][ri * JN + ji];
      const double n3 = prev[c][ri * JN + (ji - 1)];
      const double n4 = prev[c][(ri - 1) * JN + (ji - 1)];
      cur[c][ri * JN + ji] = quo[jj][0] * n1 + quo[jj][1] * n2 + quo[jj][2] * n3 + quo[jj][3] * n4;  // :98-101
    }
    __syncthreads();
  }
  for (int e = threadIdx.x; e < k * k; e += kBasisThreads) {
    const int r = e / k + 1, c = e % k;
    out[e] = tab[d & 1][c][(r - R0) * JN + (I - J0)];
  }
}

// One CTA per span: the u direction's spans, then the v direction's.
__global__ void __launch_bounds__(kBasisThreads)
    k_basis(const double* __restrict__ ku, int p, const int* __restrict__ idx_u, int ns_u, double* __restrict__ bas_u,
            const double* __restrict__ kv, int q, const int* __restrict__ idx_v, double* __restrict__ bas_v) {
  const int b = blockIdx.x;
  if (b < ns_u) basis_span(ku, p, idx_u[b], bas_u + (size_t)b * (p + 1) * (p + 1));
  else basis_span(kv, q, idx_v[b - ns_u], bas_v + (size_t)(b - ns_u) * (q + 1) * (q + 1));
}

// Batched over many (surface, direction) jobs: CTA b belongs to the job with the largest item0 <= b.
__global__ void __launch_bounds__(kBasisThreads) k_basis_batched(const BasisJob* __restrict__ jobs, int njobs) {
  const int64_t t = blockIdx.x;
  int lo = 0, hi = njobs - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].item0 <= t) lo = mid;
    else hi = mid - 1;
  }
  const BasisJob J = jobs[lo];
  const int k = J.degree + 1;
  const int sidx = (int)(t - J.item0);
  basis_span(J.knots, J.degree, J.knot_idx[sidx], J.out + (size_t)sidx * k * k);
}

// out_c = Nu . (Mid_c . NvT) for span_group(q) spans from `first` on, by one CTA.  Dense output
// (m64/m32) or, when ref_out != nullptr, the reference MatrixN layout.
constexpr int kSpanThreads = 128;
static_assert(kSpanThreads == kSpanGroupThreads, "span_group counts this kernel's threads");
__device__ __forceinline__ void span_group_matrices(const SurfDev& s, const double* __restrict__ basis_u,
                                                    const double* __restrict__ basis_v, int first,
                                                    double* __restrict__ m64, float* __restrict__ m32,
                                                    double* __restrict__ ref_out) {
  // Middle_c = P_c * w (Evaluate.cu:35-43) of the CTA's spans; and for the FP32 table that of the
  // surface translated by -org (the matrix form is linear in the weighted control points), computed
  // in FP64 and rounded once
  __shared__ double mid[kSpanThreads * (kMaxDegree + 1)];
  __shared__ double mid32[kSpanThreads * (kMaxDegree + 1)];
  const int p = s.p, q = s.q, k1 = p + 1, k2 = q + 1, k12 = k1 * k2;
  const int nspans = s.ns_u * s.ns_v, group = span_group(q), here = min(group, nspans - first);
  for (int e = threadIdx.x; e < here * k12 * 4; e += kSpanThreads) {
    const int c = e & 3, x = e >> 2, ab = x % k12, span = first + x / k12;
    const int i = s.knot_u[span / s.ns_v], j = s.knot_v[span % s.ns_v];
    const size_t idx = (size_t)(ab / k2 + i - p) * s.nv + (ab % k2 + j - q);
    const double w = s.weights[idx];
    if (c < 3) {
      const double x3 = s.cps[3 * idx + c];
      mid[e] = x3 * w;
      mid32[e] = (x3 - s.org[c]) * w;
    } else {
      mid[e] = w;
    }
  }
  __syncthreads();
  const int c = threadIdx.x & 3, l = (threadIdx.x >> 2) % k2, g = (threadIdx.x >> 2) / k2;
  if (g >= here) return;
  const int span = first + g, su = span / s.ns_v, sv = span % s.ns_v;
  const double* Nu = basis_u + (size_t)su * k1 * k1;
  const double* Nv = basis_v + (size_t)sv * k2 * k2 + l * k2;
  // column l of the product: temp = Middle . NvT with NvT[t][l] = Nv[l][t] (matrix_mult, Matrix.cu:43-52
  // order), out = Nu . temp
  auto column = [&](const double* m, auto&& put) {
    double tmp[kMaxDegree + 1];
#pragma unroll
    for (int a = 0; a <= kMaxDegree; ++a) {
      if (a < k1) {
        double acc = 0;
        for (int tt = 0; tt < k2; ++tt) acc += m[(a * k2 + tt) * 4] * Nv[tt];
        tmp[a] = acc;
      }
    }
    for (int a = 0; a < k1; ++a) {
      double acc = 0;
#pragma unroll
      for (int ss = 0; ss <= kMaxDegree; ++ss)
        if (ss < k1) acc += Nu[a * k1 + ss] * tmp[ss];
      put(a, acc);
    }
  };
  const size_t o32 = ((size_t)span * span_coefs32(p, q) + l) * 4 + c;
  column(mid + (size_t)g * k12 * 4 + c, [&](int a, double x) {
    if (ref_out) {
      // MatrixNPosition(i, j, p, q, nu, nv, c) + a*k2 + l   (Evaluate.cu:110-112)
      const size_t pos = (((size_t)s.knot_u[su] * (q + s.nv) + s.knot_v[sv]) * 4 + c) * (size_t)k12 + a * k2 + l;
      ref_out[pos] = x;
    } else {
      m64[((size_t)span * k12 + a * k2 + l) * 4 + c] = x;
      if (c == 3) m32[o32 + (size_t)a * k2 * 4] = (float)x;
    }
  });
  if (ref_out || c == 3) return;
  column(mid32 + (size_t)g * k12 * 4 + c, [&](int a, double x) { m32[o32 + (size_t)a * k2 * 4] = (float)x; });
}

__global__ void __launch_bounds__(kSpanThreads)
    k_span_matrices(SurfDev s, const double* __restrict__ basis_u, const double* __restrict__ basis_v,
                    double* __restrict__ m64, float* __restrict__ m32, double* __restrict__ ref_out) {
  span_group_matrices(s, basis_u, basis_v, blockIdx.x * span_group(s.q), m64, m32, ref_out);
}

// Batched: CTA b belongs to the job with the largest item0 <= b.
__global__ void __launch_bounds__(kSpanThreads) k_span_matrices_batched(const SurfDev* __restrict__ table,
                                                                        const SpanJob* __restrict__ jobs, int njobs) {
  const int64_t t = blockIdx.x;
  int lo = 0, hi = njobs - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].item0 <= t) lo = mid;
    else hi = mid - 1;
  }
  const SurfDev s = table[jobs[lo].surf];
  span_group_matrices(s, s.basis_u, s.basis_v, (int)(t - jobs[lo].item0) * span_group(s.q),
                      const_cast<double*>(s.m64), const_cast<float*>(s.m32), nullptr);
}

// Dense -> reference MatrixN layout, one thread per double.
__global__ void k_export_ref(SurfDev s, double* __restrict__ ref_out) {
  const int k1 = s.p + 1, k2 = s.q + 1, k12 = k1 * k2;
  int64_t total = (int64_t)s.ns_u * s.ns_v * k12 * 4;
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return;
  int c = (int)(t & 3);
  int64_t e = t >> 2;
  int ab = (int)(e % k12);
  int64_t span = e / k12;
  int su = (int)(span / s.ns_v), sv = (int)(span % s.ns_v);
  int i = s.knot_u[su], j = s.knot_v[sv];
  size_t pos = (((size_t)i * (s.q + s.nv) + j) * 4 + c) * (size_t)k12 + ab;
  ref_out[pos] = s.m64[t];
}

cudaError_t launch_basis_pair(const double* knots_u, int p, const int* idx_u, int ns_u, double* basis_u,
                              const double* knots_v, int q, const int* idx_v, int ns_v, double* basis_v,
                              cudaStream_t st) {
  if (ns_u + ns_v <= 0) return cudaSuccess;
  k_basis<<<ns_u + ns_v, kBasisThreads, 0, st>>>(knots_u, p, idx_u, ns_u, basis_u, knots_v, q, idx_v, basis_v);
  return cudaGetLastError();
}

cudaError_t launch_span_matrices(const SurfDev& s, const double* basis_u, const double* basis_v, double* m64,
                                 float* m32, cudaStream_t st) {
  const int64_t blocks = span_blocks(s.q, (int64_t)s.ns_u * s.ns_v);
  if (blocks <= 0) return cudaSuccess;
  double* ref_out = (m32 == nullptr) ? m64 : nullptr;
  k_span_matrices<<<(unsigned)blocks, kSpanThreads, 0, st>>>(s, basis_u, basis_v, ref_out ? nullptr : m64, m32, ref_out);
  return cudaGetLastError();
}

cudaError_t launch_basis_batched(const BasisJob* jobs, int njobs, int64_t nspans, cudaStream_t st) {
  if (nspans <= 0) return cudaSuccess;
  k_basis_batched<<<(unsigned)nspans, kBasisThreads, 0, st>>>(jobs, njobs);
  return cudaGetLastError();
}

cudaError_t launch_span_matrices_batched(const SurfDev* table, const SpanJob* jobs, int njobs, int64_t nblocks,
                                         cudaStream_t st) {
  if (nblocks <= 0) return cudaSuccess;
  k_span_matrices_batched<<<(unsigned)nblocks, kSpanThreads, 0, st>>>(table, jobs, njobs);
  return cudaGetLastError();
}

cudaError_t launch_export_ref_layout(const SurfDev& s, double* matrix_n, cudaStream_t st) {
  int64_t total = (int64_t)s.ns_u * s.ns_v * (s.p + 1) * (s.q + 1) * 4;
  if (total <= 0) return cudaSuccess;
  k_export_ref<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(s, matrix_n);
  return cudaGetLastError();
}

}  // namespace gnurbs
