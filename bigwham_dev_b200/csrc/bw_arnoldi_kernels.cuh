// One Arnoldi step of GMRES after the operator: classical Gram-Schmidt with one
// re-orthogonalisation and the new basis vector, FP64.
//
//   h = V w, w -= V^T h;  h2 = V w, w -= V^T h2;  v = w / |w|
//
// with V the j + 1 basis vectors so far (rows of length n).  Four launches: a
// grid-wide sum ends each, so a launch leaves every CTA's partial sums and the
// next one adds them, every CTA for itself and in the CTAs' order (results
// repeat bit for bit).  The step reads V four times, from L2 at the sizes GMRES
// restarts keep; what bounds it is the latency of four short launches, against
// some sixteen of separate vector operations before: a cycle of 30 steps at
// 12,288 DoF 3.83 -> 2.86 ms, 2.19 of them the matvecs.
#pragma once

#include "bw_kernels.cuh"

namespace bw {

constexpr int kArnoldiThreads = 512;
constexpr int kArnoldiWarps = kArnoldiThreads / 32;
constexpr int kArnoldiMaxSteps = 4096;  // the coefficients fit the default 48 KB of shared memory

struct ArnoldiArgs {
  double *V;           // (m + 1) x n, row j + 1 is written
  double *H;           // (m + 1) x m, column j is written
  double *w;           // operator output, length n; overwritten
  const double *minv;  // optional: z = minv * v for the next step
  double *z;
  double *part;        // 3 x gridDim x (m + 2) partial sums
  long long n;
  int j, m;
  double breakdown;    // |w| below this share of the operator output's norm: the space is exhausted
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// This CTA's slice of the vectors.
__device__ __forceinline__ void arnoldi_slice(long long n, long long &c0, long long &c1) {
  c0 = n * blockIdx.x / gridDim.x;
  c1 = n * (blockIdx.x + 1) / gridDim.x;
}

// part[i] = <V_i, w> over the slice, i = 0 .. j (a warp per i), part[j + 1] = <w, w>.
__device__ __forceinline__ void arnoldi_dots(const ArnoldiArgs &a, long long c0, long long c1, double *part) {
  const int lane = threadIdx.x & 31;
  for (int i = threadIdx.x >> 5; i <= a.j + 1; i += kArnoldiWarps) {
    const double *v = i <= a.j ? a.V + static_cast<long long>(i) * a.n : a.w;
    double s = 0.0;
#pragma unroll 4
    for (long long q = c0 + lane; q < c1; q += 32) s = fma(v[q], a.w[q], s);
    s = warp_sum(s);
    if (lane == 0) part[i] = s;
  }
}

// out[i] = sum over the CTAs of part[cta (m + 2) + i], i = 0 .. count - 1.
__device__ __forceinline__ void arnoldi_total(const ArnoldiArgs &a, const double *part, int count, double *out) {
  const int lane = threadIdx.x & 31;
  for (int i = threadIdx.x >> 5; i < count; i += kArnoldiWarps) {
    double s = 0.0;
    for (int c = lane; c < static_cast<int>(gridDim.x); c += 32) s += part[static_cast<long long>(c) * (a.m + 2) + i];
    s = warp_sum(s);
    if (lane == 0) out[i] = s;
  }
  __syncthreads();
}

// w -= V^T h over the slice.  A short slice is shared by groups of threads that
// take every groups-th basis vector and meet in red (kArnoldiThreads doubles).
__device__ __forceinline__ void arnoldi_update(const ArnoldiArgs &a, long long c0, long long c1, const double *h,
                                               double *red) {
  const int len = static_cast<int>(c1 - c0 < kArnoldiThreads ? c1 - c0 : kArnoldiThreads);
  const int width = len > 0 ? (len + 31) / 32 * 32 : 32, groups = kArnoldiThreads / width;
  const int q = threadIdx.x % width, g = threadIdx.x / width;
  for (long long t0 = c0; t0 < c1; t0 += width) {  // uniform over the CTA
    const long long p = t0 + q;
    double s = 0.0;
    if (p < c1 && g < groups) {
#pragma unroll 8
      for (int i = g; i <= a.j; i += groups) s = fma(a.V[static_cast<long long>(i) * a.n + p], h[i], s);
    }
    red[threadIdx.x] = s;
    __syncthreads();
    if (g == 0 && p < c1) {
      for (int k = 1; k < groups; k++) s += red[k * width + q];
      a.w[p] -= s;
    }
    __syncthreads();
  }
}

// Step 0: h partials.  Steps 1 and 2: w -= V^T h with the step before's sums,
// then the partials of the next sums (h2; |w|^2).  Step 3: the column of H and
// the next basis vector.
template <int kStep>
__global__ void __launch_bounds__(kArnoldiThreads) arnoldi_kernel(ArnoldiArgs a) {
  extern __shared__ double s_h[];  // m + 2
  __shared__ double red[kArnoldiThreads];
  pdl_wait();
  pdl_launch_dependents();
  long long c0, c1;
  arnoldi_slice(a.n, c0, c1);
  const long long stride = static_cast<long long>(gridDim.x) * (a.m + 2);
  double *own = a.part + (kStep < 3 ? kStep : 0) * stride + static_cast<long long>(blockIdx.x) * (a.m + 2);
  if constexpr (kStep == 0) {
    arnoldi_dots(a, c0, c1, own);
  } else if constexpr (kStep < 3) {
    arnoldi_total(a, a.part + (kStep - 1) * stride, a.j + 1, s_h);
    arnoldi_update(a, c0, c1, s_h, red);
    if constexpr (kStep == 1) {
      arnoldi_dots(a, c0, c1, own);
    } else {
      double s = 0.0;
      for (long long q = c0 + threadIdx.x; q < c1; q += kArnoldiThreads) s = fma(a.w[q], a.w[q], s);
      s = warp_sum(s);
      if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
      __syncthreads();
      if (threadIdx.x == 0) {
        for (int k = 1; k < kArnoldiWarps; k++) s += red[k];
        own[0] = s;
      }
    }
  } else {
    // |w|^2 (third sums) and, for the breakdown test, that of the operator's
    // output (behind the first sums)
    if (threadIdx.x < 64) {
      const double *p = threadIdx.x < 32 ? a.part + 2 * stride : a.part + a.j + 1;
      const int lane = threadIdx.x & 31;
      double s = 0.0;
      for (int c = lane; c < static_cast<int>(gridDim.x); c += 32) s += p[static_cast<long long>(c) * (a.m + 2)];
      s = warp_sum(s);
      if (lane == 0) red[threadIdx.x >> 5] = sqrt(s);
    }
    __syncthreads();
    const double nrm = red[0], live = nrm > a.breakdown * red[1] ? 1.0 : 0.0;
    const double safe = live != 0.0 ? nrm : 1.0;
    double *v = a.V + static_cast<long long>(a.j + 1) * a.n;
    for (long long q = c0 + threadIdx.x; q < c1; q += kArnoldiThreads) {
      const double x = a.w[q] / safe * live;
      v[q] = x;
      if (a.minv) a.z[q] = x * a.minv[q];
    }
    if (blockIdx.x == 0) {
      __syncthreads();
      arnoldi_total(a, a.part, a.j + 1, s_h);  // h
      for (int i = threadIdx.x >> 5; i <= a.j; i += kArnoldiWarps) {
        const int lane = threadIdx.x & 31;
        double s = 0.0;
        for (int c = lane; c < static_cast<int>(gridDim.x); c += 32)
          s += a.part[stride + static_cast<long long>(c) * (a.m + 2) + i];  // h2
        s = warp_sum(s);
        if (lane == 0) a.H[static_cast<long long>(i) * a.m + a.j] = s_h[i] + s;
      }
      if (threadIdx.x == 0) a.H[static_cast<long long>(a.j + 1) * a.m + a.j] = live != 0.0 ? nrm : 0.0;
    }
  }
}

}  // namespace bw
