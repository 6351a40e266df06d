// Stresses and displacements at observation points from a 2DS0 or 3DR0
// solution (the reference's BigWhamIO::ComputeStresses / ComputeDisplacements,
// src/io/bigwham_io.cc:1166-1324): for every point the sum over all elements
// of the element's field times its local DD (bw_s0.h, bw_r0_fields.h).
//
// Both kernels are bound by FP64 arithmetic: per (point, element) pair one or
// two logs and atan2, one (2DS0) or six (3DR0) divisions and 100 to 400 other operations,
// against 9 or 17 doubles of element data that a tile in shared memory gives
// to all points of the CTA.  What a pair needs is in the element headers; what
// is left is to keep the FP64 pipe busy:
// * `lanes` neighbouring lanes share a point, each taking every lanes-th
//   element of the tile, and add their sums by shuffles at the end (a fixed
//   order: results repeat bit for bit).  With one thread per point the usual
//   grids of 10^4 to 10^5 points leave most SMs with 4 to 8 warps and the last
//   wave half empty; field_lanes gives each call at least kFieldThreadsWanted
//   threads.
// * the tile holds everything that depends on the element alone.
// The outputs that are not asked for are not computed.
#pragma once

#include "bw_r0_fields.h"
#include "bw_s0.h"

namespace bw {

constexpr int kFieldThreads = 128;  // per CTA
constexpr int kFieldTile = 128;     // elements per shared-memory tile

// Lanes per point: the fewest (a power of two up to a warp) that give a call
// two threads for each of 1,024 per SM.  2DS0, 4,000 segments: 50,000 points
// 8.05 -> 2.46 ms with the element's combined forms, 300 to 1,000 points up to
// 60 times faster; 3DR0, 4,096 elements, 20,000 points 36.0 -> 4.52 ms.
constexpr long long kFieldThreadsWanted = 2 * 1024;  // per SM

inline int field_lanes(long long n_pts, int sms) {
  int lanes = 1;
  while (lanes < 32 && n_pts * lanes < kFieldThreadsWanted * sms) lanes <<= 1;
  return lanes;
}

template <bool kStress, bool kDisp>
__global__ void __launch_bounds__(kFieldThreads) s0_fields_kernel(const double *__restrict__ rec,
                                                                  const double *__restrict__ dd, int n_elems,
                                                                  const double *__restrict__ pts, long long n_pts,
                                                                  double G, double nu, int lanes,
                                                                  double *__restrict__ stress,
                                                                  double *__restrict__ disp) {
  __shared__ double s_el[kFieldTile * s0::kFieldDoubles];
  const int per_cta = kFieldThreads / lanes, sub = threadIdx.x & (lanes - 1);
  for (long long p0 = static_cast<long long>(blockIdx.x) * per_cta; p0 < n_pts;
       p0 += static_cast<long long>(gridDim.x) * per_cta) {  // uniform over the CTA
    const long long p = p0 + threadIdx.x / lanes;
    const bool live = p < n_pts;
    const double px = live ? pts[2 * p] : 0.0, py = live ? pts[2 * p + 1] : 0.0;
    double acc[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    for (int e0 = 0; e0 < n_elems; e0 += kFieldTile) {
      const int ne = min(kFieldTile, n_elems - e0);
      __syncthreads();  // the previous tile is no longer read
      for (int e = threadIdx.x; e < ne; e += kFieldThreads)
        s0::field_data(rec + static_cast<long long>(e0 + e) * s0::kRecordDoubles, dd[2LL * (e0 + e)],
                       dd[2LL * (e0 + e) + 1], nu, s_el + e * s0::kFieldDoubles);
      __syncthreads();
      if (live)
        for (int e = sub; e < ne; e += lanes)
          s0::add_fields<kStress, kDisp>(s_el + e * s0::kFieldDoubles, px, py, G, nu, acc);
    }
#pragma unroll
    for (int k = 0; k < 5; k++)
      for (int o = lanes >> 1; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
    if (live && sub == 0) {
      if (kStress)
        for (int k = 0; k < 3; k++) stress[3 * p + k] = acc[k];
      if (kDisp)
        for (int k = 0; k < 2; k++) disp[2 * p + k] = acc[3 + k];
    }
  }
}

// 3DR0: as s0_fields_kernel, with the element's kFieldDoubles values (from the
// 17-double assembly records and the local DDs) staged per tile.
template <bool kStress, bool kDisp>
__global__ void __launch_bounds__(kFieldThreads) r0_fields_kernel(const double *__restrict__ rec,
                                                                  const double *__restrict__ dd, int n_elems,
                                                                  const double *__restrict__ pts, long long n_pts,
                                                                  double G, double nu, int lanes,
                                                                  double *__restrict__ stress,
                                                                  double *__restrict__ disp) {
  __shared__ double s_el[kFieldTile * r0::kFieldDoubles];
  const int per_cta = kFieldThreads / lanes, sub = threadIdx.x & (lanes - 1);
  for (long long p0 = static_cast<long long>(blockIdx.x) * per_cta; p0 < n_pts;
       p0 += static_cast<long long>(gridDim.x) * per_cta) {  // uniform over the CTA
    const long long p = p0 + threadIdx.x / lanes;
    const bool live = p < n_pts;
    double q[3] = {0.0, 0.0, 0.0};
    if (live)
      for (int k = 0; k < 3; k++) q[k] = pts[3 * p + k];
    double acc[9] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    for (int e0 = 0; e0 < n_elems; e0 += kFieldTile) {
      const int ne = min(kFieldTile, n_elems - e0);
      __syncthreads();  // the previous tile is no longer read
      // record layout: cp 0-2, rotation 3-11, normal 12-14, a 15, b 16
      for (int w = threadIdx.x; w < ne * 14; w += kFieldThreads) {
        const int e = w / 14, k = w % 14;
        s_el[e * r0::kFieldDoubles + k] =
            rec[static_cast<long long>(e0 + e) * r0::kFrameDoubles + (k < 12 ? k : k + 3)];
      }
      for (int w = threadIdx.x; w < ne * 3; w += kFieldThreads)
        s_el[(w / 3) * r0::kFieldDoubles + 14 + w % 3] = dd[3 * static_cast<long long>(e0) + w];
      __syncthreads();
      if (live)
        for (int e = sub; e < ne; e += lanes)
          r0::add_point_fields<kStress, kDisp>(s_el + e * r0::kFieldDoubles, q, G, nu, acc);
    }
#pragma unroll
    for (int k = 0; k < 9; k++)
      for (int o = lanes >> 1; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
    if (live && sub == 0) {
      if (kStress)
        for (int k = 0; k < 6; k++) stress[6 * p + k] = acc[k];
      if (kDisp)
        for (int k = 0; k < 3; k++) disp[3 * p + k] = acc[6 + k];
    }
  }
}

}  // namespace bw
