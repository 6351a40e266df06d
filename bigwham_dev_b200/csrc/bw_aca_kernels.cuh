// Device block ACA of the admissible blocks of a 3DR0-H H-matrix.
//
// One CTA compresses one block at a time, running the steps of
// bw::aca::block_aca_host with the work of each step spread over the CTA's
// threads:
//   * residual row / column bands: one thread per point pair (kernel entry +
//     the subtraction of the current approximation);
//   * pivot searches: per-thread smallest singular values, then a CTA argmax
//     that keeps the first index on ties (the reference scans in order and
//     replaces only on a strictly larger value);
//   * Frobenius terms of the new rank block with every earlier one and with
//     itself, together: A_r^T A_k by a warp per r, lanes along A's contiguous
//     columns; B_k B_r^T by a lane per r, which B's storage keeps side by
//     side, warps along the points.
// The arithmetic is small (about 1 GFLOP for a 64 x 64 crack); a step's time is
// the latency of what it does one after the other, so the steps have a fixed
// number of barriers (ten, at any rank: two CTA reductions per earlier rank
// block took most of the time before), and the blocks come from a queue,
// longest first, so that the largest does not start last.
// A 64 x 64 crack's 1,584 blocks, one call of bw_r0_aca: 18.5 ms at first, 6.1 ms
// with this pass, the queue and a launch per size (kAcaSide).  The three sizes are
// held to 128 registers and spill 224 to 312 bytes of the off-plane entry.
// Every stop decision is taken from values in shared memory that all threads
// read, so all threads leave the loop together.  Factor storage per block is
// capacity-bounded (cap blocks of rank); a block that needs more reports
// rank -1 and writes nothing past its capacity.
#pragma once

#include "bw_aca.h"
#include "bw_kernels.cuh"
#include "bw_r0.h"

namespace bw {

// Threads per block of points: a warp for blocks of up to kAcaSide[0] points a
// side, whose bands one warp covers in one or two rounds, 128 up to kAcaSide[1],
// 512 above.  With 128 threads for all, three of the four warps of a 32-point
// block waited at barriers and held registers, and each of a 64 x 64 crack's 24
// blocks of 512 points took 9 ms, as long as the whole launch.
constexpr int kAcaSide[2] = {48, 128};
constexpr int kAcaResident = 512;  // threads per SM that the registers are limited for

struct AcaBlock {
  long long a_off, b_off;  // factor storage (doubles): A n0 3 x cap 3, B cap 3 x n1 3, column-major
  long long s_off;         // unused here (kept for alignment of the record)
  int i0, j0, n0, n1;      // first row / column point (permuted numbering), sizes in points
  int cap, pad;            // rank capacity in blocks
};

template <int NT> __device__ __forceinline__ void aca_sync() {
  if constexpr (NT == 32)
    __syncwarp();
  else
    __syncthreads();
}

// CTA argmax of (value, index) pairs: largest value, smallest index on ties;
// index -1 when no thread had a candidate.
template <int NT> __device__ __forceinline__ void aca_argmax(double v, int idx, double *sv, int *si, int &bi) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto better = [](double v2, int i2, double v1, int i1) {
    return i2 >= 0 && (i1 < 0 || v2 > v1 || (v2 == v1 && i2 < i1));
  };
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double v2 = __shfl_xor_sync(0xffffffffu, v, o);
    const int i2 = __shfl_xor_sync(0xffffffffu, idx, o);
    if (better(v2, i2, v, idx)) {
      v = v2;
      idx = i2;
    }
  }
  if (lane == 0) {
    sv[warp] = v;
    si[warp] = idx;
  }
  aca_sync<NT>();
  bi = si[0];
  double best = sv[0];
  for (int w = 1; w < (NT / 32); w++)
    if (better(sv[w], si[w], best, bi)) {
      best = sv[w];
      bi = si[w];
    }
  aca_sync<NT>();
}

// K -= A B over `rank` scalar columns: A's three rows of one point, B's three
// columns of another.
__device__ __forceinline__ void aca_subtract(const double *A, long long lda, const double *B, long long ldb, int rank,
                                             double (&K)[3][3]) {
#pragma unroll 3
  for (int k = 0; k < rank; k++) {
    const double a0 = A[k * lda], a1 = A[k * lda + 1], a2 = A[k * lda + 2];
#pragma unroll
    for (int b = 0; b < 3; b++) {
      const double v = B[b * ldb + k];
      K[0][b] -= a0 * v;
      K[1][b] -= a1 * v;
      K[2][b] -= a2 * v;
    }
  }
}

constexpr int kAcaPass = 32;  // earlier rank blocks whose Frobenius terms one pass takes (a lane each)

template <int NT> struct AcaFrob {
  double m1[kAcaPass][9];           // A_r^T A_k
  double m2[NT / 32][9][kAcaPass];  // per warp: part of (B_k B_r^T)^T
};

// Frobenius products <A_r B_r, A_k B_k>_F for r = 0 .. k: their sum over r < k
// in `cross` and the term r = k in `self` (all threads).
template <int NT>
__device__ __forceinline__ void aca_frobenius(const double *A, long long lda, const double *B, long long ldb, int k,
                                              long long cols, AcaFrob<NT> &f, double *s_out, double &cross,
                                              double &self) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  cross = 0.0;
  self = 0.0;
  const double *Ak = A + 3LL * k * lda;
  for (int r0 = 0; r0 <= k; r0 += kAcaPass) {
    const int nr = min(kAcaPass, k + 1 - r0);
    // warp: one r at a time, lanes along the rows
    for (int q = warp; q < nr; q += (NT / 32)) {
      const double *Ar = A + 3LL * (r0 + q) * lda;
      double m[9] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll 2
      for (long long i = lane; i < lda; i += 32) {
        const double a0 = Ar[i], a1 = Ar[lda + i], a2 = Ar[2 * lda + i];
#pragma unroll
        for (int b = 0; b < 3; b++) {
          const double v = Ak[b * lda + i];
          m[3 * b] += a0 * v;
          m[3 * b + 1] += a1 * v;
          m[3 * b + 2] += a2 * v;
        }
      }
#pragma unroll
      for (int e = 0; e < 9; e++)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m[e] += __shfl_xor_sync(0xffffffffu, m[e], o);
      if (lane == 0)
#pragma unroll
        for (int e = 0; e < 9; e++) f.m1[q][e] = m[e];
    }
    // lane: one r, warps along the columns
    double m[9] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (lane < nr) {
      const double *Br = B + 3LL * (r0 + lane), *Bk = B + 3LL * k;
#pragma unroll 4
      for (long long j = warp; j < cols; j += (NT / 32)) {
        const double *c = Br + j * ldb, *d = Bk + j * ldb;
        const double a0 = c[0], a1 = c[1], a2 = c[2];
#pragma unroll
        for (int b = 0; b < 3; b++) {
          m[3 * b] += a0 * d[b];
          m[3 * b + 1] += a1 * d[b];
          m[3 * b + 2] += a2 * d[b];
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 9; e++) f.m2[warp][e][lane] = m[e];
    aca_sync<NT>();
    if (warp == 0) {
      double v = 0.0;
      if (lane < nr)
#pragma unroll
        for (int e = 0; e < 9; e++) {
          double m2 = f.m2[0][e][lane];
          for (int w = 1; w < (NT / 32); w++) m2 += f.m2[w][e][lane];
          v += f.m1[lane][e] * m2;
        }
      const bool last = r0 + lane == k;
      const double own = __shfl_sync(0xffffffffu, v, (k - r0) & 31);
      v = last || lane >= nr ? 0.0 : v;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) {
        s_out[0] = v;
        s_out[1] = own;
      }
    }
    aca_sync<NT>();
    cross += s_out[0];
    self = s_out[1];  // the last pass holds r = k
  }
}

template <int NT>
__global__ void __launch_bounds__(NT, kAcaResident / NT)
    r0_aca_kernel(const double *__restrict__ records, const int *__restrict__ perm,
                  const AcaBlock *__restrict__ blocks, int n_blocks, double G, double nu, double eps,
                  double *factors_a, double *factors_b, double *scratch, long long slot_doubles, const int *order,
                  int *queue, int *rank_out, double *err_out) {
  __shared__ double s_val[NT / 32];
  __shared__ int s_idx[NT / 32];
  __shared__ AcaFrob<NT> s_frob;
  __shared__ double s_gamma[9], s_sum[2];
  __shared__ int s_ctl[2];  // [0] continue, [1] the CTA's next block
  const int t = threadIdx.x;
  pdl_launch_dependents();  // the other size's launch, independent of this one, may run beside it
  double *row = scratch + (long long)blockIdx.x * slot_doubles;  // 3 x n1 3 (ld 3)
  for (;;) {
    if (t == 0) s_ctl[1] = atomicAdd(queue, 1);
    aca_sync<NT>();
    const int place = s_ctl[1];
    if (place >= n_blocks) break;
    const int bk = order[place];
    const AcaBlock B_ = blocks[bk];
    const int n0 = B_.n0, n1 = B_.n1, cap = B_.cap;
    const long long lda = 3LL * n0, ldb = 3LL * cap;
    double *A = factors_a + B_.a_off;
    double *Bf = factors_b + B_.b_off;
    int *used0 = reinterpret_cast<int *>(row + 9LL * n1);
    int *used1 = used0 + n0;
    for (int i = t; i < n0; i += NT) used0[i] = 0;
    for (int j = t; j < n1; j += NT) used1[j] = 0;
    aca_sync<NT>();
    auto entry = [&](int i, int j, double K[3][3]) {
      const double *src = records + r0::kFrameDoubles * perm[B_.j0 + j];
      const double *rec = records + r0::kFrameDoubles * perm[B_.i0 + i];
      r0::influence_h(src, src + 3, src[15], src[16], rec, rec + 3, rec + 12, G, nu, K);
    };
    int rank = 0, i0 = 0, status = 0;  // status: 0 running, 1 done, 2 overflow
    double s_norm = 0.0, err = 0.0;
    const int max_rank = n0 < n1 ? n0 : n1;
    while (status == 0) {
      if (rank >= cap) {
        status = 2;
        break;
      }
      // residual row band of row block i0
      for (int j = t; j < n1; j += NT) {
        double K[3][3];
        entry(i0, j, K);
        aca_subtract(A + 3LL * i0, lda, Bf + 3LL * j * ldb, ldb, 3 * rank, K);
#pragma unroll
        for (int b = 0; b < 3; b++)
#pragma unroll
          for (int a = 0; a < 3; a++) row[(3LL * j + b) * 3 + a] = K[a][b];
      }
      aca_sync<NT>();
      // pivot column block
      double best = 0.0;
      int bi = -1;
      for (int j = t; j < n1; j += NT) {
        if (used1[j]) continue;
        const double sv = aca::smallest_singular_value(row + 9LL * j);
        if (sv > best) {  // ascending j per thread: the first maximum stays
          best = sv;
          bi = j;
        }
      }
      int i1;
      aca_argmax<NT>(best, bi, s_val, s_idx, i1);
      if (i1 < 0) break;  // uniform: every thread read the same i1
      if (t == 0) {
        used0[i0] = 1;
        used1[i1] = 1;
        s_ctl[0] = aca::invert3(row + 9LL * i1, s_gamma) ? 1 : 0;
      }
      aca_sync<NT>();
      if (!s_ctl[0]) break;
      // A_k: residual column band of column block i1
      for (int i = t; i < n0; i += NT) {
        double K[3][3];
        entry(i, i1, K);
        aca_subtract(A + 3LL * i, lda, Bf + 3LL * i1 * ldb, ldb, 3 * rank, K);
#pragma unroll
        for (int b = 0; b < 3; b++)
#pragma unroll
          for (int a = 0; a < 3; a++) A[(3LL * rank + b) * lda + 3LL * i + a] = K[a][b];
      }
      // B_k = Gamma R
      for (int j = t; j < 3 * n1; j += NT)
        for (int a = 0; a < 3; a++) {
          double v = 0.0;
          for (int c = 0; c < 3; c++) v += s_gamma[c * 3 + a] * row[3LL * j + c];
          Bf[(long long)j * ldb + 3LL * rank + a] = v;
        }
      aca_sync<NT>();
      // |A_k B_k|_F^2 and cross terms with the earlier rank blocks
      double ab, cross;
      aca_frobenius<NT>(A, lda, Bf, ldb, rank, 3LL * n1, s_frob, s_sum, cross, ab);
      s_norm += 2.0 * cross + ab;
      // next row block from A_k
      best = 0.0;
      bi = -1;
      for (int i = t; i < n0; i += NT) {
        if (used0[i]) continue;
        double blk[9];
        for (int b = 0; b < 3; b++)
          for (int a = 0; a < 3; a++) blk[b * 3 + a] = A[(3LL * rank + b) * lda + 3LL * i + a];
        const double sv = aca::smallest_singular_value(blk);
        if (sv > best) {
          best = sv;
          bi = i;
        }
      }
      int next;
      aca_argmax<NT>(best, bi, s_val, s_idx, next);
      rank++;
      if (next < 0 || rank == max_rank) break;
      if (fabs(ab) <= eps * eps * fabs(s_norm)) {
        err = sqrt(fabs(ab) / fabs(s_norm));
        break;
      }
      i0 = next;
    }
    if (t == 0) {
      rank_out[bk] = status == 2 ? -1 : rank;
      err_out[bk] = err;
    }
    aca_sync<NT>();
  }
  pdl_wait();  // completes after the launch before it
}

}  // namespace bw
