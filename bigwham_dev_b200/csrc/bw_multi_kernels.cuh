// Device code of the FP64 / FP32 product with several right-hand sides,
// Y = H X in passes of K = 4 or 8 columns (sm_100a).
//
// One matvec per column reads the whole block data once per column; these
// kernels read it once per K columns.  They walk the matvec's own plan (the
// chunks, queue units and the split between the CTA-wide and the unstaged
// kernel of bw_kernels.cuh) and keep its arithmetic order in every column, so
// column j equals the matvec of column j bit for bit.
//
// The vectors are stored K values per row (x of row i at [i K, i K + K)), which
// is a multiple of 16 bytes for every K and type used.  A chunk's vector values
// therefore need no gathered copy: each of its runs (a piece of x or of t) is
// one bulk copy of its own from the interleaved x or t, straight into the
// stage.  A G2 of K columns would be written and read once more per pass: on a
// 27,648-DoF 3DR0 crack 97 MB on top of 530 MB of FP32 blocks.
//
// What bounds it: shared memory and the per-chunk round trip.  Per staged 16
// bytes a thread reads K values of the vector window (broadcasts within a column
// group, bank conflicts between groups) and issues 4 K (FP32) or 2 K (FP64) FMAs,
// which keep the FMA pipes about a third busy.  A pass of 8 columns costs 1.5 to
// 1.7 matvecs (3DR0 FP32, 27,648 DoF: 176 us, the matvec 111, the block data 83).
// K = 16 would take twice the registers and stage room and be bound by the FMAs.
// Four stages of 48 KB (K = 8) fit beside one reduction buffer.
#pragma once

#include "bw_kernels.cuh"

namespace bw {

constexpr int kMultiMax = 8;             // right-hand sides per pass

// Chunk's runs in the phase's run list (phase 2).
struct RunRange {
  int32_t first, count;
};

struct MultiArgs {
  StreamArgs s;             // data, chunks, queue, row permutation, error word
  const void *xk;           // interleaved x (K values per row), compute type
  void *tk;                 // interleaved t: phase-1 output, phase-2 source
  const GatherSeg *runs;    // phase 2: the runs of all chunks
  const RunRange *ranges;   // phase 2: each chunk's runs, in the chunks' order
  long long ldy;
  int nrhs;                 // columns of y to write (<= K)
};

template <typename S, int K> struct MultiLayout {
  using G = typename Store<S>::G;
  static_assert(Store<S>::kRows > 0, "FMA paths only");
  static constexpr int kDataBytes = kStageBytes + 32;
  // vector window: kMaxCols columns in FP32, kMaxColsFp64 in FP64
  static constexpr int kCols = sizeof(G) == 8 ? kMaxColsFp64 : kMaxCols;
  static constexpr int kGBytes = kCols * K * (int)sizeof(G);
  static constexpr int kStageSize = kDataBytes + kGBytes + (int)sizeof(Chunk);
  // partial sums of one column; the pad spreads the columns over the banks
  static constexpr int kRedPer = Store<S>::kRed + 4;
  static constexpr int kRedBytes = kRedPer * K * (int)sizeof(G);
  static constexpr int kLimit = 232448;
  static constexpr int kFit = (kLimit - kRedBytes - 256) / kStageSize;
  static constexpr int kStagesM = kFit < kStages ? kFit : kStages;
  static constexpr int kBarBytes = (2 * kStagesM + 2) * 8;
  static constexpr int kTotal = kStagesM * kStageSize + kRedBytes + kBarBytes;
  static_assert(kStageSize % 16 == 0 && kRedBytes % 16 == 0, "16-byte aligned regions");
  static_assert(kStagesM >= 3 && kTotal <= kLimit, "shared memory above the 227 KB per-CTA limit");
};

// chunk_dot (bw_kernels.cuh) for K columns: the vector values of column c are
// g[c K .. c K + K).  The same two partial sums per row and column of the
// right-hand sides, taken over the same columns in the same order.
template <typename G, int R, int K>
__device__ __forceinline__ void chunk_dot_multi(const unsigned char *base, const G *g, int hv, int rv, int c0, int c1,
                                                G (&o)[R][K]) {
  using V = typename std::conditional<sizeof(G) == 8, double2, float4>::type;
  static_assert(R * sizeof(G) == 16, "16-byte rows");
  constexpr int kPer = 16 / (int)sizeof(G);
  const V *d = reinterpret_cast<const V *>(base) + rv;
  G a[R][K], b[R][K];
#pragma unroll
  for (int r = 0; r < R; r++)
#pragma unroll
    for (int j = 0; j < K; j++) a[r][j] = b[r][j] = 0;
  auto add = [&](const V &w, int c, G(&p)[R][K]) {
    const G *e = reinterpret_cast<const G *>(&w);
    const V *gv = reinterpret_cast<const V *>(g + (long long)c * K);
#pragma unroll
    for (int q = 0; q < K / kPer; q++) {
      const V xv = gv[q];
      const G *x = reinterpret_cast<const G *>(&xv);
#pragma unroll
      for (int u = 0; u < kPer; u++)
#pragma unroll
        for (int r = 0; r < R; r++) p[r][q * kPer + u] = fma(e[r], x[u], p[r][q * kPer + u]);
    }
  };
  int c = c0;
#pragma unroll 1
  for (; c + 4 <= c1; c += 4) {
    const V w0 = d[(c + 0) * hv], w1 = d[(c + 1) * hv], w2 = d[(c + 2) * hv], w3 = d[(c + 3) * hv];
    add(w0, c, a);
    add(w1, c + 1, b);
    add(w2, c + 2, a);
    add(w3, c + 3, b);
  }
#pragma unroll 1
  for (; c < c1; c++) {
    const V w = d[c * hv];
    add(w, c, a);
  }
#pragma unroll
  for (int r = 0; r < R; r++)
#pragma unroll
    for (int j = 0; j < K; j++) o[r][j] += a[r][j] + b[r][j];
}

// Output row of an item: the row of t (phase 1) or the caller's row of y.
__device__ __forceinline__ long long multi_row(const StreamArgs &a, int row) {
  if (a.phase == 1 || !a.perm_out) return row;
  return static_cast<long long>(a.dof) * a.perm_out[row / a.dof] + (row % a.dof);
}

template <typename G, int K>
__device__ __forceinline__ void multi_store(const MultiArgs &m, long long dst, int j, G v) {
  if (m.s.phase == 1)
    static_cast<G *>(m.tk)[dst * K + j] = v;
  else if (j < m.nrhs)
    m.s.y_out[j * m.ldy + dst] = static_cast<double>(v);
}

// The CTA-wide kernel (stream_panels_kernel) with K columns: the same ring of
// stages, work queue and reduction order.  The producer's lanes issue a
// chunk's runs side by side; the next chunk's runs load meanwhile.
template <typename S, int K>
__global__ void __launch_bounds__(threads_of<S>(), 1) stream_multi_kernel(MultiArgs m) {
  using G = typename Store<S>::G;
  using L = MultiLayout<S, K>;
  constexpr int es = Store<S>::kEsize;
  constexpr int R = Store<S>::kRows;
  constexpr int kConsumerWarps = Store<S>::kWarps;
  constexpr int kConsumers = consumers_of<S>();
  constexpr int kSt = L::kStagesM;
  const StreamArgs &a = m.s;
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char *stage0 = smem;
  G *red = reinterpret_cast<G *>(smem + kSt * L::kStageSize);
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + kSt * L::kStageSize + L::kRedBytes);
  uint64_t *empty = full + kSt;
  uint64_t *redbar = empty + kSt;   // partial sums of the item written
  uint64_t *redfree = redbar + 1;   // ... and read: the buffer may be reused

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kSt; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kConsumerWarps);
    }
    mbar_init(redbar, kConsumerWarps);
    mbar_init(redfree, kConsumerWarps);
    fence_barrier_init();
  }
  __syncthreads();

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    const unsigned char *gdata = static_cast<const unsigned char *>(a.data);
    const unsigned char *gx = static_cast<const unsigned char *>(m.xk);
    const unsigned char *gt = static_cast<const unsigned char *>(m.tk);
    constexpr uint32_t kRowBytes = K * (uint32_t)sizeof(G);
    // test hook: a withheld chunk of phase 1 is never staged, so its wait runs out
    const int hold = a.phase == 1 && blockIdx.x == 0 ? a.withhold : -1;
    bool ok = true;
    int issued = 0;
    ItemQueue iq;
    iq.init(a.item_ptr, a.n_items, a.queue, lane);
    auto load_range = [&](int idx, int end) {
      return a.phase == 2 && idx < end ? m.ranges[idx] : RunRange{0, 0};
    };
    auto load_run = [&](int first, int count) {
      return lane < count ? m.runs[first + lane] : GatherSeg{0, 0, 0u, 0.f};
    };
    int bb = iq.cb;
    DescRegs cur_d;
    load_desc(a.chunks, bb + lane, iq.ce, cur_d);
    RunRange cur_r = load_range(bb + lane, iq.ce);
    int first = __shfl_sync(0xffffffffu, cur_r.first, 0), count = __shfl_sync(0xffffffffu, cur_r.count, 0);
    GatherSeg run = load_run(first, count);
    // the launch may have started before the one that writes x or t is done
    pdl_wait();
    fence_proxy_async_global();
    pdl_launch_dependents();
    while (iq.valid() && ok) {
      const int be = min(bb + 32, iq.ce);
      const bool same = be < iq.ce;
      DescRegs nxt_d;
      load_desc(a.chunks, (same ? be : iq.ncb) + lane, same ? iq.ce : iq.nce, nxt_d);
      const RunRange nxt_r = load_range((same ? be : iq.ncb) + lane, same ? iq.ce : iq.nce);
      const int nb = be - bb;
      for (int k = 0; k < nb; k++) {
        const int s = issued % kSt;
        const uint32_t use = static_cast<uint32_t>(issued / kSt);
        // the next chunk's first 32 runs, in flight while this one waits
        const int src_lane = k + 1 < nb ? k + 1 : 0;
        const int nfirst = __shfl_sync(0xffffffffu, k + 1 < nb ? cur_r.first : nxt_r.first, src_lane);
        const int ncount = __shfl_sync(0xffffffffu, k + 1 < nb ? cur_r.count : nxt_r.count, src_lane);
        const GatherSeg nrun = load_run(nfirst, ncount);
        if (!mbar_wait(&empty[s], (use & 1u) ^ 1u, a.spin_limit)) {
          if (lane == 0) set_error(a.err, kErrTimeoutEmpty);
          ok = false;
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        uint32_t w[kChunkWords];
#pragma unroll
        for (int q = 0; q < kChunkWords; q++) w[q] = __shfl_sync(0xffffffffu, cur_d.w[q], k);
        const long long data_off = static_cast<long long>((static_cast<unsigned long long>(w[1]) << 32) | w[0]);
        const int ncols = static_cast<int>(w[2]);
        const int hpad = static_cast<int>(w[3]);
        const int g_off = static_cast<int>(w[7]);
        unsigned char *st = stage0 + s * L::kStageSize;
        const unsigned long long bytes =
            static_cast<unsigned long long>(ncols > 0 ? ncols : 0) * static_cast<unsigned long long>(hpad) * es;
        bool good = ncols > 0 && ncols <= L::kCols && bytes <= static_cast<unsigned long long>(kStageBytes);
        if (good && a.phase == 2) {
          // the runs must tile the window [0, ncols) in order of their places
          int cols = 0;
          bool in = true;
          for (int q = lane; q < count; q += 32) {
            const GatherSeg r = q < 32 ? run : m.runs[first + q];
            const int c = static_cast<int>(r.cols_src & 0x7fffffffu), at = r.dst - g_off;
            in = in && c > 0 && at >= 0 && at + c <= ncols;
            cols += c;
          }
          good = __all_sync(0xffffffffu, in) && __reduce_add_sync(0xffffffffu, cols) == ncols;
        }
        if (lane == 0 && issued != hold) {
          uint4 *dd = reinterpret_cast<uint4 *>(st + L::kDataBytes + L::kGBytes);
#pragma unroll
          for (int q = 0; q < kChunkWords / 4; q++)
            dd[q] = make_uint4(w[4 * q], w[4 * q + 1], good ? w[4 * q + 2] : (q == 0 ? 0u : w[4 * q + 2]),
                               w[4 * q + 3]);
          if (good) {
            const unsigned long long src = reinterpret_cast<unsigned long long>(gdata) +
                                           static_cast<unsigned long long>(data_off) * es;
            const unsigned long long lo = src & ~15ull, hi = (src + bytes + 15ull) & ~15ull;
            mbar_arrive_expect_tx(&full[s],
                                  static_cast<uint32_t>(hi - lo) + static_cast<uint32_t>(ncols) * kRowBytes);
            bulk_g2s(st, reinterpret_cast<const void *>(lo), static_cast<uint32_t>(hi - lo), &full[s]);
            if (a.phase == 1)
              bulk_g2s(st + L::kDataBytes, gx + static_cast<unsigned long long>(g_off) * kRowBytes,
                       static_cast<uint32_t>(ncols) * kRowBytes, &full[s]);
          } else {
            if (ncols > 0) set_error(a.err, kErrBadChunk);
            mbar_arrive(&full[s]);
          }
        }
        __syncwarp();
        if (good && a.phase == 2) {
          for (int q = lane; q < count; q += 32) {
            const GatherSeg r = q < 32 ? run : m.runs[first + q];
            const unsigned char *base = (r.cols_src >> 31) ? gt : gx;
            bulk_g2s(st + L::kDataBytes + static_cast<uint32_t>(r.dst - g_off) * kRowBytes,
                     base + static_cast<unsigned long long>(r.src_off) * kRowBytes,
                     (r.cols_src & 0x7fffffffu) * kRowBytes, &full[s]);
          }
          __syncwarp();
        }
        first = nfirst;
        count = ncount;
        run = nrun;
        issued++;
      }
      if (same) {
        bb = be;
      } else {
        iq.advance(lane);
        bb = iq.cb;
      }
      cur_d = nxt_d;
      cur_r = nxt_r;
    }
    if (ok) {
      const int s = issued % kSt;
      const uint32_t use = static_cast<uint32_t>(issued / kSt);
      if (mbar_wait(&empty[s], (use & 1u) ^ 1u, a.spin_limit)) {
        if (lane == 0) {
          uint4 *dd = reinterpret_cast<uint4 *>(stage0 + s * L::kStageSize + L::kDataBytes + L::kGBytes);
          dd[0] = make_uint4(0, 0, 0, 0);
          dd[1] = make_uint4(0, 0, kEnd, 0);
          mbar_arrive(&full[s]);
        }
      } else {
        if (lane == 0) set_error(a.err, kErrTimeoutEmpty);
        ok = false;
      }
    }
    if (!ok) {
      // let the copies already in flight land before the CTA can exit
      for (int i = max(0, issued - kSt); i < issued; i++) {
        if (i == hold) continue;  // nothing in flight for it
        mbar_wait(&full[i % kSt], static_cast<uint32_t>(i / kSt) & 1u, kDrainLimitNs);
      }
    }
    if (lane == 0) {
      __threadfence();
      if (atomicAdd(&a.queue[1], 1) == static_cast<int>(gridDim.x) - 1) {
        a.queue[0] = 0;
        a.queue[1] = 0;
        __threadfence();
      }
    }
    return;
  }

  // -------------------------------------------------------------------- consumers
  pdl_wait();  // as in stream_panels_kernel: the wait limit counts from here
  const int ct = threadIdx.x - 32, cw = warp - 1;
  // phase 2 output rows of this thread: row0, row0 + kRowStep, ...; the first
  // kPre places in y are loaded at an item's first chunk
  constexpr int kRowStep = 32 * (kConsumerWarps / K), kPre = 4;
  const int row0 = (cw / K) * 32 + lane;
  long long pre_dst[kPre];
  uint32_t items = 0;
  int hv = 1, Q = 1, rv = 0, cq = 0;
  SmallDivisor by_q{0u};
  bool active = false;
  G acc[R][K];
#pragma unroll
  for (int r = 0; r < R; r++)
#pragma unroll
    for (int j = 0; j < K; j++) acc[r][j] = 0;

  for (int i = 0;; i++) {
    const int s = i % kSt;
    const uint32_t use = static_cast<uint32_t>(i / kSt);
    if (!mbar_wait(&full[s], use & 1u, a.spin_limit)) {
      if (lane == 0) set_error(a.err, kErrTimeoutFull);
      return;
    }
    const unsigned char *st = stage0 + s * L::kStageSize;
    const Chunk &d = *reinterpret_cast<const Chunk *>(st + L::kDataBytes + L::kGBytes);
    if (d.flags & kEnd) return;
    const G *gs = reinterpret_cast<const G *>(st + L::kDataBytes);
    const uint32_t flags = d.flags;
    const int ncols = d.ncols;
    const int hpad = d.hpad;
    const int rows = d.rows, out_off = d.out_off;
    if (flags & kFirst) {
      hv = hpad / R;
      Q = kConsumers / hv;
      by_q.set(Q);
      rv = ct % hv;
      cq = ct / hv;
      active = cq < Q;
#pragma unroll
      for (int r = 0; r < R; r++)
#pragma unroll
        for (int j = 0; j < K; j++) acc[r][j] = 0;
      if (a.phase == 2) {
#pragma unroll
        for (int q = 0; q < kPre; q++)
          if (row0 + q * kRowStep < rows) pre_dst[q] = multi_row(a, out_off + row0 + q * kRowStep);
      }
    }
    if (active && ncols > 0 && ncols <= L::kCols) {
      const int c0 = by_q.divide(cq * ncols), c1 = by_q.divide((cq + 1) * ncols);
      const int soff = static_cast<int>((static_cast<unsigned long long>(d.data_off) * es) & 15ull);
      chunk_dot_multi<G, R, K>(st + soff, gs, hv, rv, c0, c1, acc);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[s]);
    if (flags & kLast) {
      // one buffer: the previous item's sums have been read by every warp
      if (items > 0 && !mbar_wait(redfree, (items - 1) & 1u, a.spin_limit)) {
        if (lane == 0) set_error(a.err, kErrTimeoutReduce);
        return;
      }
      if (active) {
#pragma unroll
        for (int j = 0; j < K; j++)
#pragma unroll
          for (int r = 0; r < R; r++) red[j * L::kRedPer + cq * hpad + R * rv + r] = acc[r][j];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(redbar);
      if (!mbar_wait(redbar, items & 1u, a.spin_limit)) {
        if (lane == 0) set_error(a.err, kErrTimeoutReduce);
        return;
      }
      // every thread sums some (row, column) pairs over the Q parts, in order.
      // Phase 1: K neighbouring lanes hold one row of t, so a warp writes 32 / K
      // whole rows; phase 2: a warp holds one column, along the rows of y.
      auto total = [&](int r, int j) {
        const G *p = red + j * L::kRedPer + r;
        G sum = 0;
#pragma unroll 4
        for (int q = 0; q < Q; q++) sum += p[q * hpad];
        return sum;
      };
      if (a.phase == 1) {
        const int j = ct % K;
        for (int r = ct / K; r < rows; r += kConsumers / K)
          static_cast<G *>(m.tk)[static_cast<long long>(out_off + r) * K + j] = total(r, j);
      } else {
        const int j = cw % K;
#pragma unroll
        for (int q = 0; q < kPre; q++) {
          const int r = row0 + q * kRowStep;
          if (r < rows && j < m.nrhs) a.y_out[j * m.ldy + pre_dst[q]] = static_cast<double>(total(r, j));
        }
        for (int r = row0 + kPre * kRowStep; r < rows; r += kRowStep)
          if (j < m.nrhs) a.y_out[j * m.ldy + multi_row(a, out_off + r)] = static_cast<double>(total(r, j));
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(redfree);
      items++;
    }
  }
}

// The unstaged kernel (narrow_items_kernel: a team of warps per unit) with K
// columns, one CTA of 16 warps per SM.  A warp first notes the source row of
// each of the chunk's columns in shared memory (phase 1: the run of x starting
// at the chunk's vector offset).
template <typename S, int K>
__global__ void __launch_bounds__(32 * kNarrowWarps, 1) narrow_multi_kernel(MultiArgs m) {
  using G = typename Store<S>::G;
  using V = typename std::conditional<sizeof(G) == 8, double2, float4>::type;
  constexpr int R = 16 / (int)sizeof(G);
  constexpr int kPer = 16 / (int)sizeof(G);
  constexpr int kAhead = sizeof(G) == 8 ? 4 : 6;
  const StreamArgs &a = m.s;
  __shared__ uint32_t s_src[kNarrowWarps][kMaxCols];
  __shared__ G red[kNarrowWarps * kNarrowRows];
  __shared__ int team_unit[kNarrowWarps];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int team = a.team, tw = wid & (team - 1), w0 = wid - tw, bar = 1 + wid / team;
  auto team_sync = [&]() {
    if (team > 1)
      bar_sync(bar, 32 * team);
    else
      __syncwarp();
  };
  uint32_t *src = s_src[wid];
  const G *xk = static_cast<const G *>(m.xk), *tk = static_cast<const G *>(m.tk);
  const unsigned char *gdata = static_cast<const unsigned char *>(a.data);
  if (a.first) pdl_wait();  // as in narrow_items_kernel
  pdl_launch_dependents();
  for (;;) {
    if (tw == 0 && lane == 0) team_unit[w0] = atomicAdd(&a.queue[0], 1);
    team_sync();
    const int it = team_unit[w0];
    team_sync();
    if (it >= a.n_items) break;
    const int cb = __ldg(a.item_ptr + it), ce = __ldg(a.item_ptr + it + 1);
    G acc[R][K];
    for (int i = cb; i < ce; i++) {
      const NarrowChunk d = narrow_desc(a, i, tw == 0 && lane == 0);
      if (d.flags & kFirst) {
#pragma unroll
        for (int r = 0; r < R; r++)
#pragma unroll
          for (int j = 0; j < K; j++) acc[r][j] = 0;
      }
      __syncwarp();  // the previous chunk's sources are no longer read
      if (a.phase == 1) {
        for (int c = lane; c < d.ncols; c += 32) src[c] = static_cast<uint32_t>(d.g_off + c);
      } else {
        const RunRange rr = m.ranges[i];
        for (int q = 0; q < rr.count; q++) {
          const uint4 g = __ldg(reinterpret_cast<const uint4 *>(m.runs + rr.first + q));
          const int at = static_cast<int>(g.x) - d.g_off, cols = static_cast<int>(g.z & 0x7fffffffu);
          for (int c = lane; c < cols; c += 32)
            if (at + c >= 0 && at + c < d.ncols) src[at + c] = (g.y + c) | (g.z & 0x80000000u);
        }
      }
      __syncwarp();
      const int lpc = narrow_lpc(d.hpad, R), cpp = (32 / lpc) * team;
      const int r0 = (lane % lpc) * R;
      if (r0 < d.hpad) {
        const G *db = reinterpret_cast<const G *>(gdata + d.data_off * Store<S>::kEsize) + r0;
#pragma unroll 1
        for (int c = lane / lpc + (32 / lpc) * tw; c < d.ncols; c += kAhead * cpp) {
          V v[kAhead];
#pragma unroll
          for (int q = 0; q < kAhead; q++) {
            const int cq = c + q * cpp;
            v[q] = cq < d.ncols ? __ldg(reinterpret_cast<const V *>(db + static_cast<long long>(cq) * d.hpad)) : V{};
          }
#pragma unroll
          for (int q = 0; q < kAhead; q++) {
            const int cq = c + q * cpp;
            const G *e = reinterpret_cast<const G *>(&v[q]);
            const uint32_t sr = cq < d.ncols ? src[cq] : 0u;
            const V *xr = reinterpret_cast<const V *>(((sr >> 31) ? tk : xk) +
                                                      static_cast<long long>(sr & 0x7fffffffu) * K);
#pragma unroll
            for (int p = 0; p < K / kPer; p++) {
              const V xv = cq < d.ncols ? xr[p] : V{};
              const G *x = reinterpret_cast<const G *>(&xv);
#pragma unroll
              for (int u = 0; u < kPer; u++)
#pragma unroll
                for (int r = 0; r < R; r++) acc[r][p * kPer + u] = fma(e[r], x[u], acc[r][p * kPer + u]);
            }
          }
        }
      }
      if (d.flags & kLast) {
        for (int o = lpc; o < 32; o <<= 1)
#pragma unroll
          for (int r = 0; r < R; r++)
#pragma unroll
            for (int j = 0; j < K; j++) acc[r][j] += __shfl_xor_sync(0xffffffffu, acc[r][j], o);
        if (team == 1) {
          if (lane < lpc) {
#pragma unroll
            for (int r = 0; r < R; r++)
              if (lane * R + r < d.rows) {
                const long long dst = multi_row(a, d.out_off + lane * R + r);
#pragma unroll
                for (int j = 0; j < K; j++) multi_store<G, K>(m, dst, j, acc[r][j]);
              }
          }
        } else {
          // column by column: the warps' rows meet in red, summed in warp order
#pragma unroll
          for (int j = 0; j < K; j++) {
            if (lane < lpc) {
#pragma unroll
              for (int r = 0; r < R; r++)
                if (lane * R + r < d.hpad) red[wid * kNarrowRows + lane * R + r] = acc[r][j];
            }
            team_sync();
            for (int r = 32 * tw + lane; r < d.rows; r += 32 * team) {
              G sum = red[w0 * kNarrowRows + r];
              for (int w = 1; w < team; w++) sum += red[(w0 + w) * kNarrowRows + r];
              multi_store<G, K>(m, multi_row(a, d.out_off + r), j, sum);
            }
            team_sync();
          }
        }
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&a.queue[1], 1) == static_cast<int>(gridDim.x) - 1) {
      a.queue[0] = 0;
      a.queue[1] = 0;
      __threadfence();
    }
  }
  pdl_wait();  // as in narrow_items_kernel
}

// X (FP64, column-major, leading dimension ldx, caller's ordering) -> xk: K
// values per row in the compute type, permuted order; columns >= nrhs are zero.
template <typename G, int K>
__global__ void __launch_bounds__(256) gather_xk_kernel(const double *__restrict__ x, long long ldx, int nrhs,
                                                        G *__restrict__ xk, const int32_t *__restrict__ perm, int dof,
                                                        int n) {
  pdl_launch_dependents();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long src = perm ? static_cast<long long>(dof) * perm[i / dof] + (i % dof) : i;
  __align__(16) G v[K];
#pragma unroll
  for (int j = 0; j < K; j++) v[j] = j < nrhs ? static_cast<G>(x[j * ldx + src]) : G(0);
  uint4 *d = reinterpret_cast<uint4 *>(xk + static_cast<long long>(i) * K);
#pragma unroll
  for (int q = 0; q < K * (int)sizeof(G) / 16; q++) d[q] = reinterpret_cast<const uint4 *>(v)[q];
}

}  // namespace bw
