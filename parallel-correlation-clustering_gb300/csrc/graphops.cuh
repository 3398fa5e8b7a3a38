// graphops.cuh -- load-balanced iteration over CSR entries of a
// degree-binned vertex list.
//
// Rows are served by three kernel shapes so that no warp walks a hub row on
// its own (a 64k-entry row walked by one warp is a ~1 ms latency chain):
//   small rows (bins d <= 32):   a warp takes 32 rows and walks their entries
//                                32 at a time (warp-level load balancing);
//   mid rows (32 < d <= 1000):   one warp per row, 4 entries per lane in
//                                flight;
//   big rows (d > 1000):         one CTA of 512 threads per row.
// The functor is called as f(u, j, slot): vertex u, entry j, and a
// per-thread slot in [0, EdgeIterSlots(ctx)) for deterministic per-thread
// accumulation.
#pragma once

#include "engine.cuh"
#include "hubs.cuh"

namespace pcc {

constexpr int kIterThreads = 256;
constexpr int kIterBigThreads = 512;

inline unsigned IterSmallGrid(const Context* ctx) { return unsigned(ctx->num_sms) * 8; }
inline unsigned IterMidGrid(const Context* ctx) { return unsigned(ctx->num_sms) * 8; }
inline unsigned IterBigGrid(const Context* ctx) { return unsigned(ctx->num_sms) * 2; }
inline uint64_t EdgeIterSlots(const Context* ctx) {
  return uint64_t(IterSmallGrid(ctx)) * kIterThreads + uint64_t(IterMidGrid(ctx)) * kIterThreads +
         uint64_t(IterBigGrid(ctx)) * kIterBigThreads;
}

struct RowAll {
  __device__ bool operator()(uint32_t) const { return true; }
};

template <class F, class R>
__global__ void __launch_bounds__(kIterThreads) EdgeIterSmallKernel(const uint32_t* __restrict__ list,
                                                                   const uint32_t* __restrict__ counts,
                                                                   const uint32_t* __restrict__ starts,
                                                                   const uint64_t* __restrict__ off, F f, R row) {
  __shared__ uint32_t incl[kIterThreads / 32][32];
  __shared__ uint64_t begin[kIterThreads / 32][32];
  __shared__ uint32_t vert[kIterThreads / 32][32];
  const uint32_t s0 = starts[kBinG4];
  const uint32_t count = starts[kBinW128] - s0;  // bins G4..G32 are contiguous
  const unsigned lane = LaneId(), warp = threadIdx.x >> 5;
  const uint64_t slot = uint64_t(blockIdx.x) * kIterThreads + threadIdx.x;
  const uint64_t stride = uint64_t(gridDim.x) * kIterThreads;
  for (uint64_t i0 = (uint64_t(blockIdx.x) * (kIterThreads / 32) + warp) * 32; i0 < count; i0 += stride) {
    const uint64_t i = i0 + lane;
    uint32_t d = 0, v = 0;
    uint64_t b = 0;
    if (i < count) {
      v = list[s0 + i];
      if (row(v)) {
        b = off[v];
        d = static_cast<uint32_t>(off[v + 1] - b);
      }
    }
    const uint32_t inc = WarpInclusiveScan<uint32_t>(d);
    incl[warp][lane] = inc;
    begin[warp][lane] = b;
    vert[warp][lane] = v;
    const uint32_t total = __shfl_sync(kFull, inc, 31);
    __syncwarp();
    for (uint32_t e = lane; e < total; e += 32) {
      int lo = 0, hi = 31;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (incl[warp][mid] > e) hi = mid; else lo = mid + 1;
      }
      const uint32_t excl = lo ? incl[warp][lo - 1] : 0u;
      f(vert[warp][lo], begin[warp][lo] + (e - excl), slot);
    }
    __syncwarp();
  }
  (void)counts;
}

template <class F, class R>
__global__ void __launch_bounds__(kIterThreads) EdgeIterMidKernel(const uint32_t* __restrict__ list,
                                                                 const uint32_t* __restrict__ counts,
                                                                 const uint32_t* __restrict__ starts,
                                                                 const uint64_t* __restrict__ off, F f,
                                                                 uint64_t slot_base, R row) {
  const uint32_t s0 = starts[kBinW128];
  const uint32_t count = starts[kBinCta] - s0;  // bins W128..W1000
  const unsigned lane = LaneId(), warp = threadIdx.x >> 5;
  const uint64_t slot = slot_base + uint64_t(blockIdx.x) * kIterThreads + threadIdx.x;
  for (uint64_t i = uint64_t(blockIdx.x) * (kIterThreads / 32) + warp; i < count;
       i += uint64_t(gridDim.x) * (kIterThreads / 32)) {
    const uint32_t v = list[s0 + i];
    if (!row(v)) continue;
    const uint64_t b = off[v], e = off[v + 1];
    for (uint64_t j = b + lane; j < e; j += 128) {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (j + 32 * k < e) f(v, j + 32 * k, slot);
    }
  }
  (void)counts;
}

template <class F, class R>
__global__ void __launch_bounds__(kIterBigThreads) EdgeIterBigKernel(const uint32_t* __restrict__ list,
                                                                    const uint32_t* __restrict__ counts,
                                                                    const uint32_t* __restrict__ starts,
                                                                    const uint64_t* __restrict__ off, F f,
                                                                    uint64_t slot_base, R row) {
  const uint32_t s0 = starts[kBinCta];
  const uint32_t count = starts[kNumBins] - s0;  // bins Cta, Global
  const uint64_t slot = slot_base + uint64_t(blockIdx.x) * kIterBigThreads + threadIdx.x;
  for (uint64_t i = blockIdx.x; i < count; i += gridDim.x) {
    const uint32_t v = list[s0 + i];
    if (!row(v)) continue;
    const uint64_t b = off[v], e = off[v + 1];
    for (uint64_t j = b + threadIdx.x; j < e; j += 4 * kIterBigThreads) {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (j + uint64_t(kIterBigThreads) * k < e) f(v, j + uint64_t(kIterBigThreads) * k, slot);
    }
  }
  (void)counts;
}

// Launches the three shapes over a BinSet-layout list (starts on device);
// rows failing `row` are skipped.  host_counts (per bin) may be null; then
// every shape is launched.
template <class F, class R = RowAll>
inline void LaunchEdgeIter(Context* ctx, const uint32_t* list, const uint32_t* counts, const uint32_t* starts,
                           const uint32_t* host_counts, const uint64_t* off, F f, R row = R()) {
  auto any = [&](int b0, int b1) {
    if (!host_counts) return true;
    for (int b = b0; b < b1; ++b)
      if (host_counts[b]) return true;
    return false;
  };
  cudaStream_t st = ctx->stream;
  if (any(kBinG4, kBinW128)) {
    EdgeIterSmallKernel<F, R><<<IterSmallGrid(ctx), kIterThreads, 0, st>>>(list, counts, starts, off, f, row);
    PCC_COUNT(1);
  }
  const uint64_t base_mid = uint64_t(IterSmallGrid(ctx)) * kIterThreads;
  if (any(kBinW128, kBinCta)) {
    EdgeIterMidKernel<F, R><<<IterMidGrid(ctx), kIterThreads, 0, st>>>(list, counts, starts, off, f, base_mid, row);
    PCC_COUNT(1);
  }
  const uint64_t base_big = base_mid + uint64_t(IterMidGrid(ctx)) * kIterThreads;
  if (any(kBinCta, kNumBins)) {
    EdgeIterBigKernel<F, R><<<IterBigGrid(ctx), kIterBigThreads, 0, st>>>(list, counts, starts, off, f, base_big,
                                                                          row);
    PCC_COUNT(1);
  }
}

// ---------------------------------------------------------------------------
// The same walk with kEdgeBatch entries of a lane at a time: f(v, j) gets
// arrays of kEdgeBatch rows and entries (rows kNone where there is none) with
// every lane of the warp converged, so that it can issue all its loads before
// it stores and can combine over the warp.
// ---------------------------------------------------------------------------
constexpr int kEdgeBatch = 4;

// Rows of more than kHubSmallMax entries in pieces of kLoopChunk (HubPlan);
// without them (num 0) these rows are taken whole.
struct RowPieces {
  const uint32_t* big_v;
  const uint32_t* chunk_hub;
  const uint32_t* chunk_start;
  uint32_t num;
};
// (For callers that have had EnsureHubPlan; the others take RowPieces{}: another
// thread may be building the plan.)
inline RowPieces PiecesOf(const DevGraph& g) {
  return RowPieces{g.hub_plan->big_v, g.hub_plan->chunk_hub, g.hub_plan->chunk_start, g.hub_plan->num_chunks};
}

// The items of one CTA (pieces of the longest rows, then the rows of bin Cta):
// each thread looks up one of 256 (a chain of dependent loads, paid once), and
// then the whole CTA walks them in turn: walk(row, first entry, entries).
template <class R, class W>
__device__ __forceinline__ void ForBigItems(const uint32_t* __restrict__ list, const uint32_t* __restrict__ starts,
                                            const uint64_t* __restrict__ off, const RowPieces& c, R row, W walk) {
  __shared__ uint64_t from[kIterThreads];
  __shared__ uint32_t len[kIterThreads], vert[kIterThreads];
  const uint32_t s0 = starts[kBinCta];
  const uint64_t items = uint64_t(c.num) + (starts[c.num ? kBinGlobal : kNumBins] - s0);
  const unsigned tid = threadIdx.x;
  for (uint64_t base = blockIdx.x; base < items; base += uint64_t(gridDim.x) * kIterThreads) {
    const uint64_t it = base + uint64_t(gridDim.x) * tid;
    uint64_t b = 0;
    uint32_t n = 0, v = 0;
    if (it < items) {
      const bool piece = it < c.num;
      v = piece ? c.big_v[c.chunk_hub[it]] : list[s0 + (it - c.num)];
      const uint64_t o0 = off[v], o1 = off[v + 1];
      b = o0 + (piece ? c.chunk_start[it] : 0u);
      if (row(v)) n = static_cast<uint32_t>(piece ? min(o1 - b, uint64_t(kLoopChunk)) : o1 - b);
    }
    from[tid] = b;
    len[tid] = n;
    vert[tid] = v;
    __syncthreads();
    const uint64_t left = (items - base + gridDim.x - 1) / gridDim.x;
    const int count = left < kIterThreads ? int(left) : kIterThreads;
    for (int q = 0; q < count; ++q) walk(vert[q], from[q], len[q]);
    __syncthreads();
  }
}

template <class F, class R>
__global__ void __launch_bounds__(kIterThreads) EdgeBatchSmallKernel(const uint32_t* __restrict__ list,
                                                                    const uint32_t* __restrict__ starts,
                                                                    const uint64_t* __restrict__ off, F f, R row) {
  __shared__ uint32_t incl[kIterThreads / 32][32];
  __shared__ uint64_t begin[kIterThreads / 32][32];
  __shared__ uint32_t vert[kIterThreads / 32][32];
  const uint32_t s0 = starts[kBinG4];
  const uint32_t count = starts[kBinW128] - s0;  // bins G4..G32 are contiguous
  const unsigned lane = LaneId(), warp = threadIdx.x >> 5;
  for (uint64_t i0 = (uint64_t(blockIdx.x) * (kIterThreads / 32) + warp) * 32; i0 < count;
       i0 += uint64_t(gridDim.x) * kIterThreads) {
    const uint64_t i = i0 + lane;
    uint32_t d = 0, vl = 0;
    uint64_t b = 0;
    if (i < count) {
      vl = list[s0 + i];
      if (row(vl)) {
        b = off[vl];
        d = static_cast<uint32_t>(off[vl + 1] - b);
      }
    }
    const uint32_t inc = WarpInclusiveScan<uint32_t>(d);
    incl[warp][lane] = inc;
    begin[warp][lane] = b - (inc - d);  // of the entry e of the 32 rows: begin + e
    vert[warp][lane] = vl;
    const uint32_t total = __shfl_sync(kFull, inc, 31);
    __syncwarp();
    for (uint32_t e0 = 0; e0 < total; e0 += 32 * kEdgeBatch) {
      uint32_t v[kEdgeBatch];
      uint64_t j[kEdgeBatch];
#pragma unroll
      for (int k = 0; k < kEdgeBatch; ++k) {
        const uint32_t e = e0 + 32 * k + lane;
        int r = 0;
#pragma unroll
        for (int step = 16; step; step >>= 1)
          if (incl[warp][r + step - 1] <= e) r += step;
        v[k] = e < total ? vert[warp][r & 31] : kNone;
        j[k] = begin[warp][r & 31] + e;
      }
      f(v, j);
    }
    __syncwarp();
  }
}

template <class F, class R>
__global__ void __launch_bounds__(kIterThreads) EdgeBatchMidKernel(const uint32_t* __restrict__ list,
                                                                  const uint32_t* __restrict__ starts,
                                                                  const uint64_t* __restrict__ off, F f, R row) {
  const uint32_t s0 = starts[kBinW128];
  const uint32_t count = starts[kBinCta] - s0;  // bins W128..W1000
  const unsigned lane = LaneId(), warp = threadIdx.x >> 5;
  for (uint64_t i = uint64_t(blockIdx.x) * (kIterThreads / 32) + warp; i < count;
       i += uint64_t(gridDim.x) * (kIterThreads / 32)) {
    const uint32_t vr = list[s0 + i];
    if (!row(vr)) continue;
    const uint64_t b = off[vr], e = off[vr + 1];
    for (uint64_t j0 = b; j0 < e; j0 += 32 * kEdgeBatch) {
      uint32_t v[kEdgeBatch];
      uint64_t j[kEdgeBatch];
#pragma unroll
      for (int k = 0; k < kEdgeBatch; ++k) {
        j[k] = j0 + 32 * k + lane;
        v[k] = j[k] < e ? vr : kNone;
      }
      f(v, j);
    }
  }
}

template <class F, class R>
__global__ void __launch_bounds__(kIterThreads) EdgeBatchBigKernel(const uint32_t* __restrict__ list,
                                                                  const uint32_t* __restrict__ starts,
                                                                  const uint64_t* __restrict__ off, RowPieces c, F f,
                                                                  R row) {
  const unsigned tid = threadIdx.x;
  ForBigItems(list, starts, off, c, row, [&](uint32_t vr, uint64_t b, uint32_t len) {
    for (uint32_t e0 = 0; e0 < len; e0 += kIterThreads * kEdgeBatch) {
      uint32_t v[kEdgeBatch];
      uint64_t j[kEdgeBatch];
#pragma unroll
      for (int k = 0; k < kEdgeBatch; ++k) {
        const uint32_t e = e0 + kIterThreads * k + tid;
        j[k] = b + e;
        v[k] = e < len ? vr : kNone;
      }
      f(v, j);
    }
  });
}

template <class F, class R = RowAll>
inline void LaunchEdgeBatch(Context* ctx, const DevGraph& g, const RowPieces& pieces, F f, R row = R()) {
  const BinSet& bins = g.bins;
  const uint64_t* off = g.off.p;
  auto any = [&](int b0, int b1) {
    for (int b = b0; b < b1; ++b)
      if (bins.host_counts[b]) return true;
    return false;
  };
  const uint32_t *list = bins.list.p, *starts = bins.counts.p + kNumBins;
  cudaStream_t st = ctx->stream;
  if (any(kBinG4, kBinW128)) {
    EdgeBatchSmallKernel<F, R><<<IterSmallGrid(ctx), kIterThreads, 0, st>>>(list, starts, off, f, row);
    PCC_COUNT(1);
  }
  if (any(kBinW128, kBinCta)) {
    EdgeBatchMidKernel<F, R><<<IterMidGrid(ctx), kIterThreads, 0, st>>>(list, starts, off, f, row);
    PCC_COUNT(1);
  }
  if (any(kBinCta, kNumBins)) {
    EdgeBatchBigKernel<F, R><<<IterMidGrid(ctx), kIterThreads, 0, st>>>(list, starts, off, pieces, f, row);
    PCC_COUNT(1);
  }
}

// ---------------------------------------------------------------------------
// Frontier push (gbbs edgeMap with an always-true update): stamp[u] = value
// for every neighbour u of a row passing `row`.  The mid and big shapes load
// kPushBatch neighbour ids per thread before storing any stamp: through the
// generic functor the compiler must assume a store may alias the next id and
// keeps one load in flight.  Small rows use EdgeBatchSmallKernel.  A stamp
// already equal to the value is not stored again: hub vertices are
// neighbours of a large share of all rows, and same-address stores
// serialise at their L2 slice while the loads are served by L1.  Without hubs
// (`blind`) rows are stored without a look: the look at a line that other
// SMs write makes it travel between the dies (120,001 vertices, 1.9M entries:
// 43 us with it, 24 without).  The line is 4,096 entries a vertex, as many
// stores as can queue at one address: an RMAT graph of scale 22 takes the same
// time either way, and a star's leaves would all queue at its centre.
// ---------------------------------------------------------------------------
constexpr int kPushBatch = 8;

struct StampValue {
  uint32_t stamp;
  const RoundState* rs;  // non-null: the value comes from here
};

// Rows of the warp bins: each lane looks up one of the warp's next 32 rows (a
// chain of dependent loads, paid once), then the warp walks the marked ones.
template <class R>
__global__ void __launch_bounds__(kIterThreads) PushMidKernel(const uint32_t* __restrict__ list,
                                                             const uint32_t* __restrict__ starts,
                                                             const uint64_t* __restrict__ off,
                                                             const uint32_t* __restrict__ nbr,
                                                             uint32_t* __restrict__ stamp, StampValue sv, bool blind,
                                                             R row) {
  const uint32_t s0 = starts[kBinW128];
  const uint32_t count = starts[kBinCta] - s0;  // bins W128..W1000
  const unsigned lane = LaneId(), warp = threadIdx.x >> 5;
  const uint32_t value = StampIn(sv.rs, sv.stamp);
  const uint64_t warps = uint64_t(gridDim.x) * (kIterThreads / 32);
  for (uint64_t i0 = uint64_t(blockIdx.x) * (kIterThreads / 32) + warp; i0 < count; i0 += 32 * warps) {
    const uint64_t i = i0 + warps * lane;
    uint64_t b = 0;
    uint32_t len = 0;
    if (i < count) {
      const uint32_t v = list[s0 + i];
      if (row(v)) {
        b = off[v];
        len = static_cast<uint32_t>(off[v + 1] - b);
      }
    }
    for (unsigned left = __ballot_sync(kFull, len != 0); left; left &= left - 1) {
      const int q = __ffs(left) - 1;
      const uint64_t bq = __shfl_sync(kFull, b, q);
      const uint32_t lq = __shfl_sync(kFull, len, q);
      for (uint32_t e0 = 0; e0 < lq; e0 += 32 * kPushBatch) {
        uint32_t u[kPushBatch], cur[kPushBatch];
#pragma unroll
        for (int k = 0; k < kPushBatch; ++k) {
          const uint32_t e = e0 + 32 * k + lane;
          u[k] = e < lq ? nbr[bq + e] : kNone;
        }
#pragma unroll
        for (int k = 0; k < kPushBatch; ++k) cur[k] = u[k] == kNone ? value : blind ? ~value : stamp[u[k]];
#pragma unroll
        for (int k = 0; k < kPushBatch; ++k)
          if (cur[k] != value) stamp[u[k]] = value;
      }
    }
  }
}

// The longest rows, in pieces dealt to all CTAs.  (RMAT scale 20, largest row
// 86k entries, a CTA of 512 threads per row: 96 us a round; 11.)
template <class R>
__global__ void __launch_bounds__(kIterThreads) PushBigKernel(const uint32_t* __restrict__ list,
                                                             const uint32_t* __restrict__ starts,
                                                             const uint64_t* __restrict__ off,
                                                             const uint32_t* __restrict__ nbr,
                                                             uint32_t* __restrict__ stamp, StampValue sv,
                                                             RowPieces c, R row) {
  const uint32_t value = StampIn(sv.rs, sv.stamp);
  const unsigned tid = threadIdx.x;
  ForBigItems(list, starts, off, c, row, [&](uint32_t, uint64_t b, uint32_t len) {
    for (uint32_t e0 = 0; e0 < len; e0 += kIterThreads * kPushBatch) {
      uint32_t u[kPushBatch], cur[kPushBatch];
#pragma unroll
      for (int k = 0; k < kPushBatch; ++k) {
        const uint32_t e = e0 + kIterThreads * k + tid;
        u[k] = e < len ? nbr[b + e] : kNone;
      }
#pragma unroll
      for (int k = 0; k < kPushBatch; ++k) cur[k] = u[k] != kNone ? stamp[u[k]] : value;
#pragma unroll
      for (int k = 0; k < kPushBatch; ++k)
        if (cur[k] != value) stamp[u[k]] = value;
    }
  });
}

struct PushStampFn {
  const uint32_t* nbr;
  uint32_t* stamp;
  StampValue sv;
  bool blind;
  __device__ void operator()(const uint32_t (&v)[kEdgeBatch], const uint64_t (&j)[kEdgeBatch]) const {
    const uint32_t value = StampIn(sv.rs, sv.stamp);
    uint32_t u[kEdgeBatch], cur[kEdgeBatch];
#pragma unroll
    for (int k = 0; k < kEdgeBatch; ++k) u[k] = v[k] != kNone ? nbr[j[k]] : kNone;
#pragma unroll
    for (int k = 0; k < kEdgeBatch; ++k) cur[k] = u[k] == kNone ? value : blind ? ~value : stamp[u[k]];
#pragma unroll
    for (int k = 0; k < kEdgeBatch; ++k)
      if (cur[k] != value) stamp[u[k]] = value;
  }
};

// The push over a graph's static bins.
template <class R>
inline void LaunchPush(Context* ctx, const DevGraph& g, uint32_t* stamp, StampValue sv, R row) {
  const BinSet& bins = g.bins;
  auto any = [&](int b0, int b1) {
    for (int b = b0; b < b1; ++b)
      if (bins.host_counts[b]) return true;
    return false;
  };
  const bool blind = g.max_deg <= kHubSmallMax;
  const uint32_t *list = bins.list.p, *starts = bins.counts.p + kNumBins;
  cudaStream_t st = ctx->stream;
  if (any(kBinG4, kBinW128)) {
    EdgeBatchSmallKernel<PushStampFn, R><<<IterSmallGrid(ctx), kIterThreads, 0, st>>>(
        list, starts, g.off.p, PushStampFn{g.nbr.p, stamp, sv, blind}, row);
    PCC_COUNT(1);
  }
  if (any(kBinW128, kBinCta)) {
    PushMidKernel<R><<<IterMidGrid(ctx), kIterThreads, 0, st>>>(list, starts, g.off.p, g.nbr.p, stamp, sv, blind, row);
    PCC_COUNT(1);
  }
  if (any(kBinCta, kNumBins)) {
    PushBigKernel<R><<<IterMidGrid(ctx), kIterThreads, 0, st>>>(list, starts, g.off.p, g.nbr.p, stamp, sv,
                                                                PiecesOf(g), row);
    PCC_COUNT(1);
  }
}

// ---------------------------------------------------------------------------
// Degree binning of a vertex predicate over [0, n): count, starts, scatter.
// The order inside a bin is not specified (warp-aggregated atomics).
// ---------------------------------------------------------------------------
struct PredAll {
  __device__ bool operator()(uint32_t) const { return true; }
};
struct PredStamp {
  const uint32_t* st;
  uint32_t stamp;
  const RoundState* rs = nullptr;  // non-null: the stamp comes from here
  __device__ bool operator()(uint32_t v) const { return st[v] == StampIn(rs, stamp); }
};

// Layout of BinSet::counts: kNumBins counts, kNumBins + 1 starts, kNumBins
// cursors, then the degree sum (64 bits), the vertices binned and the largest
// degree.
constexpr int kBinCursors = 2 * kNumBins + 1;
constexpr int kBinDegSum = 32;
constexpr int kBinSize = 34;
constexpr int kBinMaxDegAt = 35;
constexpr int kBinWords = 36;
static_assert(kBinCursors + kNumBins <= kBinDegSum, "bin header");

template <class P>
__global__ void __launch_bounds__(256) BinCountKernel(uint32_t n, const uint64_t* __restrict__ off, P pred,
                                                      uint32_t* head) {
  __shared__ uint32_t sh[kNumBins];
  __shared__ unsigned long long sh_deg;
  __shared__ uint32_t sh_cnt, sh_max;
  if (threadIdx.x < kNumBins) sh[threadIdx.x] = 0;
  if (threadIdx.x == 0) {
    sh_deg = 0;
    sh_cnt = 0;
    sh_max = 0;
  }
  __syncthreads();
  uint32_t local[kNumBins];
#pragma unroll
  for (int b = 0; b < kNumBins; ++b) local[b] = 0;
  unsigned long long deg_acc = 0;
  uint32_t cnt = 0, mx = 0;
  for (uint64_t v = uint64_t(blockIdx.x) * 256 + threadIdx.x; v < n; v += uint64_t(gridDim.x) * 256) {
    if (!pred(static_cast<uint32_t>(v))) continue;
    const uint64_t d = off[v + 1] - off[v];
    const int b = BinOf(d);
#pragma unroll
    for (int q = 0; q < kNumBins; ++q) local[q] += (q == b);
    deg_acc += d;
    mx = max(mx, static_cast<uint32_t>(d));
    cnt++;
  }
#pragma unroll
  for (int q = 0; q < kNumBins; ++q)
    if (local[q]) atomicAdd(&sh[q], local[q]);
  if (deg_acc) atomicAdd(&sh_deg, deg_acc);
  if (cnt) atomicAdd(&sh_cnt, cnt);
  if (mx) atomicMax(&sh_max, mx);
  __syncthreads();
  if (threadIdx.x < kNumBins && sh[threadIdx.x]) atomicAdd(&head[threadIdx.x], sh[threadIdx.x]);
  if (threadIdx.x == 0) {
    if (sh_deg) atomicAdd(reinterpret_cast<unsigned long long*>(head + kBinDegSum), sh_deg);
    if (sh_cnt) atomicAdd(head + kBinSize, sh_cnt);
    if (sh_max) atomicMax(head + kBinMaxDegAt, sh_max);
  }
}

// Number and degree sum of the vertices satisfying pred (one pass over n).
template <class P, class CountT = uint32_t>
__global__ void __launch_bounds__(256) CountDegreesKernel(uint32_t n, const uint64_t* __restrict__ off, P pred,
                                                          unsigned long long* deg_sum, CountT* vcount) {
  unsigned long long dacc = 0;
  CountT cnt = 0;
  for (uint64_t v = uint64_t(blockIdx.x) * 256 + threadIdx.x; v < n; v += uint64_t(gridDim.x) * 256) {
    if (!pred(static_cast<uint32_t>(v))) continue;
    dacc += off[v + 1] - off[v];
    cnt++;
  }
  for (int o = 16; o >= 1; o >>= 1) {
    dacc += __shfl_xor_sync(kFull, dacc, o);
    cnt += __shfl_xor_sync(kFull, cnt, o);
  }
  __shared__ unsigned long long sd[8];
  __shared__ CountT sc[8];
  if (LaneId() == 0) {
    sd[threadIdx.x >> 5] = dacc;
    sc[threadIdx.x >> 5] = cnt;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
    CountT c = 0;
    for (int w = 0; w < 8; ++w) {
      t += sd[w];
      c += sc[w];
    }
    if (t) atomicAdd(deg_sum, t);
    if (c) atomicAdd(vcount, c);
  }
}

// Writes the binned vertices to the list; every block derives the starts from
// the counts, block 0 stores them.
template <class P>
__global__ void __launch_bounds__(256) BinScatterKernel(uint32_t n, const uint64_t* __restrict__ off, P pred,
                                                        uint32_t* head, uint32_t* list) {
  __shared__ uint32_t starts[kNumBins + 1];
  if (threadIdx.x == 0) {
    uint32_t acc = 0;
    for (int b = 0; b < kNumBins; ++b) {
      starts[b] = acc;
      acc += head[b];
    }
    starts[kNumBins] = acc;
  }
  __syncthreads();
  if (blockIdx.x == 0 && threadIdx.x <= kNumBins) head[kNumBins + threadIdx.x] = starts[threadIdx.x];
  uint32_t* cursor = head + kBinCursors;
  const uint64_t stride = uint64_t(gridDim.x) * 256;
  const uint64_t limit = (uint64_t(n) + 31) & ~uint64_t(31);
  for (uint64_t v = uint64_t(blockIdx.x) * 256 + threadIdx.x; v < limit; v += stride) {
    const bool in = v < n && pred(static_cast<uint32_t>(v));
    const int bin = in ? BinOf(off[v + 1] - off[v]) : kNumBins + int(LaneId());
    const unsigned peers = __match_any_sync(kFull, bin);
    uint32_t base = 0;
    const int leader = __ffs(peers) - 1;
    if (in && int(LaneId()) == leader) base = atomicAdd(&cursor[bin], uint32_t(__popc(peers)));
    base = __shfl_sync(kFull, base, leader);
    if (in) list[starts[bin] + base + __popc(peers & LaneMaskLt())] = static_cast<uint32_t>(v);
  }
}

// Bins the vertices of [0, n) that satisfy pred into b.
template <class P>
Status BinVertices(Context* ctx, uint32_t n, const uint64_t* off, P pred, BinSet* b) {
  PCC_RETURN_IF_ERROR(b->list.Reserve(ctx, std::max<uint64_t>(n, 1)));
  PCC_RETURN_IF_ERROR(b->counts.Reserve(ctx, kBinWords));
  PCC_CUDA(cudaMemsetAsync(b->counts.p, 0, sizeof(uint32_t) * kBinWords, ctx->stream));
  const unsigned grid = Blocks(n, 256, unsigned(ctx->num_sms) * 16);
  if (n) {
    BinCountKernel<P><<<grid, 256, 0, ctx->stream>>>(n, off, pred, b->counts.p);
    BinScatterKernel<P><<<grid, 256, 0, ctx->stream>>>(n, off, pred, b->counts.p, b->list.p);
    PCC_COUNT(2);
  }
  return LaunchCheck();
}

}  // namespace pcc
