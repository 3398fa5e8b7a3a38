// bestmove.cu -- degree-binned best-move kernels.
//
// Restates ClusteringHelper::EfficientBestMove
// (clustering/clusterers/parallel-correlation-clusterer-internal.cc:448-583)
// with EdgeSum (correlation-clusterer-util.h:26-43), the sync decision of
// BestMovesForVertexSubset (parallel-correlation-clusterer.cc:139-157) and
// AsyncMove (parallel-correlation-clusterer-internal.cc:371-403).
//
// For vertex v in cluster c with node weight kv, over neighbours u != v:
//   S_D    = sum over neighbours in cluster D of (w - offset)
//   T      = S_c
//   change = 0 - (T - res * (kv * (K_c - kv)))
//   val_D  = change + (S_D - res * (kv * K_D))
// The chosen move is argmax_D val_D (ties -> lowest D), unless change >= max
// val, in which case it is "new cluster" (target n, value change).  Every
// operation is a separately rounded IEEE double op (no FMA), as in the
// reference.
//
// Accumulation of S_D:
//   INT mode  (SumMode::exact, engine.cuh): exact integer sums of fixed-point
//             units, so any order gives the reference's doubles.
//   FP64 mode: degree <= 1000 adds in adjacency order (the reference's
//             sequential flat_hash_map path, bit-exact); hubs add in any
//             order, as the reference's concurrent map does.
#include "certmoves.cuh"

namespace pcc {

namespace {

// ---------------------------------------------------------------------------
// Lane groups of G lanes, one vertex per group, degree <= G (one chunk).
// Equal cluster ids inside the group are found with match.any; the group
// leader of each id sums its peers in lane (= adjacency) order.
// ---------------------------------------------------------------------------
template <int G, bool kInt, bool kAsync>
__global__ void __launch_bounds__(256) BestMoveGroupKernel(BMArgs a, const uint32_t* __restrict__ list,
                                                          const uint32_t* __restrict__ bin_counts,
                                                          const uint32_t* __restrict__ bin_starts, int bin) {
  __shared__ double stage[8][32];
  __shared__ uint32_t mover_buf[8][64];
  WarpMoverBuffer mb{mover_buf[threadIdx.x >> 5]};
  const uint32_t count = bin_counts[bin];
  const uint32_t start = bin_starts[bin];
  const unsigned lane = LaneId(), warp = threadIdx.x >> 5;
  constexpr unsigned kVpw = 32 / G;
  const unsigned g = lane / G, gl = lane % G;
  const unsigned gmask = G == 32 ? kFull : (((1u << G) - 1u) << (g * G));
  unsigned long long fam_e = 0, fam_v = 0;
  const uint64_t stride = uint64_t(gridDim.x) * 8 * kVpw;
  // Vertex ids are loaded one iteration ahead (latency-bound kernel).
  uint64_t base = (uint64_t(blockIdx.x) * 8 + warp) * kVpw;
  uint32_t vid = base + g < count ? list[start + base + g] : 0u;
  for (; base < count; base += stride) {
    const uint64_t idx = base + g;
    const uint32_t nvid = base + stride + g < count ? list[start + base + stride + g] : 0u;
    bool vvalid = idx < count;
    VertexCtx x{};
    if (vvalid) {
      vvalid = InFront(a, vid);
      if (vvalid) x = LoadVertex<kAsync>(a, vid);
    }
    vid = nvid;
    if (__ballot_sync(kFull, vvalid) == 0) continue;
    if (vvalid && gl == 0) {
      fam_e += x.d;
      fam_v += 1;
    }  // no frontier vertex in this warp
    const bool has = vvalid && gl < x.d;
    uint32_t u = x.v;
    float wt = 0.f;
    if (has) {
      u = a.nbr[x.b + gl];
      wt = a.w ? a.w[x.b + gl] : 1.0f;
    }
    const bool cand = has && u != x.v;
    const uint32_t cu = cand ? LdC<kAsync>(a.C + u) : kNone;
    const unsigned peers = __match_any_sync(kFull, cand ? cu : LaneSentinel(lane)) & gmask;
    const bool leader = cand && int(lane) == __ffs(peers) - 1;
    double S;
    if (kInt) {
      const int xi = cand ? (WeightToInt(wt) - a.ioffset) : 0;
      S = static_cast<double>(GroupSumInt<int>(peers, xi, a.w == nullptr, leader, reinterpret_cast<int*>(stage[warp])));
    } else {
      stage[warp][lane] = cand ? Dsub(static_cast<double>(wt), a.offset) : 0.0;
      __syncwarp();
      S = 0.0;
      if (leader) {
        unsigned mm = peers;
        while (mm) {
          const int j = __ffs(mm) - 1;
          S = Dadd(S, stage[warp][j]);
          mm &= mm - 1;
        }
      }
      __syncwarp();
    }
    const unsigned tmask = __ballot_sync(kFull, leader && cu == x.c) & gmask;
    const double Tsh = __shfl_sync(kFull, S, tmask ? __ffs(tmask) - 1 : int(lane));
    const double T = tmask ? Tsh : 0.0;
    const double change = ChangeOf(a, x, T);
    double val = -CUDART_INF;
    uint32_t id = kNone;
    if (leader) {
      val = ValOf(a, x, change, S, LdK<kAsync>(a.K + cu));
      id = cu;
    }
#pragma unroll
    for (int o = G / 2; o >= 1; o >>= 1) {
      const double ov = __shfl_xor_sync(kFull, val, o);
      const uint32_t oid = __shfl_xor_sync(kFull, id, o);
      if (Better(ov, oid, val, id)) {
        val = ov;
        id = oid;
      }
    }
    bool append = false;
    if (vvalid && gl == 0) append = Decide<kAsync>(a, x, val, id, change, StampIn(a.rs, a.stamp));
    if (!kAsync) mb.Add(&a.ctr->movers, a.movers, append, x.v);
  }
  if (!kAsync) mb.Flush(&a.ctr->movers, a.movers);
  FlushFamily(a, kFamGroup, fam_e, fam_v);
}

// ---------------------------------------------------------------------------
// One warp per vertex, degree <= 1000, shared-memory hash of HC slots.
// Chunks of 32 entries in adjacency order; per chunk the leader of each
// cluster id adds its peers one by one (FP64) onto the slot's running sum,
// which keeps the reference's adjacency-order summation exactly.
// ---------------------------------------------------------------------------
constexpr int kWarpKernelWarps = 4;

template <int HC>
constexpr size_t WarpKernelSmem() {
  // per warp: vals HC*8, keys HC*4, used HC/2 * 2, stage 32*8, count 16
  return size_t(kWarpKernelWarps) * (size_t(HC) * 13 + 32 * 8 + 16);
}

template <int HC, bool kInt, bool kAsync>
__global__ void __launch_bounds__(kWarpKernelWarps * 32) BestMoveWarpKernel(BMArgs a,
                                                                           const uint32_t* __restrict__ list,
                                                                           const uint32_t* __restrict__ bin_counts,
                                                                           const uint32_t* __restrict__ bin_starts,
                                                                           int bin) {
  __shared__ uint32_t mover_buf[kWarpKernelWarps][64];
  WarpMoverBuffer mb{mover_buf[threadIdx.x >> 5]};
  extern __shared__ __align__(16) unsigned char smem[];
  const uint32_t count = bin_counts[bin];
  const uint32_t start = bin_starts[bin];
  const unsigned lane = LaneId(), warp = threadIdx.x >> 5;
  unsigned char* base = smem + size_t(warp) * (size_t(HC) * 13 + 32 * 8 + 16);
  unsigned long long* vals = reinterpret_cast<unsigned long long*>(base);
  uint32_t* keys = reinterpret_cast<uint32_t*>(base + size_t(HC) * 8);
  double* stage = reinterpret_cast<double*>(base + size_t(HC) * 12);
  uint16_t* used = reinterpret_cast<uint16_t*>(base + size_t(HC) * 12 + 32 * 8);
  uint32_t* used_count = reinterpret_cast<uint32_t*>(base + size_t(HC) * 13 + 32 * 8);
  unsigned long long fam_e = 0, fam_v = 0;
  for (int i = lane; i < HC; i += 32) {
    keys[i] = kNone;
    vals[i] = 0ull;
  }
  if (lane == 0) *used_count = 0;
  __syncwarp();
  // The next vertex id is loaded one iteration ahead and each vertex's
  // entries kCertUnroll chunks at a time (the loads of the chunks are in
  // flight together; the sums still run chunk by chunk, in adjacency order).
  const uint64_t wstride = uint64_t(gridDim.x) * kWarpKernelWarps;
  uint64_t idx = uint64_t(blockIdx.x) * kWarpKernelWarps + warp;
  uint32_t vid = idx < count ? list[start + idx] : 0u;
  for (; idx < count; idx += wstride) {
    const uint64_t nidx = idx + wstride;
    const uint32_t nvid = nidx < count ? list[start + nidx] : 0u;
    if (!InFront(a, vid)) {
      vid = nvid;
      continue;
    }
    const VertexCtx x = LoadVertex<kAsync>(a, vid);
    vid = nvid;
    if (lane == 0) {
      fam_e += x.d;
      fam_v += 1;
    }
    for (uint32_t e00 = 0; e00 < x.d; e00 += 32 * kCertUnroll) {
      uint32_t uu[kCertUnroll], cc[kCertUnroll];
      float ww[kCertUnroll];
#pragma unroll
      for (int k = 0; k < kCertUnroll; ++k) {
        const uint32_t e = e00 + 32 * k + lane;
        uu[k] = x.v;
        ww[k] = 0.f;
        if (e < x.d) {
          uu[k] = a.nbr[x.b + e];
          ww[k] = a.w ? a.w[x.b + e] : 1.0f;
        }
      }
#pragma unroll
      for (int k = 0; k < kCertUnroll; ++k) cc[k] = uu[k] != x.v ? LdC<kAsync>(a.C + uu[k]) : kNone;
#pragma unroll
      for (int k = 0; k < kCertUnroll; ++k) {
      if (e00 + 32 * k >= x.d) break;  // warp-uniform
      const uint32_t u = uu[k];
      const float wt = ww[k];
      const bool cand = u != x.v;
      const uint32_t cu = cc[k];
      const unsigned peers = __match_any_sync(kFull, cand ? cu : LaneSentinel(lane));
      const bool leader = cand && int(lane) == __ffs(peers) - 1;
      uint32_t slot = kNone;
      bool ins = false;
      if (leader) {
        slot = FindOrInsertT<false>(keys, HC, cu, &ins);
        if (slot == kNone) atomicExch(&a.ctr->error, kErrHashFull);
      }
      const unsigned im = __ballot_sync(kFull, ins);
      if (im) {
        uint32_t base = 0;
        const int ld = __ffs(im) - 1;
        if (int(lane) == ld) base = atomicAdd(used_count, uint32_t(__popc(im)));
        base = __shfl_sync(kFull, base, ld);
        if (ins) used[base + __popc(im & LaneMaskLt())] = static_cast<uint16_t>(slot);
      }
      if (kInt) {
        const int xi = cand ? (WeightToInt(wt) - a.ioffset) : 0;
        const int S = GroupSumInt<int>(peers, xi, a.w == nullptr, leader, reinterpret_cast<int*>(stage));
        if (slot != kNone) vals[slot] += static_cast<unsigned long long>(static_cast<long long>(S));
      } else {
        stage[lane] = cand ? Dsub(static_cast<double>(wt), a.offset) : 0.0;
        __syncwarp();
        if (slot != kNone) {
          double acc = __longlong_as_double(static_cast<long long>(vals[slot]));
          unsigned mm = peers;
          while (mm) {
            const int j = __ffs(mm) - 1;
            acc = Dadd(acc, stage[j]);
            mm &= mm - 1;
          }
          vals[slot] = static_cast<unsigned long long>(__double_as_longlong(acc));
        }
      }
      __syncwarp();
      }
    }
    double T = 0.0;
    if (lane == 0) {
      const uint32_t slot = FindT<false>(keys, HC, x.c);
      if (slot != kNone) T = AsDouble<kInt>(vals[slot]);
    }
    T = __shfl_sync(kFull, T, 0);
    const double change = ChangeOf(a, x, T);
    const uint32_t nused = *used_count;
    double best = -CUDART_INF;
    uint32_t bid = kNone;
    for (uint32_t i = lane; i < nused; i += 32) {
      const uint32_t slot = used[i];
      const uint32_t key = keys[slot];
      const double S = AsDouble<kInt>(vals[slot]);
      const double val = ValOf(a, x, change, S, LdK<kAsync>(a.K + key));
      if (Better(val, key, best, bid)) {
        best = val;
        bid = key;
      }
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
      const double ov = __shfl_xor_sync(kFull, best, o);
      const uint32_t oid = __shfl_xor_sync(kFull, bid, o);
      if (Better(ov, oid, best, bid)) {
        best = ov;
        bid = oid;
      }
    }
    __syncwarp();
    for (uint32_t i = lane; i < nused; i += 32) {
      const uint32_t slot = used[i];
      keys[slot] = kNone;
      vals[slot] = 0ull;
    }
    bool append = false;
    if (lane == 0) append = Decide<kAsync>(a, x, best, bid, change, StampIn(a.rs, a.stamp));
    if (!kAsync) mb.Add(&a.ctr->movers, a.movers, append, x.v);
    __syncwarp();
    if (lane == 0) *used_count = 0;
    __syncwarp();
  }
  if (!kAsync) mb.Flush(&a.ctr->movers, a.movers);
  FlushFamily(a, kFamWarp, fam_e, fam_v);
}

// ---------------------------------------------------------------------------
// INT-mode synchronous rounds: the certified bodies of certmoves.cuh over one
// degree bin each.
// ---------------------------------------------------------------------------
template <int G, typename V>
__global__ void __launch_bounds__(256, 4) CertGroupKernel(BMArgs a, const uint32_t* __restrict__ list,
                                                      const uint32_t* __restrict__ bin_counts,
                                                      const uint32_t* __restrict__ bin_starts, int bin) {
  __shared__ V stage[8][32];
  __shared__ uint32_t mover_buf[8][64];
  WarpMoverBuffer mb{mover_buf[threadIdx.x >> 5]};
  const uint32_t count = bin_counts[bin];
  const uint32_t start = bin_starts[bin];
  const unsigned warp = threadIdx.x >> 5;
  constexpr unsigned kVpw = 32 / G;
  const unsigned g = LaneId() / G;
  uint32_t fam_e = 0, fam_v = 0;
  const bool replay = a.out_target != nullptr;
  const RoundView rv = RoundOf(a);
  Pending<V> pend;
  auto exact = [&](uint32_t v, int cres, uint32_t cmove) {
    return GroupExact<V, ConstLoads>(a, rv, v, cres, cmove);
  };
  const uint64_t stride = uint64_t(gridDim.x) * 8 * kVpw;
  // The next step's rows are loaded during this one, their ids one step
  // before that (latency-bound kernel).
  uint64_t base = (uint64_t(blockIdx.x) * 8 + warp) * kVpw;
  auto id_at = [&](uint64_t i) { return i < count ? list[start + i] : 0u; };
  GroupRow row, next;
  GroupHead<ConstLoads>(a, rv, base + g < count, id_at(base + g), row);
  GroupEntry<G>(a, row);
  uint32_t vid = id_at(base + stride + g);
  while (true) {
    const bool more = base < count;
    if (!more || pend.n + kVpw > 32) DecidePending<V, ConstLoads>(a, rv, pend, replay, mb, &a.ctr->movers, exact);
    if (!more) break;
    base += stride;
    GroupHead<ConstLoads>(a, rv, base + g < count, vid, next);
    vid = id_at(base + stride + g);
    GroupScan<G, V, ConstLoads>(a, row, stage[warp], pend, fam_e, fam_v, [&] { GroupEntry<G>(a, next); });
    row = next;
  }
  mb.Flush(&a.ctr->movers, a.movers);
  FlushFamily(a, kFamGroup, fam_e, fam_v);
}

// Per-warp shared bytes: vals HC*sizeof(V), keys HC*4, stage 32*4, used
// HC/2 * 2, count 16.
template <int HC, typename V>
__host__ __device__ constexpr size_t CertWarpStride() {
  return size_t(HC) * (sizeof(V) + 5) + 32 * 4 + 16;
}
template <int HC, typename V>
constexpr size_t CertWarpSmem() {
  return size_t(kWarpKernelWarps) * CertWarpStride<HC, V>();
}

template <int HC, typename V, bool kConv = sizeof(V) == 8>
__global__ void __launch_bounds__(kWarpKernelWarps * 32, 9) CertWarpKernel(BMArgs a, const uint32_t* __restrict__ list,
                                                                       const uint32_t* __restrict__ bin_counts,
                                                                       const uint32_t* __restrict__ bin_starts,
                                                                       int bin) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint32_t mover_buf[kWarpKernelWarps][64];
  WarpMoverBuffer mb{mover_buf[threadIdx.x >> 5]};
  const uint32_t count = bin_counts[bin];
  const uint32_t start = bin_starts[bin];
  const unsigned lane = LaneId(), warp = threadIdx.x >> 5;
  unsigned char* base = smem + size_t(warp) * CertWarpStride<HC, V>();
  V* vals = reinterpret_cast<V*>(base);
  uint32_t* keys = reinterpret_cast<uint32_t*>(base + size_t(HC) * sizeof(V));
  uint16_t* used = reinterpret_cast<uint16_t*>(base + size_t(HC) * (sizeof(V) + 4) + 32 * 4);
  unsigned long long fam_e = 0, fam_v = 0;
  const bool replay = a.out_target != nullptr;
  const RoundView rv = RoundOf(a);
  for (int i = lane; i < HC; i += 32) {
    keys[i] = kNone;
    vals[i] = 0;
  }
  __syncwarp();
  // The next vertex id is loaded one iteration ahead, and each vertex's
  // entries are loaded kCertUnroll chunks at a time (up to 128 neighbour ids
  // and their cluster ids in flight per warp): the kernel is bound by the
  // latency of the dependent loads list -> offsets -> neighbours -> clusters.
  const uint64_t wstride = uint64_t(gridDim.x) * kWarpKernelWarps;
  uint64_t idx = uint64_t(blockIdx.x) * kWarpKernelWarps + warp;
  uint32_t vid = idx < count ? list[start + idx] : 0u;
  for (; idx < count; idx += wstride) {
    const uint64_t nidx = idx + wstride;
    const uint32_t nvid = nidx < count ? list[start + nidx] : 0u;
    if (!InFront(a, rv, vid)) {
      vid = nvid;
      continue;
    }
    const VertexCtx x = LoadVertexAs<ConstLoads>(a, vid);
    vid = nvid;
    if (lane == 0) {
      fam_e += x.d;
      fam_v += 1;
    }
    const bool append = WarpStep<HC, V, kConv, ConstLoads>(a, rv, x, vals, keys, used, replay);
    mb.Add(&a.ctr->movers, a.movers, append, x.v);
    __syncwarp();
  }
  mb.Flush(&a.ctr->movers, a.movers);
  FlushFamily(a, kFamWarp, fam_e, fam_v);
}

// ---------------------------------------------------------------------------
// One CTA of kCtaWarps warps per vertex (degree 129-1000, INT mode, sync):
// the same certified decision as CertWarpKernel, with the row and the
// epilogue split over the CTA's warps.  One table of HC slots per CTA
// instead of one per warp, so several times more vertices are in flight per
// SM for the same shared memory, and each vertex's chain of dependent loads
// and candidate loops is kCtaWarps times shorter.  Inserts claim slots with
// atomicCAS and add with shared-memory atomics (any order: INT-mode sums
// are exact); the warp maxima and lexicographic leaders are combined through
// shared memory.  An uncertain (or replayed) vertex takes WarpExact on warp 0
// over the whole table, exactly as in the warp kernel.
// ---------------------------------------------------------------------------
template <int HC, typename V>
constexpr size_t CertCtaSmem() {
  return size_t(HC) * (sizeof(V) + 4 + 2);  // vals, keys, used
}

template <int HC, typename V, bool kConv = sizeof(V) == 8>
__global__ void __launch_bounds__(kCtaWarps * 32) CertCtaKernel(BMArgs a, const uint32_t* __restrict__ list,
                                                               const uint32_t* __restrict__ bin_counts,
                                                               const uint32_t* __restrict__ bin_starts, int bin) {
  constexpr int BT = kCtaWarps * 32;
  extern __shared__ __align__(16) unsigned char smem[];
  V* vals = reinterpret_cast<V*>(smem);
  uint32_t* keys = reinterpret_cast<uint32_t*>(smem + size_t(HC) * sizeof(V));
  uint16_t* used = reinterpret_cast<uint16_t*>(smem + size_t(HC) * (sizeof(V) + 4));
  __shared__ CtaShared<V> sh;
  __shared__ uint32_t mover_buf[64];  // warp 0's
  WarpMoverBuffer mb{mover_buf};
  const uint32_t count = bin_counts[bin];
  const uint32_t start = bin_starts[bin];
  const unsigned tid = threadIdx.x, warp = tid >> 5;
  unsigned long long fam_e = 0, fam_v = 0;
  const bool replay = a.out_target != nullptr;
  const RoundView rv = RoundOf(a);
  for (int i = tid; i < HC; i += BT) {
    keys[i] = kNone;
    vals[i] = 0;
  }
  if (tid == 0) sh.nused = 0;
  __syncthreads();
  uint32_t vid = blockIdx.x < count ? list[start + blockIdx.x] : 0u;
  for (uint64_t idx = blockIdx.x; idx < count; idx += gridDim.x) {
    const uint64_t nidx = idx + gridDim.x;
    const uint32_t nvid = nidx < count ? list[start + nidx] : 0u;
    if (!InFront(a, rv, vid)) {  // uniform over the CTA
      vid = nvid;
      continue;
    }
    const VertexCtx x = LoadVertexAs<ConstLoads>(a, vid);
    vid = nvid;
    if (tid == 0) {
      fam_e += x.d;
      fam_v += 1;
    }
    const bool append = CtaStep<HC, V, kConv, ConstLoads>(a, rv, x, vals, keys, used, sh, tid, 0, replay);
    if (warp == 0) mb.Add(&a.ctr->movers, a.movers, append, x.v);
  }
  if (warp == 0) {
    mb.Flush(&a.ctr->movers, a.movers);
    FlushFamily(a, kFamWarp, fam_e, fam_v);
  }
}

// (Each kernel is launched with one fixed shared-memory size.)
template <class K>
Status SetSmem(K kernel, size_t bytes, int threads, int* per_sm) {
  return PrepareKernel(kernel, threads, bytes, bytes, per_sm);
}

template <bool kInt, bool kAsync>
Status LaunchAll(Context* ctx, const BMArgs& a, const uint32_t* list, const uint32_t* counts,
                 const uint32_t* starts, const uint32_t* host_counts, uint32_t max_deg, int families) {
  const unsigned sms = unsigned(ctx->num_sms);
  const LaunchTuning tune = TuningFor(ctx, a.n);
  // Resident CTAs of one wave scaled by the tuned wave count.
  auto waves = [&](unsigned one_wave) -> unsigned {
    return std::max(1u, unsigned(double(one_wave) * double(tune.grid_waves) + 0.5));
  };
  auto grid = [&](int bin, uint64_t per_block, unsigned cap) -> unsigned {
    if (!host_counts) return cap;
    return Blocks(host_counts[bin], unsigned(per_block), cap);
  };
  // Warp bins above the tuned degree run one CTA per vertex (INT mode).
  auto on_cta = [&](int bin) {
    return bin >= kBinW128 && bin <= kBinW1000 && kBinMaxDeg[bin] > tune.cta_min_degree;
  };
  // Lane-group bins above the tuned degree run on the 256-slot warp kernel,
  // as part of the warp family (launched, timed and counted with it).
  auto routed = [&](int bin) { return bin <= kBinG32 && kBinMaxDeg[bin] > tune.group_max_degree; };
  auto want = [&](int bin) {
    const int fam = bin <= kBinG32 && !routed(bin) ? kLaunchGroups : kLaunchWarps;
    return (families & fam) && (!host_counts || host_counts[bin] > 0);
  };
  cudaStream_t st = ctx->stream;
  constexpr bool kCert = kInt && !kAsync;
  // Grid-stride kernels: at most one wave of resident CTAs, so no partial
  // last wave.
  auto warp_bin = [&](auto k, size_t smem, int bin, unsigned cap) -> Status {
    if (!want(bin)) return Status::Ok();
    int per_sm = 0;
    PCC_RETURN_IF_ERROR(SetSmem(k, smem, kWarpKernelWarps * 32, &per_sm));
    if (per_sm > 0) cap = sms * unsigned(per_sm);
    k<<<grid(bin, kWarpKernelWarps, waves(cap)), kWarpKernelWarps * 32, smem, st>>>(a, list, counts, starts, bin);
    PCC_COUNT(1);
    return Status::Ok();
  };
  auto cta_bin = [&](auto k, size_t smem, int bin) -> Status {
    if (!want(bin)) return Status::Ok();
    int per_sm = 0;
    PCC_RETURN_IF_ERROR(SetSmem(k, smem, kCtaWarps * 32, &per_sm));
    const unsigned cap = sms * unsigned(per_sm > 0 ? per_sm : 4);
    k<<<grid(bin, 1, waves(cap)), kCtaWarps * 32, smem, st>>>(a, list, counts, starts, bin);
    PCC_COUNT(1);
    return Status::Ok();
  };
  // A certified warp bin on the warp kernel or, above the tuned degree, the
  // CTA kernel of the same table size.
  auto cert_bin = [&](auto kw, size_t smem_w, auto kc, size_t smem_c, int bin, unsigned cap) -> Status {
    return on_cta(bin) ? cta_bin(kc, smem_c, bin) : warp_bin(kw, smem_w, bin, cap);
  };
  // The routed lane-group bins, on the warp kernel of the smallest table.
  auto routed_bins = [&](auto k, size_t smem, unsigned cap) -> Status {
    for (int b = kBinG4; b <= kBinG32; ++b)
      if (routed(b)) PCC_RETURN_IF_ERROR(warp_bin(k, smem, b, cap));
    return Status::Ok();
  };
  int ng = 0;
  for (int b = kBinG4; b <= kBinG32; ++b) ng += want(b) && !routed(b) ? 1 : 0;
  if (families & kLaunchGroups) FamBegin(ctx, kFamGroup);
  if constexpr (kCert) {
    // One wave of resident CTAs (grid-stride kernels).
    auto group_bin = [&](auto k, int bin, uint64_t per_block) -> Status {
      if (!want(bin) || routed(bin)) return Status::Ok();
      int per_sm = 0;
      PCC_RETURN_IF_ERROR(SetSmem(k, 0, 256, &per_sm));
      k<<<grid(bin, per_block, waves(sms * unsigned(per_sm > 0 ? per_sm : 8))), 256, 0, st>>>(a, list, counts, starts,
                                                                                          bin);
      PCC_COUNT(1);
      return Status::Ok();
    };
    if (a.narrow || !a.conv) {  // 32 entries of at most 2^22 always fit
      PCC_RETURN_IF_ERROR(group_bin(CertGroupKernel<4, int>, kBinG4, 64));
      PCC_RETURN_IF_ERROR(group_bin(CertGroupKernel<8, int>, kBinG8, 32));
      PCC_RETURN_IF_ERROR(group_bin(CertGroupKernel<16, int>, kBinG16, 16));
      PCC_RETURN_IF_ERROR(group_bin(CertGroupKernel<32, int>, kBinG32, 8));
    } else {
      PCC_RETURN_IF_ERROR(group_bin(CertGroupKernel<4, long long>, kBinG4, 64));
      PCC_RETURN_IF_ERROR(group_bin(CertGroupKernel<8, long long>, kBinG8, 32));
      PCC_RETURN_IF_ERROR(group_bin(CertGroupKernel<16, long long>, kBinG16, 16));
      PCC_RETURN_IF_ERROR(group_bin(CertGroupKernel<32, long long>, kBinG32, 8));
    }
  } else {
    if (want(kBinG4) && !routed(kBinG4)) {
      BestMoveGroupKernel<4, kInt, kAsync><<<grid(kBinG4, 64, waves(sms * 8)), 256, 0, st>>>(a, list, counts, starts,
                                                                                            kBinG4);
      PCC_COUNT(1);
    }
    if (want(kBinG8) && !routed(kBinG8)) {
      BestMoveGroupKernel<8, kInt, kAsync><<<grid(kBinG8, 32, waves(sms * 8)), 256, 0, st>>>(a, list, counts, starts,
                                                                                            kBinG8);
      PCC_COUNT(1);
    }
    if (want(kBinG16) && !routed(kBinG16)) {
      BestMoveGroupKernel<16, kInt, kAsync><<<grid(kBinG16, 16, waves(sms * 8)), 256, 0, st>>>(a, list, counts, starts,
                                                                                            kBinG16);
      PCC_COUNT(1);
    }
    if (want(kBinG32) && !routed(kBinG32)) {
      BestMoveGroupKernel<32, kInt, kAsync><<<grid(kBinG32, 8, waves(sms * 8)), 256, 0, st>>>(a, list, counts, starts,
                                                                                            kBinG32);
      PCC_COUNT(1);
    }
  }
  if (families & kLaunchGroups) FamEnd(ctx, kFamGroup, ng);
  int nw = 0;
  for (int b = kBinG4; b <= kBinW1000; ++b) nw += want(b) && (b > kBinG32 || routed(b)) ? 1 : 0;
  if (families & kLaunchWarps) FamBegin(ctx, kFamWarp);
  if constexpr (kCert) {
    // The certified warp bins for one sum type: int or long long sums, with
    // (kConv) or without the general weight conversion.
    auto cert_bins = [&](auto sum, auto conv) -> Status {
      using V = decltype(sum);
      constexpr bool kC = decltype(conv)::value;
      PCC_RETURN_IF_ERROR(routed_bins(CertWarpKernel<256, V, kC>, CertWarpSmem<256, V>(), sms * 16));
      PCC_RETURN_IF_ERROR(cert_bin(CertWarpKernel<256, V, kC>, CertWarpSmem<256, V>(), CertCtaKernel<256, V, kC>,
                                   CertCtaSmem<256, V>(), kBinW128, sms * 16));
      PCC_RETURN_IF_ERROR(cert_bin(CertWarpKernel<512, V, kC>, CertWarpSmem<512, V>(), CertCtaKernel<512, V, kC>,
                                   CertCtaSmem<512, V>(), kBinW256, sms * 8));
      PCC_RETURN_IF_ERROR(cert_bin(CertWarpKernel<1024, V, kC>, CertWarpSmem<1024, V>(), CertCtaKernel<1024, V, kC>,
                                   CertCtaSmem<1024, V>(), kBinW512, sms * 4));
      return cert_bin(CertWarpKernel<2048, V, kC>, CertWarpSmem<2048, V>(), CertCtaKernel<2048, V, kC>,
                      CertCtaSmem<2048, V>(), kBinW1000, sms * 2);
    };
    if (!a.narrow) {
      PCC_RETURN_IF_ERROR(cert_bins(0ll, std::true_type{}));
    } else if (a.conv) {
      PCC_RETURN_IF_ERROR(cert_bins(0, std::true_type{}));
    } else {
      PCC_RETURN_IF_ERROR(cert_bins(0, std::false_type{}));
    }
  } else {
    PCC_RETURN_IF_ERROR(routed_bins(BestMoveWarpKernel<256, kInt, kAsync>, WarpKernelSmem<256>(), sms * 16));
    PCC_RETURN_IF_ERROR(warp_bin(BestMoveWarpKernel<256, kInt, kAsync>, WarpKernelSmem<256>(), kBinW128, sms * 16));
    PCC_RETURN_IF_ERROR(warp_bin(BestMoveWarpKernel<512, kInt, kAsync>, WarpKernelSmem<512>(), kBinW256, sms * 8));
    PCC_RETURN_IF_ERROR(warp_bin(BestMoveWarpKernel<1024, kInt, kAsync>, WarpKernelSmem<1024>(), kBinW512, sms * 4));
    PCC_RETURN_IF_ERROR(warp_bin(BestMoveWarpKernel<2048, kInt, kAsync>, WarpKernelSmem<2048>(), kBinW1000, sms * 2));
  }
  if (families & kLaunchWarps) FamEnd(ctx, kFamWarp, nw);
  return LaunchCheck();
}

template <class K>
Status Prep(K kernel, size_t smem, int threads) {
  int per_sm = 0;
  return SetSmem(kernel, smem, threads, &per_sm);
}

Status PrepareAll() {
  PCC_RETURN_IF_ERROR(Prep(CertGroupKernel<4, int>, 0, 256));
  PCC_RETURN_IF_ERROR(Prep(CertGroupKernel<8, int>, 0, 256));
  PCC_RETURN_IF_ERROR(Prep(CertGroupKernel<16, int>, 0, 256));
  PCC_RETURN_IF_ERROR(Prep(CertGroupKernel<32, int>, 0, 256));
  PCC_RETURN_IF_ERROR(Prep(CertGroupKernel<4, long long>, 0, 256));
  PCC_RETURN_IF_ERROR(Prep(CertGroupKernel<8, long long>, 0, 256));
  PCC_RETURN_IF_ERROR(Prep(CertGroupKernel<16, long long>, 0, 256));
  PCC_RETURN_IF_ERROR(Prep(CertGroupKernel<32, long long>, 0, 256));
  constexpr int kW = kWarpKernelWarps * 32;
  PCC_RETURN_IF_ERROR(Prep(CertWarpKernel<256, int, false>, CertWarpSmem<256, int>(), kW));
  PCC_RETURN_IF_ERROR(Prep(CertWarpKernel<256, int, true>, CertWarpSmem<256, int>(), kW));
  PCC_RETURN_IF_ERROR(Prep(CertWarpKernel<512, int, false>, CertWarpSmem<512, int>(), kW));
  PCC_RETURN_IF_ERROR(Prep(CertWarpKernel<512, int, true>, CertWarpSmem<512, int>(), kW));
  PCC_RETURN_IF_ERROR(Prep(CertWarpKernel<1024, int, false>, CertWarpSmem<1024, int>(), kW));
  PCC_RETURN_IF_ERROR(Prep(CertWarpKernel<1024, int, true>, CertWarpSmem<1024, int>(), kW));
  PCC_RETURN_IF_ERROR(Prep(CertWarpKernel<2048, int, false>, CertWarpSmem<2048, int>(), kW));
  PCC_RETURN_IF_ERROR(Prep(CertWarpKernel<2048, int, true>, CertWarpSmem<2048, int>(), kW));
  PCC_RETURN_IF_ERROR(Prep(CertWarpKernel<256, long long>, CertWarpSmem<256, long long>(), kW));
  PCC_RETURN_IF_ERROR(Prep(CertWarpKernel<512, long long>, CertWarpSmem<512, long long>(), kW));
  PCC_RETURN_IF_ERROR(Prep(CertWarpKernel<1024, long long>, CertWarpSmem<1024, long long>(), kW));
  PCC_RETURN_IF_ERROR(Prep(CertWarpKernel<2048, long long>, CertWarpSmem<2048, long long>(), kW));
  constexpr int kC = kCtaWarps * 32;
  PCC_RETURN_IF_ERROR(Prep(CertCtaKernel<256, int, false>, CertCtaSmem<256, int>(), kC));
  PCC_RETURN_IF_ERROR(Prep(CertCtaKernel<256, int, true>, CertCtaSmem<256, int>(), kC));
  PCC_RETURN_IF_ERROR(Prep(CertCtaKernel<512, int, false>, CertCtaSmem<512, int>(), kC));
  PCC_RETURN_IF_ERROR(Prep(CertCtaKernel<512, int, true>, CertCtaSmem<512, int>(), kC));
  PCC_RETURN_IF_ERROR(Prep(CertCtaKernel<1024, int, false>, CertCtaSmem<1024, int>(), kC));
  PCC_RETURN_IF_ERROR(Prep(CertCtaKernel<1024, int, true>, CertCtaSmem<1024, int>(), kC));
  PCC_RETURN_IF_ERROR(Prep(CertCtaKernel<2048, int, false>, CertCtaSmem<2048, int>(), kC));
  PCC_RETURN_IF_ERROR(Prep(CertCtaKernel<2048, int, true>, CertCtaSmem<2048, int>(), kC));
  PCC_RETURN_IF_ERROR(Prep(CertCtaKernel<256, long long>, CertCtaSmem<256, long long>(), kC));
  PCC_RETURN_IF_ERROR(Prep(CertCtaKernel<512, long long>, CertCtaSmem<512, long long>(), kC));
  PCC_RETURN_IF_ERROR(Prep(CertCtaKernel<1024, long long>, CertCtaSmem<1024, long long>(), kC));
  PCC_RETURN_IF_ERROR(Prep(CertCtaKernel<2048, long long>, CertCtaSmem<2048, long long>(), kC));
  PCC_RETURN_IF_ERROR(Prep(BestMoveWarpKernel<256, false, false>, WarpKernelSmem<256>(), kW));
  PCC_RETURN_IF_ERROR(Prep(BestMoveWarpKernel<512, false, false>, WarpKernelSmem<512>(), kW));
  PCC_RETURN_IF_ERROR(Prep(BestMoveWarpKernel<1024, false, false>, WarpKernelSmem<1024>(), kW));
  PCC_RETURN_IF_ERROR(Prep(BestMoveWarpKernel<2048, false, false>, WarpKernelSmem<2048>(), kW));
  return Status::Ok();
}

}  // namespace

Status PrepareBestMoveKernels() {
  static PerDevice done;
  return OncePerDevice(done, PrepareAll);
}

Status LaunchBestMoves(Context* ctx, const BMArgs& a, const uint32_t* list, const uint32_t* bin_counts,
                       const uint32_t* bin_starts, const uint32_t* host_counts, bool int_mode,
                       uint32_t max_deg, int families) {
  if (a.async) {
    return int_mode ? LaunchAll<true, true>(ctx, a, list, bin_counts, bin_starts, host_counts, max_deg, families)
                    : LaunchAll<false, true>(ctx, a, list, bin_counts, bin_starts, host_counts, max_deg, families);
  }
  return int_mode ? LaunchAll<true, false>(ctx, a, list, bin_counts, bin_starts, host_counts, max_deg, families)
                  : LaunchAll<false, false>(ctx, a, list, bin_counts, bin_starts, host_counts, max_deg, families);
}

}  // namespace pcc
