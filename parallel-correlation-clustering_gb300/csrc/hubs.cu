// hubs.cu -- best moves of hub vertices (degree > 1000); the scheme is in
// hubs.cuh.  Restates the hub branch of ClusteringHelper::EfficientBestMove
// (parallel-correlation-clusterer-internal.cc:516-582): per-cluster sums in
// any order (the reference adds concurrently), FP64-mode weights rounded to
// float after the offset, the argmax by (value desc, id asc), and "no
// entries" giving the reduce identity (0, 0.0) unless change >= 0.
#include <algorithm>
#include <numeric>
#include <vector>

#include "certmoves.cuh"
#include "hubeval.cuh"

namespace pcc {
namespace {

constexpr int kSmallThreads = 256;         // small hubs: CTA size, table slots
constexpr uint32_t kSmallSlots = 2 * kHubSmallMax;
constexpr uint32_t kSmallMidSlots = 3 * kHubSmallMax / 2;  // hubs with 2d + 2 <= kSmallMidSlots
constexpr uint32_t kSmallNarrowSlots = kHubSmallMax;  // hubs with 2d + 2 <= kSmallNarrowSlots
constexpr int kBigThreads = 1024;          // big hubs
// Big-hub table: ~192 KB of (key, sum) slots.
template <typename V>
__host__ __device__ constexpr uint32_t BigSlots() {
  return sizeof(V) == 4 ? 2 * kHubBigKeys : 16384;
}

struct HubArgs {
  BMArgs a;
  const uint32_t* small_v;
  uint32_t small_lo, small_hi;  // this launch's items of small_v
  const uint32_t* big_v;
  const uint32_t* big_parts;
  const uint32_t* big_pbase;
  const uint32_t* item_hub;
  const uint32_t* item_part;
  uint32_t num_items;
  double* part_val;
  uint32_t* part_id;
  uint32_t* done;
  // Global path (sync): tables, accumulators, plan (num_glob 0: none).
  uint32_t num_glob;
  uint32_t num_glob_items;
  const uint32_t* glob_hub;
  const unsigned long long* glob_base;
  const uint32_t* glob_cap;
  const uint32_t* glob_item;
  const uint32_t* glob_item_start;
  const uint32_t* big_glob;
  uint32_t* gkeys;
  unsigned long long* gvals;
  long long* gt_int;
  double* gt_dbl;
  long long* gsmax;
  uint32_t num_glob_slices;
  const uint32_t* glob_nslices;
  const uint32_t* glob_sbase;
  const uint32_t* slice_hub;
  const uint32_t* slice_start;
  double* gpart_val;
  uint32_t* gpart_id;
  uint32_t* gdone;
};

// ---------------------------------------------------------------------------
// Small hubs: one CTA per hub, a table of 2 * degree slots (never full).
// ---------------------------------------------------------------------------
template <bool kInt, bool kAsync, typename V, uint32_t kSlots>
__global__ void __launch_bounds__(kSmallThreads) HubSmallKernel(HubArgs h) {
  constexpr int BT = kSmallThreads;
  extern __shared__ __align__(16) unsigned char smem[];
  V* svals = reinterpret_cast<V*>(smem);
  uint32_t* skeys = reinterpret_cast<uint32_t*>(smem + size_t(kSlots) * sizeof(V));
  __shared__ HubShared<BT> sh;
  const BMArgs& a = h.a;
  const unsigned tid = threadIdx.x;
  unsigned long long fam_e = 0, fam_v = 0;  // entries and vertices evaluated (tid 0)
  for (uint32_t i = tid; i < kSlots; i += BT) {
    skeys[i] = kNone;
    svals[i] = V(0);
  }
  if (tid == 0) {
    sh.overflow = 0;
    sh.nkeys = 0;
  }
  __syncthreads();
  for (uint32_t item = h.small_lo + blockIdx.x; item < h.small_hi; item += gridDim.x) {
    const uint32_t v = h.small_v[item];
    if (!InFront(a, v)) continue;  // uniform over the CTA
    const VertexCtx x = LoadVertex<kAsync>(a, v);
    const uint32_t cap = min(kSlots, 2 * x.d + 2);
    if (tid == 0) {
      fam_e += x.d;
      fam_v += 1;
    }
    long long t_int = 0, smax = LLONG_MIN;
    double t_dbl = 0.0;
    ScanRow<BT, kInt, kAsync, V>(a, x, 1, 0, 1, 0, true, skeys, svals, cap, cap, sh, &t_int, &t_dbl, &smax);
    // Its barriers also complete the table and sh.overflow before they are read.
    const double change = HubChangeSmax<BT, kInt>(a, x, t_int, t_dbl, &smax, sh);
    if (tid == 0) {
      if (sh.overflow) atomicExch(&a.ctr->error, kErrHashFull);  // cannot happen: 2d + 2 slots
      sh.nkeys = 0;
    }
    double bv;
    uint32_t bi;
    EvalTable<BT, kInt, kAsync, V>(a, x, a.kf[v], change, smax, skeys, svals, cap, sh, &bv, &bi);
    if (tid == 0) HubDecide<kAsync>(a, x, bv, bi, change, StampIn(a.rs, a.stamp), &a.ctr->movers);
    __syncthreads();
  }
  if (tid == 0 && fam_v) {
    atomicAdd(&a.ctr->fam_entries[kFamHubSmall], fam_e);
    atomicAdd(&a.ctr->fam_vertices[kFamHubSmall], fam_v);
  }
}

// Small hubs with exact sums, synchronous moves: a CTA of TW warps takes a hub
// the way the warp rows go (CtaStep, certmoves.cuh): certified FP32 decisions
// over the used slots instead of HubSmallKernel's evaluation of every slot of
// the table.  Two table sizes: HC = 4096 slots with 8 warps, 8192 with 16, so
// that 48 warps of 32-bit sums fit an SM with either.  Bound by the gathers of
// the neighbours' clusters and shared-memory atomics.  (All rounds of RMAT
// scale 20: 34.9 ms by HubSmallKernel, 14.9; scale 22: 28.1, 22.0; 1M vertices
// with real weights, 64-bit sums: 39.6, 20.6.)
// Degrees 4,097 to 12,288 go the same way with 16,384 slots and 32 warps
// (up to three quarters full).
template <int HC, int TW, typename V>
__host__ __device__ constexpr size_t HubCertSmem() {
  return size_t(HC) * (sizeof(V) + sizeof(uint32_t)) +
         size_t(TW == 32 ? kHubBigKeys : HC / 2) * sizeof(uint16_t);  // vals, keys, used
}

template <int HC, int TW, typename V, bool kConv>
__global__ void __launch_bounds__(TW * 32) HubCertKernel(HubArgs h) {
  constexpr int BT = TW * 32;
  extern __shared__ __align__(16) unsigned char smem[];
  V* vals = reinterpret_cast<V*>(smem);
  uint32_t* keys = reinterpret_cast<uint32_t*>(smem + size_t(HC) * sizeof(V));
  uint16_t* used = reinterpret_cast<uint16_t*>(smem + size_t(HC) * (sizeof(V) + sizeof(uint32_t)));
  __shared__ CtaShared<V, TW> sh;
  const BMArgs& a = h.a;
  const unsigned tid = threadIdx.x;
  unsigned long long fam_e = 0, fam_v = 0;  // entries and vertices evaluated (tid 0)
  const bool replay = a.out_target != nullptr;
  const RoundView rv = RoundOf(a);
  for (uint32_t i = tid; i < HC; i += BT) {
    keys[i] = kNone;
    vals[i] = 0;
  }
  if (tid == 0) sh.nused = 0;
  __syncthreads();
  for (uint32_t item = h.small_lo + blockIdx.x; item < h.small_hi; item += gridDim.x) {
    const uint32_t v = h.small_v[item];
    if (!InFront(a, rv, v)) continue;  // uniform over the CTA
    const VertexCtx x = LoadVertexAs<ConstLoads>(a, v);
    if (tid == 0) {
      fam_e += x.d;
      fam_v += 1;
    }
    const bool append =
        CtaStep<HC, V, kConv, ConstLoads, TW>(a, rv, x, vals, keys, used, sh, tid, 0, replay);
    if (tid == 0 && append) a.movers[atomicAdd(&a.ctr->movers, 1u)] = v;
  }
  if (tid == 0 && fam_v) {
    constexpr int fam = TW == 32 ? kFamHubBig : kFamHubSmall;
    atomicAdd(&a.ctr->fam_entries[fam], fam_e);
    atomicAdd(&a.ctr->fam_vertices[fam], fam_v);
  }
}

// ---------------------------------------------------------------------------
// Big hubs: one CTA per (hub, partition), sub-passes on overflow.
// ---------------------------------------------------------------------------
template <bool kInt, bool kAsync, typename V>
__global__ void __launch_bounds__(kBigThreads) HubBigKernel(HubArgs h) {
  constexpr int BT = kBigThreads;
  constexpr uint32_t kSlots = BigSlots<V>();
  extern __shared__ __align__(16) unsigned char smem[];
  V* svals = reinterpret_cast<V*>(smem);
  uint32_t* skeys = reinterpret_cast<uint32_t*>(smem + size_t(kSlots) * sizeof(V));
  __shared__ HubShared<BT> sh;
  const BMArgs& a = h.a;
  const unsigned tid = threadIdx.x;
  unsigned long long fam_e = 0, fam_v = 0;  // entries and vertices evaluated once per hub (tid 0)
  for (uint32_t i = tid; i < kSlots; i += BT) {
    skeys[i] = kNone;
    svals[i] = V(0);
  }
  if (tid == 0) {
    sh.overflow = 0;
    sh.nkeys = 0;
  }
  __syncthreads();
  for (uint32_t item = blockIdx.x; item < h.num_items; item += gridDim.x) {
    const uint32_t hb = h.item_hub[item];
    const uint32_t p = h.item_part[item];
    const uint32_t v = h.big_v[hb];
    if (!kAsync && h.num_glob && h.big_glob[hb] != kNone) continue;  // global path
    if (!InFront(a, v)) continue;  // uniform over the CTA
    const VertexCtx x = LoadVertex<kAsync>(a, v);
    const uint32_t P = h.big_parts[hb];
    if (tid == 0 && p == 0) {
      fam_e += x.d;
      fam_v += 1;
    }
    const uint32_t cap = min(kSlots, 2 * ((x.d + P - 1) / P) + 2);
    const uint32_t maxkeys = cap - cap / 4;
    uint32_t Q = 1, q = 0;
    bool have_T = false;
    double change = 0.0;
    long long shift = 0;  // sub-passes of 64-bit sums: the first one's
    double bestv = 0.0;
    uint32_t bestid = kNone;
    while (true) {
      long long t_int = 0, smax = LLONG_MIN;
      double t_dbl = 0.0;
      ScanRow<BT, kInt, kAsync, V>(a, x, P, p, Q, q, !have_T, skeys, svals, cap, maxkeys, sh, &t_int, &t_dbl,
                                   &smax);
      // The reductions' barriers also order the reads of sh.overflow.
      if (!have_T) {
        change = HubChangeSmax<BT, kInt>(a, x, t_int, t_dbl, &smax, sh);
        shift = smax;
        have_T = true;
      } else {
        __syncthreads();
        if (kInt) smax = BlockMaxLL<BT>(smax, sh.red_ll);
        if (kInt && smax == LLONG_MIN) smax = shift;
      }
      const bool overflow = sh.overflow != 0;
      __syncthreads();
      if (tid == 0) {
        sh.overflow = 0;
        sh.nkeys = 0;
      }
      if (overflow) {
        // Split the partition further and rescan from the first sub-pass.
        for (uint32_t s = tid; s < cap; s += BT) {
          skeys[s] = kNone;
          svals[s] = V(0);
        }
        __syncthreads();
        Q *= 2;
        q = 0;
        bestv = 0.0;
        bestid = kNone;
        if (Q > kHubMaxSub) {
          if (tid == 0) atomicExch(&a.ctr->error, kErrHashFull);
          break;
        }
        continue;
      }
      double lv;
      uint32_t lid;
      EvalTable<BT, kInt, kAsync, V>(a, x, a.kf[v], change, smax, skeys, svals, cap, sh, &lv, &lid);
      KeepBest(bestv, bestid, lv, lid);
      __syncthreads();
      if (++q == Q) break;
    }
    // Partial result; the hub's last CTA combines and decides.
    if (tid == 0) {
      const uint32_t pb = h.big_pbase[hb];
      h.part_val[pb + p] = bestv;
      h.part_id[pb + p] = bestid;
      __threadfence();
      if (atomicAdd(&h.done[hb], 1u) == P - 1) {
        __threadfence();
        double bv = 0.0;
        uint32_t bi = kNone;
        for (uint32_t j = 0; j < P; ++j) KeepBest(bv, bi, __ldcg(h.part_val + pb + j), __ldcg(h.part_id + pb + j));
        h.done[hb] = 0;
        HubDecide<kAsync>(a, x, bv, bi, change, StampIn(a.rs, a.stamp), &a.ctr->movers);
      }
    }
    __syncthreads();
  }
  if (tid == 0 && fam_v) {
    atomicAdd(&a.ctr->fam_entries[kFamHubBig], fam_e);
    atomicAdd(&a.ctr->fam_vertices[kFamHubBig], fam_v);
  }
}

// ---------------------------------------------------------------------------
// Global path: rows of the largest hubs split over many CTAs.
// ---------------------------------------------------------------------------
constexpr int kGlobThreads = 256;
constexpr uint32_t kGlobChunk = kGlobThreads;  // row entries per work item: one per thread

// Accumulates row chunks into the hubs' HBM tables (warp-aggregated inserts
// and adds), the together-sum and (INT) the largest running sum.
template <bool kInt, typename V>
__global__ void __launch_bounds__(kGlobThreads) HubGlobalAccumKernel(HubArgs h) {
  constexpr int BT = kGlobThreads;
  __shared__ HubShared<BT> sh;
  const BMArgs& a = h.a;
  const unsigned tid = threadIdx.x, lane = LaneId();
  for (uint32_t item = blockIdx.x; item < h.num_glob_items; item += gridDim.x) {
    const uint32_t gi = h.glob_item[item];
    const uint32_t v = h.big_v[h.glob_hub[gi]];
    if (!InFront(a, v)) continue;  // uniform over the CTA
    const VertexCtx x = LoadVertex<false>(a, v);
    const uint32_t e_begin = h.glob_item_start[item];
    const uint32_t e_end = min(x.d, e_begin + kGlobChunk);
    uint32_t* keys = h.gkeys + h.glob_base[gi];
    V* vals = reinterpret_cast<V*>(h.gvals) + h.glob_base[gi];
    const uint32_t cap = h.glob_cap[gi];
    long long t_int = 0, smax = LLONG_MIN;
    double t_dbl = 0.0;
    for (uint32_t e0 = e_begin; e0 < e_end; e0 += BT * kHubUnroll) {
      uint32_t uu[kHubUnroll], cc[kHubUnroll];
      float ww[kHubUnroll];
#pragma unroll
      for (int k = 0; k < kHubUnroll; ++k) {
        const uint32_t e = e0 + k * BT + tid;
        uu[k] = v;
        ww[k] = 0.f;
        if (e < e_end) {
          uu[k] = a.nbr[x.b + e];
          ww[k] = a.w ? a.w[x.b + e] : 1.0f;
        }
      }
#pragma unroll
      for (int k = 0; k < kHubUnroll; ++k) cc[k] = uu[k] != v ? __ldg(a.C + uu[k]) : kNone;
#pragma unroll
      for (int k = 0; k < kHubUnroll; ++k) {
        if (e0 + k * BT >= e_end) break;  // uniform over the CTA
        const bool cand = uu[k] != v;
        const uint32_t cu = cc[k];
        V xi = 0;
        double xd = 0.0;
        if (cand) EntryWeight<kInt, V>(a, ww[k], &xi, &xd);
        if (cand && cu == x.c) {
          if (kInt)
            t_int += xi;
          else
            t_dbl = Dadd(t_dbl, xd);
        }
        unsigned peers = 0;
        bool leader = cand;
        double Sd = 0.0;
        if constexpr (!kInt) {
          peers = __match_any_sync(kFull, cand ? cu : LaneSentinel(lane));
          leader = cand && int(lane) == __ffs(peers) - 1;
          Sd = GroupWeights<BT>(peers, leader, xd);
        }
        if (leader) {
          bool ins;
          const uint32_t slot = HubInsert(keys, cap, SlotHash(cu), cu, &ins);
          if (slot == kNone) {
            atomicExch(&a.ctr->error, kErrHashFull);  // cannot happen: 2 * degree + 2 slots
          } else if (kInt) {
            const V old = AtomicAddV<V>(vals + slot, xi);
            smax = max(smax, static_cast<long long>(old) + static_cast<long long>(xi));
          } else {
            AtomicAddV<V>(vals + slot, static_cast<V>(Sd));
          }
        }
      }
    }
    if (kInt) {
      const long long t = BlockSum<BT, long long>(t_int, sh.red_ll);
      const long long mx = BlockMaxLL<BT>(smax, sh.red_ll);
      if (tid == 0) {
        if (t) atomicAdd(reinterpret_cast<unsigned long long*>(h.gt_int + gi), static_cast<unsigned long long>(t));
        atomicMax(h.gsmax + gi, mx);
      }
    } else {
      const double t = BlockSum<BT, double>(t_dbl, sh.red_d);
      if (tid == 0 && t != 0.0) atomicAdd(h.gt_dbl + gi, t);
    }
  }
}

// Evaluates the HBM tables of the frontier hubs, one slice per CTA (the
// small-hub evaluation of the slice's keys: FP32 pre-filter, certified leading
// class, FP64 survivors), clearing the slots (EvalTable).  The hub's last CTA
// combines the slices' (value, id) bests, decides and resets the hub's
// accumulators.
template <bool kInt, typename V>
__global__ void __launch_bounds__(kGlobThreads) HubGlobalEvalKernel(HubArgs h) {
  constexpr int BT = kGlobThreads;
  __shared__ HubShared<BT> sh;
  const BMArgs& a = h.a;
  const unsigned tid = threadIdx.x;
  unsigned long long fam_e = 0, fam_v = 0;
  for (uint32_t item = blockIdx.x; item < h.num_glob_slices; item += gridDim.x) {
    const uint32_t gi = h.slice_hub[item];
    const uint32_t v = h.big_v[h.glob_hub[gi]];
    if (!InFront(a, v)) continue;  // uniform over the CTA
    const VertexCtx x = LoadVertex<false>(a, v);
    const uint32_t s0 = h.slice_start[item];
    const uint32_t len = min(kHubGlobalSlice, h.glob_cap[gi] - s0);
    const long long smax = __ldcg(h.gsmax + gi);
    if (tid == 0) {
      if (s0 == 0) {
        fam_e += x.d;
        fam_v += 1;
      }
      const double T = kInt ? UnitsToDouble<long long>(a, __ldcg(h.gt_int + gi)) : __ldcg(h.gt_dbl + gi);
      sh.change = ChangeOf(a, x, T);
      sh.change32 = static_cast<float>(sh.change);
    }
    __syncthreads();
    const double change = sh.change;
    double bv;
    uint32_t bi;
    const unsigned long long base = h.glob_base[gi] + s0;
    EvalTable<BT, kInt, false, V>(a, x, a.kf[v], change, smax, h.gkeys + base, reinterpret_cast<V*>(h.gvals) + base,
                                  len, sh, &bv, &bi);
    const uint32_t sb = h.glob_sbase[gi];
    const uint32_t ns = h.glob_nslices[gi];
    if (tid == 0) {
      h.gpart_val[sb + s0 / kHubGlobalSlice] = bv;
      h.gpart_id[sb + s0 / kHubGlobalSlice] = bi;
      __threadfence();
      sh.last = atomicAdd(&h.gdone[gi], 1u) == ns - 1 ? 1u : 0u;
    }
    __syncthreads();
    if (sh.last) {  // uniform: the whole CTA combines the slices' bests
      __threadfence();
      double cv = 0.0;
      uint32_t ci = kNone;
      for (uint32_t j = tid; j < ns; j += BT) KeepBest(cv, ci, __ldcg(h.gpart_val + sb + j), __ldcg(h.gpart_id + sb + j));
      BlockArgmax<BT>(cv, ci, sh.red_k, sh.red_i);
      if (tid == 0) {
        HubDecide<false>(a, x, cv, ci, change, StampIn(a.rs, a.stamp), &a.ctr->movers);
        h.gdone[gi] = 0;
        h.gt_int[gi] = 0;
        h.gt_dbl[gi] = 0.0;
        h.gsmax[gi] = LLONG_MIN;
      }
    }
    __syncthreads();
  }
  if (tid == 0 && fam_v) {
    atomicAdd(&a.ctr->fam_entries[kFamHubBig], fam_e);
    atomicAdd(&a.ctr->fam_vertices[kFamHubBig], fam_v);
  }
}

__global__ void GlobalStateInitKernel(uint32_t num, long long* gt_int, double* gt_dbl, long long* gsmax,
                                      uint32_t* gdone) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < num; i += gridDim.x * blockDim.x) {
    gt_int[i] = 0;
    gt_dbl[i] = 0.0;
    gsmax[i] = LLONG_MIN;
    gdone[i] = 0;
  }
}

__global__ void HubDegreesKernel(const uint32_t* list, uint32_t count, const uint64_t* off, uint32_t* deg) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x)
    deg[i] = static_cast<uint32_t>(off[list[i] + 1] - off[list[i]]);
}

// Resident CTAs per SM of a kernel at `smem` bytes; 0 when it cannot be set up.
template <class K>
int PrepareOnce(K kernel, int threads, size_t smem) {
  int per_sm = 0;
  return PrepareKernel(kernel, threads, smem, smem, &per_sm).ok() ? per_sm : 0;
}

// One small-hub table class over small_v[lo, hi).
template <bool kInt, bool kAsync, typename V, uint32_t kSlots>
Status LaunchSmallClass(Context* ctx, const HubArgs& h, uint32_t lo, uint32_t hi) {
  if (hi <= lo) return Status::Ok();
  constexpr size_t smem = size_t(kSlots) * (sizeof(V) + sizeof(uint32_t));
  auto k = HubSmallKernel<kInt, kAsync, V, kSlots>;
  const int per_sm = PrepareOnce(k, kSmallThreads, smem);
  if (per_sm <= 0) return MakeError(PCC_INTERNAL, "small-hub kernel cannot be configured");
  HubArgs hc = h;
  hc.small_lo = lo;
  hc.small_hi = hi;
  k<<<Blocks(hi - lo, 1, unsigned(ctx->num_sms) * unsigned(per_sm)), kSmallThreads, smem, ctx->stream>>>(hc);
  PCC_COUNT(1);
  return Status::Ok();
}

// The same for HubCertKernel.
template <int HC, int TW, typename V>
Status LaunchCertClass(Context* ctx, const HubArgs& h, uint32_t lo, uint32_t hi) {
  if (hi <= lo) return Status::Ok();
  constexpr size_t smem = HubCertSmem<HC, TW, V>();
  auto k = HubCertKernel<HC, TW, V, true>;
  if constexpr (sizeof(V) == 4) {
    if (!h.a.conv) k = HubCertKernel<HC, TW, V, false>;
  }
  const int per_sm = PrepareOnce(k, TW * 32, smem);
  if (per_sm <= 0) return MakeError(PCC_INTERNAL, "small-hub kernel cannot be configured");
  HubArgs hc = h;
  hc.small_lo = lo;
  hc.small_hi = hi;
  k<<<Blocks(hi - lo, 1, unsigned(ctx->num_sms) * unsigned(per_sm)), TW * 32, smem, ctx->stream>>>(hc);
  PCC_COUNT(1);
  return Status::Ok();
}

template <bool kInt, bool kAsync, typename V>
Status LaunchHubT(Context* ctx, const HubArgs& h, const HubPlan& plan, int families) {
  const uint32_t num_small = plan.num_small, num_wide = plan.num_small_wide, num_mid = plan.num_small_mid;
  const uint32_t num_big = plan.num_big, num_multi = plan.num_multi, num_multi_items = plan.num_multi_items;
  const unsigned sms = unsigned(ctx->num_sms);
  if (num_small && (families & kLaunchSmallHubs)) {
    // Each hub in the smallest table that holds its 2d + 2 slots (the classes
    // are consecutive in small_v, widest first): smaller tables fit more CTAs
    // per SM.
    const uint32_t end_mid = num_wide + num_mid;
    int nl = (num_wide > 0) + (num_mid > 0) + (num_small > end_mid);
    FamBegin(ctx, kFamHubSmall);
    if constexpr (kInt && !kAsync) {
      PCC_RETURN_IF_ERROR((LaunchCertClass<2 * kHubSmallMax, 16, V>(ctx, h, 0, end_mid)));
      PCC_RETURN_IF_ERROR((LaunchCertClass<kHubSmallMax, 8, V>(ctx, h, end_mid, num_small)));
      nl = (end_mid > 0) + (num_small > end_mid);
    } else {
      PCC_RETURN_IF_ERROR((LaunchSmallClass<kInt, kAsync, V, kSmallSlots>(ctx, h, 0, num_wide)));
      PCC_RETURN_IF_ERROR((LaunchSmallClass<kInt, kAsync, V, kSmallMidSlots>(ctx, h, num_wide, end_mid)));
      PCC_RETURN_IF_ERROR((LaunchSmallClass<kInt, kAsync, V, kSmallNarrowSlots>(ctx, h, end_mid, num_small)));
    }
    FamEnd(ctx, kFamHubSmall, nl);
  }
  const bool glob = !kAsync && h.num_glob;
  if (h.num_items && (families & kLaunchBigHubs)) {
    FamBegin(ctx, kFamHubBig);
    if (glob) {
      HubGlobalAccumKernel<kInt, V><<<std::min<unsigned>(h.num_glob_items, sms * 8), kGlobThreads, 0,
                                      ctx->stream>>>(h);
      PCC_COUNT(1);
    }
    FamEnd(ctx, kFamHubBig, glob ? 1 : 0);
    HubArgs hm = h;
    if constexpr (kInt && !kAsync) {
      hm.num_items = num_multi_items;
      if (num_big > num_multi) {
        HubArgs hs = h;
        hs.small_v = h.big_v;
        FamBegin(ctx, kFamHubBig);
        PCC_RETURN_IF_ERROR((LaunchCertClass<16384, 32, V>(ctx, hs, num_multi, num_big)));
        FamEnd(ctx, kFamHubBig, 1);
      }
    }
    if (hm.num_items) {
      constexpr size_t smem = size_t(BigSlots<V>()) * (sizeof(V) + sizeof(uint32_t));
      auto k = HubBigKernel<kInt, kAsync, V>;
      const int per_sm = PrepareOnce(k, kBigThreads, smem);
      if (per_sm <= 0) return MakeError(PCC_INTERNAL, "big-hub kernel cannot be configured");
      const unsigned grid = Blocks(hm.num_items, 1, sms * unsigned(std::max(per_sm, 1)));
      FamBegin(ctx, kFamHubBig);
      k<<<grid, kBigThreads, smem, ctx->stream>>>(hm);
      FamEnd(ctx, kFamHubBig, 1);
      PCC_COUNT(1);
    }
    if (glob) {
      FamBegin(ctx, kFamHubBig);
      HubGlobalEvalKernel<kInt, V><<<std::min<unsigned>(h.num_glob_slices, 8 * sms), kGlobThreads, 0,
                                     ctx->stream>>>(h);
      FamEnd(ctx, kFamHubBig, 1);
      PCC_COUNT(1);
    }
  }
  return LaunchCheck();
}

}  // namespace

Status BuildHubPlan(Context* ctx, const DevGraph& g, const BinSet& bins, HubPlan* plan) {
  // Hubs are the static bins above the warp bins (degree > 1000).
  uint32_t start = 0, count = 0;
  for (int b = 0; b < kBinCta; ++b) start += bins.host_counts[b];
  for (int b = kBinCta; b < kNumBins; ++b) count += bins.host_counts[b];
  plan->num_hubs = count;
  if (count == 0) return Status::Ok();
  std::vector<uint32_t> hv(count), hd(count);
  DBuf<uint32_t> ddeg;
  PCC_RETURN_IF_ERROR(ddeg.Alloc(ctx, count));
  HubDegreesKernel<<<Blocks(count, 256, 1024), 256, 0, ctx->stream>>>(bins.list.p + start, count, g.off.p, ddeg.p);
  PCC_COUNT(1);
  PCC_CUDA(cudaMemcpyAsync(hv.data(), bins.list.p + start, sizeof(uint32_t) * count, cudaMemcpyDeviceToHost,
                           ctx->stream));
  PCC_RETURN_IF_ERROR(ddeg.ToHost(hd.data(), count));
  PCC_RETURN_IF_ERROR(Sync(ctx));
  // Largest hubs first (the longest work items start first); a big hub's
  // partitions are consecutive items, so they run at the same time and share
  // the row through L2.
  std::vector<uint32_t> order(count);
  std::iota(order.begin(), order.end(), 0u);
  std::stable_sort(order.begin(), order.end(), [&](uint32_t i, uint32_t j) { return hd[i] > hd[j]; });
  std::vector<uint32_t> small_v, big_v, parts, pbase, item_hub, item_part;
  std::vector<uint32_t> big_glob, glob_hub, glob_cap, glob_item, glob_item_start;
  std::vector<uint32_t> glob_nslices, glob_sbase, slice_hub, slice_start;
  std::vector<uint32_t> loop_cap, loop_nslices, loop_sbase, chunk_hub, chunk_start, loop_slice_hub,
      loop_slice_start;
  std::vector<unsigned long long> glob_base, loop_base;
  uint64_t total = 0;
  for (uint32_t r = 0; r < count; ++r) {
    const uint32_t i = order[r];
    if (hd[i] <= kHubSmallMax) {
      small_v.push_back(hv[i]);
      if (2 * hd[i] + 2 > kSmallMidSlots) plan->num_small_wide++;
      else if (2 * hd[i] + 2 > kSmallNarrowSlots) plan->num_small_mid++;
      continue;
    }
    const uint32_t P = std::max<uint32_t>(1, (hd[i] + kHubBigKeys - 1) / kHubBigKeys);
    const uint32_t hb = static_cast<uint32_t>(big_v.size());
    big_v.push_back(hv[i]);
    if (P >= kHubGlobalParts) {
      const uint32_t gi = static_cast<uint32_t>(glob_hub.size());
      big_glob.push_back(gi);
      glob_hub.push_back(hb);
      glob_base.push_back(plan->glob_slots);
      const uint32_t gcap = 2 * hd[i] + 2;
      glob_cap.push_back(gcap);
      plan->glob_slots += gcap;
      glob_sbase.push_back(static_cast<uint32_t>(slice_hub.size()));
      glob_nslices.push_back((gcap + kHubGlobalSlice - 1) / kHubGlobalSlice);
      for (uint32_t s0 = 0; s0 < gcap; s0 += kHubGlobalSlice) {
        slice_hub.push_back(gi);
        slice_start.push_back(s0);
      }
      for (uint32_t e = 0; e < hd[i]; e += kGlobChunk) {
        glob_item.push_back(gi);
        glob_item_start.push_back(e);
      }
    } else {
      big_glob.push_back(kNone);
    }
    for (uint32_t e = 0; e < hd[i]; e += kLoopChunk) {
      chunk_hub.push_back(hb);
      chunk_start.push_back(e);
    }
    if (g.m <= kLoopMaxEntries) {
      const uint32_t cap = 2 * hd[i] + 2;
      loop_base.push_back(plan->loop_slots);
      plan->loop_slots += cap;
      loop_cap.push_back(cap);
      loop_nslices.push_back((cap + kLoopSlice - 1) / kLoopSlice);
      loop_sbase.push_back(static_cast<uint32_t>(loop_slice_hub.size()));
      for (uint32_t s0 = 0; s0 < cap; s0 += kLoopSlice) {
        loop_slice_hub.push_back(hb);
        loop_slice_start.push_back(s0);
      }
    }
    parts.push_back(P);
    pbase.push_back(static_cast<uint32_t>(total));
    total += P;
    if (P > 1) {
      plan->num_multi = hb + 1;
      plan->num_multi_items = static_cast<uint32_t>(total);
    }
    for (uint32_t p = 0; p < P; ++p) {
      item_hub.push_back(hb);
      item_part.push_back(p);
    }
  }
  if (total > 0xFFFFFFFFull) return MakeError(PCC_OUT_OF_RANGE, "too many hub partitions");
  plan->num_small = static_cast<uint32_t>(small_v.size());
  plan->num_big = static_cast<uint32_t>(big_v.size());
  plan->num_items = static_cast<uint32_t>(item_hub.size());
  plan->num_partials = total;
  // One upload for the 32-bit lists, one for the 64-bit ones.
  std::vector<uint32_t> pack;
  std::vector<std::pair<const uint32_t**, size_t>> at;
  auto add = [&](const uint32_t** field, const std::vector<uint32_t>& x) {
    at.emplace_back(field, pack.size());
    pack.insert(pack.end(), x.begin(), x.end());
  };
  add(&plan->small_v, small_v);
  add(&plan->big_v, big_v);
  add(&plan->big_parts, parts);
  add(&plan->big_pbase, pbase);
  add(&plan->item_hub, item_hub);
  add(&plan->item_part, item_part);
  plan->num_glob = static_cast<uint32_t>(glob_hub.size());
  plan->num_glob_items = static_cast<uint32_t>(glob_item.size());
  plan->num_glob_slices = static_cast<uint32_t>(slice_hub.size());
  if (plan->num_glob) {
    add(&plan->big_glob, big_glob);
    add(&plan->glob_hub, glob_hub);
    add(&plan->glob_cap, glob_cap);
    add(&plan->glob_item, glob_item);
    add(&plan->glob_item_start, glob_item_start);
    add(&plan->glob_nslices, glob_nslices);
    add(&plan->glob_sbase, glob_sbase);
    add(&plan->slice_hub, slice_hub);
    add(&plan->slice_start, slice_start);
  }
  std::vector<unsigned long long> pack64 = glob_base;
  const size_t loop_base_at = pack64.size();
  pack64.insert(pack64.end(), loop_base.begin(), loop_base.end());
  plan->num_chunks = static_cast<uint32_t>(chunk_hub.size());
  plan->num_loop_slices = static_cast<uint32_t>(loop_slice_hub.size());
  add(&plan->loop_cap, loop_cap);
  add(&plan->loop_nslices, loop_nslices);
  add(&plan->loop_sbase, loop_sbase);
  add(&plan->chunk_hub, chunk_hub);
  add(&plan->chunk_start, chunk_start);
  add(&plan->loop_slice_hub, loop_slice_hub);
  add(&plan->loop_slice_start, loop_slice_start);
  PCC_RETURN_IF_ERROR(plan->pack.Alloc(ctx, std::max<size_t>(pack.size(), 1)));
  PCC_RETURN_IF_ERROR(plan->pack.FromHost(pack.data(), pack.size()));
  for (const auto& f : at) *f.first = plan->pack.p + f.second;
  if (!pack64.empty()) {
    PCC_RETURN_IF_ERROR(plan->pack64.Alloc(ctx, pack64.size()));
    PCC_RETURN_IF_ERROR(plan->pack64.FromHost(pack64.data(), pack64.size()));
    plan->glob_base = plan->pack64.p;
    plan->loop_base = plan->pack64.p + loop_base_at;
  }
  return Status::Ok();  // (the host lists are spent; EnsureHubPlan waits for the device where it must)
}

namespace {

Status AllocTables(Context* ctx, uint64_t slots, uint32_t hubs, uint32_t slices, HubState* st, bool reset) {
  if (!slots) return Status::Ok();
  if (st->gkeys.count < slots || st->gt_int.count < hubs || st->gpart_val.count < slices) {
    auto grow = [&]() -> Status {
      if (st->gkeys.count < slots) {
        PCC_RETURN_IF_ERROR(st->gkeys.Alloc(ctx, slots));
        PCC_RETURN_IF_ERROR(st->gvals.Alloc(ctx, slots));
      }
      if (st->gt_int.count < hubs) {
        PCC_RETURN_IF_ERROR(st->gt_int.Alloc(ctx, hubs));
        PCC_RETURN_IF_ERROR(st->gt_dbl.Alloc(ctx, hubs));
        PCC_RETURN_IF_ERROR(st->gsmax.Alloc(ctx, hubs));
        PCC_RETURN_IF_ERROR(st->gdone.Alloc(ctx, hubs));
      }
      if (st->gpart_val.count < slices) {
        PCC_RETURN_IF_ERROR(st->gpart_val.Alloc(ctx, slices));
        PCC_RETURN_IF_ERROR(st->gpart_id.Alloc(ctx, slices));
      }
      return Status::Ok();
    };
    const Status got = grow();
    if (!got.ok()) {
      st->ReleaseTables();
      return got;
    }
    reset = true;
  }
  if (!reset) return Status::Ok();
  // The rounds leave the tables clean; they are cleared at every new level all
  // the same, so that a run cut short cannot leave keys behind.
  PCC_CUDA(cudaMemsetAsync(st->gkeys.p, 0xFF, slots * sizeof(uint32_t), ctx->stream));  // kNone
  PCC_CUDA(cudaMemsetAsync(st->gvals.p, 0, slots * sizeof(unsigned long long), ctx->stream));
  GlobalStateInitKernel<<<Blocks(hubs, 256, 1024), 256, 0, ctx->stream>>>(hubs, st->gt_int.p, st->gt_dbl.p,
                                                                          st->gsmax.p, st->gdone.p);
  PCC_COUNT(1);
  return LaunchCheck();
}

}  // namespace

Status AllocHubState(Context* ctx, const HubPlan& plan, HubState* st, bool reset) {
  const uint64_t np = std::max<uint64_t>(plan.num_partials, 1);
  if (st->part_val.count < np) {
    PCC_RETURN_IF_ERROR(st->part_val.Alloc(ctx, np));
    PCC_RETURN_IF_ERROR(st->part_id.Alloc(ctx, np));
  }
  const uint64_t nh = std::max<uint32_t>(plan.num_big, 1);
  if (st->done.count < nh) {
    PCC_RETURN_IF_ERROR(st->done.Alloc(ctx, nh));
    reset = true;
  }
  PCC_RETURN_IF_ERROR(AllocTables(ctx, plan.glob_slots, plan.num_glob, plan.num_glob_slices, st, reset));
  return reset ? st->done.Zero() : Status::Ok();
}

Status AllocLoopTables(Context* ctx, const HubPlan& plan, HubState* st, bool reset) {
  return AllocTables(ctx, plan.loop_slots, plan.num_big, plan.num_loop_slices, st, reset);
}

namespace {

Status PrepareAllHubKernels() {
  bool ok = true;
  auto small = [&](auto k, size_t slots, size_t vsize) {
    ok = ok && PrepareOnce(k, kSmallThreads, slots * (vsize + sizeof(uint32_t))) > 0;
  };
  auto big = [&](auto k, size_t slots, size_t vsize) {
    ok = ok && PrepareOnce(k, kBigThreads, slots * (vsize + sizeof(uint32_t))) > 0;
  };
  small(HubSmallKernel<false, false, double, kSmallMidSlots>, kSmallMidSlots, sizeof(double));
  small(HubSmallKernel<false, false, double, kSmallSlots>, kSmallSlots, sizeof(double));
  small(HubSmallKernel<false, false, double, kSmallNarrowSlots>, kSmallNarrowSlots, sizeof(double));
  auto cert = [&](auto sum, auto conv) {
    using V = decltype(sum);
    constexpr bool kC = decltype(conv)::value;
    ok = ok && PrepareOnce(HubCertKernel<2 * kHubSmallMax, 16, V, kC>, 512, HubCertSmem<2 * kHubSmallMax, 16, V>()) > 0 &&
         PrepareOnce(HubCertKernel<kHubSmallMax, 8, V, kC>, 256, HubCertSmem<kHubSmallMax, 8, V>()) > 0 &&
         PrepareOnce(HubCertKernel<16384, 32, V, kC>, 1024, HubCertSmem<16384, 32, V>()) > 0;
  };
  cert(0, std::false_type{});
  cert(0, std::true_type{});
  cert(0ll, std::true_type{});
  big(HubBigKernel<true, false, int>, BigSlots<int>(), sizeof(int));
  big(HubBigKernel<true, false, long long>, BigSlots<long long>(), sizeof(long long));
  big(HubBigKernel<false, false, double>, BigSlots<double>(), sizeof(double));
  return ok ? Status::Ok() : MakeError(PCC_INTERNAL, "hub kernels cannot be configured");
}

}  // namespace

Status PrepareHubKernels() {
  static PerDevice done;
  return OncePerDevice(done, PrepareAllHubKernels);
}

Status LaunchHubBestMoves(Context* ctx, const BMArgs& a, const HubPlan& plan, HubState& st, bool int_mode,
                          bool narrow, int families) {
  if (plan.num_hubs == 0) return Status::Ok();
  HubArgs h;
  h.a = a;
  h.small_v = plan.small_v;
  h.small_lo = 0;
  h.small_hi = plan.num_small;
  h.big_v = plan.big_v;
  h.big_parts = plan.big_parts;
  h.big_pbase = plan.big_pbase;
  h.item_hub = plan.item_hub;
  h.item_part = plan.item_part;
  h.num_items = plan.num_items;
  h.part_val = st.part_val.p;
  h.part_id = st.part_id.p;
  h.done = st.done.p;
  h.num_glob = plan.num_glob;
  h.num_glob_items = plan.num_glob_items;
  h.glob_hub = plan.glob_hub;
  h.glob_base = plan.glob_base;
  h.glob_cap = plan.glob_cap;
  h.glob_item = plan.glob_item;
  h.glob_item_start = plan.glob_item_start;
  h.big_glob = plan.big_glob;
  h.gkeys = st.gkeys.p;
  h.gvals = st.gvals.p;
  h.gt_int = st.gt_int.p;
  h.gt_dbl = st.gt_dbl.p;
  h.gsmax = st.gsmax.p;
  h.num_glob_slices = plan.num_glob_slices;
  h.glob_nslices = plan.glob_nslices;
  h.glob_sbase = plan.glob_sbase;
  h.slice_hub = plan.slice_hub;
  h.slice_start = plan.slice_start;
  h.gpart_val = st.gpart_val.p;
  h.gpart_id = st.gpart_id.p;
  h.gdone = st.gdone.p;
  if (a.async) {
    if (!int_mode) return LaunchHubT<false, true, double>(ctx, h, plan, families);
    return narrow ? LaunchHubT<true, true, int>(ctx, h, plan, families)
                  : LaunchHubT<true, true, long long>(ctx, h, plan, families);
  }
  if (!int_mode) return LaunchHubT<false, false, double>(ctx, h, plan, families);
  return narrow ? LaunchHubT<true, false, int>(ctx, h, plan, families)
                : LaunchHubT<true, false, long long>(ctx, h, plan, families);
}

}  // namespace pcc
