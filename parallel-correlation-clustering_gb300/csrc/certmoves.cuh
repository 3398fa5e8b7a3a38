// certmoves.cuh -- the certified best move of one vertex (INT mode,
// synchronous rounds), by a lane group, a warp or a team of warps: the bodies
// shared by the degree-binned kernels (bestmove.cu) and the kernel that runs
// a whole level's rounds (roundloop.cu).
#pragma once

#include "certify.cuh"
#include "moves.cuh"

namespace pcc {
namespace {

constexpr int kCertUnroll = 4;  // chunks of 32 entries loaded together
constexpr int kCertRegRounds = 1;  // candidates per lane held in registers
constexpr int kCtaWarps = 4;  // warps of a team on a vertex of degree 257-1000

// ---------------------------------------------------------------------------
// INT-mode synchronous rounds: certified decisions (certify.cuh).  The FP32
// pre-filter selects the survivors; when they form one (S, K) class and the
// FP32 bounds decide the move, no FP64 instruction runs for the vertex.
// Otherwise -- and always in replay mode, where the exact values are outputs
// -- the exact FP64 values decide; in replay mode a certified decision that
// differs from the FP64 one raises kErrCertMismatch (a self-check).
// ---------------------------------------------------------------------------
// Exact FP64 fallbacks of the certified kernels.  They are separate
// non-inlined functions so that the compiler cannot hoist their FP64
// arithmetic onto the certified path (an FP64 warp instruction costs ~19
// SM cycles on this GPU).  Both return whether the vertex must be appended
// to the movers list; in replay mode they also run the self-check.
template <int G, typename V>
__device__ __noinline__ bool GroupExact(const BMArgs& a, const VertexCtx& x, bool fp64, bool contender, unsigned gl,
                                        V T, V S, double KD, uint32_t cu, bool replay, int cres,
                                        uint32_t cmove, uint32_t stamp) {
  double change = 0.0, val = -CUDART_INF;
  uint32_t id = kNone;
  if (fp64) {
    change = ChangeOf(a, x, UnitsToDouble<V>(a, T));
    if (contender) {
      val = ValOf(a, x, change, UnitsToDouble<V>(a, S), KD);
      id = cu;
    }
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
  if (fp64 && gl == 0) {
    append = Decide<false>(a, x, val, id, change, stamp);
    if (replay && cres != kUncertain && a.out_moves && a.out_moves[x.v] != cmove)
      atomicExch(&a.ctr->error, kErrCertMismatch);
  }
  return append;
}

template <int HC, typename V>
__device__ __noinline__ bool WarpExact(const BMArgs& a, const VertexCtx& x, V T, const uint32_t* keys,
                                       const V* vals, const uint16_t* used, uint32_t nused, bool replay, int cres,
                                       uint32_t cmove, uint32_t stamp) {
  const unsigned lane = LaneId();
  const double change = ChangeOf(a, x, UnitsToDouble<V>(a, T));
  double best = -CUDART_INF;
  uint32_t bid = kNone;
  for (uint32_t i = lane; i < nused; i += 32) {
    const uint32_t slot = used[i];
    if (slot == 0xFFFFu) continue;
    const uint32_t key = keys[slot];
    const double val = ValOf(a, x, change, UnitsToDouble<V>(a, vals[slot]), a.K[key]);
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
  bool append = false;
  if (lane == 0) {
    append = Decide<false>(a, x, best, bid, change, stamp);
    if (replay && cres != kUncertain && a.out_moves && a.out_moves[x.v] != cmove)
      atomicExch(&a.ctr->error, kErrCertMismatch);
  }
  return append;
}

template <typename V>
__device__ __forceinline__ V WarpMaxV(V x) {
  if constexpr (sizeof(V) == 4) return __reduce_max_sync(kFull, x);
  else return WarpMaxLL(x);
}

// Lane groups of G lanes, one vertex (degree <= G) per group: vid is the
// group's vertex when `in`.  Returns whether this lane's vertex must be
// appended to the movers list (the group's first lane).  stage: 32 values of
// the calling warp.  V: int when every sum of a row fits in 32 bits, else long
// long.
template <int G, typename V, class L>
__device__ __forceinline__ bool GroupStep(const BMArgs& a, const RoundView& rv, bool in, uint32_t vid, V* stage,
                                          bool replay, unsigned long long& fam_e, unsigned long long& fam_v) {
  const unsigned lane = LaneId();
  const unsigned g = lane / G, gl = lane % G;
  const unsigned gmask = G == 32 ? kFull : (((1u << G) - 1u) << (g * G));
  const bool unit = a.w == nullptr;
  bool vvalid = in;
  VertexCtx x{};
  if (vvalid) {
    vvalid = InFront(a, rv, vid);
    if (vvalid) x = LoadVertexAs<L>(a, vid);
  }
  if (__ballot_sync(kFull, vvalid) == 0) return false;  // no frontier vertex in this warp
  if (vvalid && gl == 0) {
    fam_e += x.d;
    fam_v += 1;
  }
  const bool has = vvalid && gl < x.d;
  uint32_t u = x.v;
  float wt = 0.f;
  if (has) {
    u = a.nbr[x.b + gl];
    wt = a.w ? a.w[x.b + gl] : 1.0f;
  }
  const bool cand = has && u != x.v;
  const uint32_t cu = cand ? L::C(a.C + u) : kNone;
  const unsigned peers = __match_any_sync(kFull, cand ? cu : LaneSentinel(lane)) & gmask;
  const bool leader = cand && int(lane) == __ffs(peers) - 1;
  const V xi = cand ? EntryUnits<V, true>(a, wt) : V(0);
  const V S = GroupSumInt<V>(peers, xi, unit, leader, stage);
  const unsigned tmask = __ballot_sync(kFull, leader && cu == x.c) & gmask;
  const V Tsh = __shfl_sync(kFull, S, tmask ? __ffs(tmask) - 1 : int(lane));
  const V T = tmask ? Tsh : V(0);
  V smax = leader ? S : (sizeof(V) == 4 ? V(INT_MIN) : V(LLONG_MIN));
  if constexpr (G == 32) {
    smax = WarpMaxV<V>(smax);
  } else {
#pragma unroll
    for (int o = G / 2; o >= 1; o >>= 1) smax = max(smax, __shfl_xor_sync(kFull, smax, o));
  }
  const float k32 = vvalid ? a.kf[x.v] : 0.f;
  const float Kc32 = vvalid ? a.Kf[x.c] : 0.f;
  const ChangeApproxT<V> ca = ApproxChange<V>(Res32Of(a, x.v), a.int_nw != 0, k32, Kc32, T);
  const float cabs = ChangeAbsBound(ca);
  // FP32 pre-filter over the group's leaders.
  FilterVal f{0.f, 0.f, false};
  float KfD = 0.f;
  float lo = -CUDART_INF_F;
  if (leader) {
    KfD = a.Kf[cu];
    f = FilterOf<V>(Res32Of(a, x.v), k32, KfD, S, smax, cabs);
    if (f.sane) lo = __fsub_rn(f.Y, f.e);
  }
  float U = lo;
  if constexpr (G == 32) {
    U = WarpMaxFinite(U);
  } else {
#pragma unroll
    for (int o = G / 2; o >= 1; o >>= 1) U = fmaxf(U, __shfl_xor_sync(kFull, U, o));
  }
  const bool contender = leader && (!f.sane || __fadd_rn(f.Y, f.e) >= U);
  // The leading (S, K) class of the contenders and the trailing one.
  LexKeyT<V> lead, tail;
  double KD = 0.0;
  if (contender) {
    KD = L::K(a.K + cu);
    const unsigned long long ko = KOrder(KD);
    lead.Keep(S, ko, cu);
    tail.Keep(-S, ~ko, cu);
  }
  bool single;
  if constexpr (G == 32) {
    single = LexWarpLead<V>(lead, tail);
  } else {
    LexGroupReduce<G>(lead);
    LexGroupReduce<G>(tail);
    single = lead.id == kNone || (-tail.S == lead.S && ~tail.K == lead.K);
  }
  int cres = kUncertain;
  uint32_t ctarget = kNone;
  if (vvalid && single) {
    const float KfA = lead.id != kNone ? a.Kf[lead.id] : 0.f;
    cres = CertifyDecision<V>(ca, Res32Of(a, x.v), k32, lead.id != kNone, lead.S, KfA, lead.id, a.n, &ctarget);
  }
  const uint32_t cmove = cres == kUncertain ? kNone : CertifiedMove(a, x, ctarget, cres == kCertMove);
  const bool fp64 = vvalid && (replay || cres == kUncertain);
  bool append = false;
  if (vvalid && !fp64 && gl == 0) append = ApplyCertified(a, x, cmove, rv.stamp);
  if (__ballot_sync(kFull, fp64)) {
    const bool app = GroupExact<G, V>(a, x, fp64, contender, gl, T, S, KD, cu, replay, cres, cmove,
                                       rv.stamp);
    append = append || app;
  }
  return append;
}

// One warp, one vertex x of degree <= HC / 2: the warp's table (vals, keys,
// HC slots, and the list of used slots) is clean before and after.  Returns
// (on lane 0) whether the vertex must be appended to the movers list.
// V: int when every cluster sum fits in 32 bits (narrow), else long long.
// Every entry inserts its cluster itself (atomicCAS claims a slot) and adds
// its integer weight with a shared-memory atomic: INT-mode sums are exact in
// any order, and grouping equal clusters first with match.any cost more than
// the atomics it saves.
template <int HC, typename V, bool kConv, class L>
__device__ __forceinline__ bool WarpStep(const BMArgs& a, const RoundView& rv, const VertexCtx& x, V* vals,
                                         uint32_t* keys, uint16_t* used, bool replay) {
  const unsigned lane = LaneId();
  uint32_t nused = 0;  // used[] entries (warp-uniform)
  V tpart = 0;         // this lane's part of T (entries in the vertex's own cluster)
  for (uint32_t e0 = 0; e0 < x.d; e0 += 32 * kCertUnroll) {
    uint32_t uu[kCertUnroll], cc[kCertUnroll];
    float ww[kCertUnroll];
#pragma unroll
    for (int k = 0; k < kCertUnroll; ++k) {
      const uint32_t e = e0 + 32 * k + lane;
      uu[k] = x.v;
      ww[k] = 0.f;
      if (e < x.d) {
        uu[k] = a.nbr[x.b + e];
        ww[k] = a.w ? a.w[x.b + e] : 1.0f;
      }
    }
#pragma unroll
    for (int k = 0; k < kCertUnroll; ++k) cc[k] = uu[k] != x.v ? L::C(a.C + uu[k]) : kNone;
#pragma unroll
    for (int k = 0; k < kCertUnroll; ++k) {
    if (e0 + 32 * k >= x.d) break;  // warp-uniform
    const float wt = ww[k];
    const bool cand = uu[k] != x.v;
    const uint32_t cu = cc[k];
    uint32_t slot = kNone;
    bool ins = false;
    if (cand) {
      slot = FindOrInsertT<false>(keys, HC, cu, &ins);
      if (slot == kNone) atomicExch(&a.ctr->error, kErrHashFull);
    }
    const unsigned im = __ballot_sync(kFull, ins);
    if (im) {
      if (ins) used[nused + __popc(im & LaneMaskLt())] = static_cast<uint16_t>(slot);
      nused += __popc(im);
    }
    const V xi = cand ? EntryUnits<V, kConv>(a, wt) : V(0);
    if (cand && cu == x.c) tpart += xi;
    if (slot != kNone) SharedAdd(&vals[slot], xi);
    __syncwarp();
    }
  }
  // T: the lanes' own-cluster parts.
  V T;
  if constexpr (sizeof(V) == 4) {
    T = __reduce_add_sync(kFull, tpart);
  } else {
    T = tpart;
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) T += __shfl_xor_sync(kFull, T, o);
  }
  const float r32 = Res32Of(a, x.v);
  const float k32 = a.kf[x.v];
  const ChangeApproxT<V> ca = ApproxChange<V>(r32, a.int_nw != 0, k32, a.Kf[x.c], T);
  const float cabs = ChangeAbsBound(ca);
  // The first kCertRegRounds candidates of each lane (i = lane + 32 r) keep
  // their slot, sum, Kf and filter value in registers across the passes;
  // any further ones are read again.
  uint32_t rslot[kCertRegRounds];
  V rS[kCertRegRounds];
  float rKf[kCertRegRounds];
  V vmax = sizeof(V) == 4 ? V(INT_MIN) : V(LLONG_MIN);
#pragma unroll
  for (int r = 0; r < kCertRegRounds; ++r) {
    const uint32_t i = lane + 32 * r;
    rslot[r] = 0xFFFFu;
    rS[r] = 0;
    rKf[r] = 0.f;
    if (i < nused) {
      rslot[r] = used[i];
      rS[r] = vals[rslot[r]];
      rKf[r] = a.Kf[keys[rslot[r]]];
      vmax = max(vmax, rS[r]);
    }
  }
  for (uint32_t i = lane + 32 * kCertRegRounds; i < nused; i += 32) vmax = max(vmax, vals[used[i]]);
  const V smax = WarpMaxV<V>(vmax);
  float U = -CUDART_INF_F;
  // The two largest upper ends (Y + e; +inf outside the error model) of
  // this lane's candidates and the index of the largest: when the second
  // is below U, only that one can be a contender.  Kept for the bins of
  // more than 128 entries, where lanes hold several candidates (in the
  // 33-128 bin it costs about what it saves).
  constexpr bool kTop2 = HC >= 512;
  float hi1 = -CUDART_INF_F, hi2 = -CUDART_INF_F;
  uint32_t i1 = kNone;
  FilterVal rf[kCertRegRounds];
#pragma unroll
  for (int r = 0; r < kCertRegRounds; ++r) {
    rf[r].sane = false;
    if (lane + 32 * r < nused) {
      rf[r] = FilterOf<V>(r32, k32, rKf[r], rS[r], smax, cabs);
      if (rf[r].sane) U = fmaxf(U, __fsub_rn(rf[r].Y, rf[r].e));
      if (kTop2) KeepTop2(hi1, hi2, i1, rf[r].sane ? __fadd_rn(rf[r].Y, rf[r].e) : CUDART_INF_F, lane + 32 * r);
    }
  }
  for (uint32_t i = lane + 32 * kCertRegRounds; i < nused; i += 32) {
    const uint32_t slot = used[i];
    const FilterVal f = FilterOf<V>(r32, k32, a.Kf[keys[slot]], vals[slot], smax, cabs);
    if (f.sane) U = fmaxf(U, __fsub_rn(f.Y, f.e));
    if (kTop2) KeepTop2(hi1, hi2, i1, f.sane ? __fadd_rn(f.Y, f.e) : CUDART_INF_F, i);
  }
  U = WarpMaxFinite(U);
  LexKeyT<V> lead, tail;
  // The contenders are the candidates with Y + e >= U (all when U = -inf).
  const bool skip = kTop2 && hi2 < U;
  if (skip) {
    // At most candidate i1 is a contender: the others are cleared and
    // marked without evaluating them again.
    for (uint32_t i = lane; i < nused; i += 32) {
      const uint32_t slot = used[i];
      if (i == i1 && !(hi1 < U)) {
        const uint32_t key = keys[slot];
        const V S = vals[slot];
        const unsigned long long ko = KOrder(L::K(a.K + key));
        lead.Keep(S, ko, key);
        tail.Keep(-S, ~ko, key);
        continue;
      }
      keys[slot] = kNone;
      vals[slot] = 0;
      used[i] = 0xFFFFu;
    }
  }
  const uint32_t rescan_end = skip ? 0u : nused;
#pragma unroll
  for (int r = 0; r < kCertRegRounds; ++r) {
    const uint32_t i = lane + 32 * r;
    if (i >= rescan_end) continue;
    const uint32_t slot = rslot[r];
    if (rf[r].sane && __fadd_rn(rf[r].Y, rf[r].e) < U) {
      keys[slot] = kNone;  // not a contender: cleared now, skipped later
      vals[slot] = 0;
      used[i] = 0xFFFFu;
      continue;
    }
    const uint32_t key = keys[slot];
    const unsigned long long ko = KOrder(L::K(a.K + key));
    lead.Keep(rS[r], ko, key);
    tail.Keep(-rS[r], ~ko, key);
  }
  for (uint32_t i = lane + 32 * kCertRegRounds; i < rescan_end; i += 32) {
    const uint32_t slot = used[i];
    const uint32_t key = keys[slot];
    const FilterVal f = FilterOf<V>(r32, k32, a.Kf[key], vals[slot], smax, cabs);
    if (f.sane && __fadd_rn(f.Y, f.e) < U) {
      keys[slot] = kNone;  // not a contender: cleared now, skipped later
      vals[slot] = 0;
      used[i] = 0xFFFFu;
      continue;
    }
    const unsigned long long ko = KOrder(L::K(a.K + key));
    const V S = vals[slot];
    lead.Keep(S, ko, key);
    tail.Keep(-S, ~ko, key);
  }
  const bool single = LexWarpLead<V>(lead, tail);
  int cres = kUncertain;
  uint32_t ctarget = kNone;
  if (single) {
    const float KfA = lead.id != kNone ? a.Kf[lead.id] : 0.f;
    cres = CertifyDecision<V>(ca, r32, k32, lead.id != kNone, lead.S, KfA, lead.id, a.n, &ctarget);
  }
  const uint32_t cmove = cres == kUncertain ? kNone : CertifiedMove(a, x, ctarget, cres == kCertMove);
  bool append = false;
  if (replay || cres == kUncertain) {
    append = WarpExact<HC, V>(a, x, T, keys, vals, used, nused, replay, cres, cmove, rv.stamp);
  } else if (lane == 0) {
    append = ApplyCertified(a, x, cmove, rv.stamp);
  }
  __syncwarp();
  // Clear the table through the key list (used[] may hold 0xFFFF marks).
  for (uint32_t i = lane; i < nused; i += 32) {
    const uint32_t slot = used[i];
    if (slot != 0xFFFFu) {
      keys[slot] = kNone;
      vals[slot] = 0;
    }
  }
  return append;
}

// Barrier of a team of BT threads of a CTA (bar: its hardware barrier, 0-15).
template <int BT>
__device__ __forceinline__ void TeamSync(unsigned bar) {
  asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(BT) : "memory");
}

template <typename V, int TW = kCtaWarps>
struct CtaShared {
  uint32_t nused;  // 0 between vertices
  V max[TW];
  float u[TW];
  V ls[TW], ts[TW];
  unsigned long long lk[TW], tk[TW];
  uint32_t li[TW], ti[TW];
};

// A team of TW warps (its thread index tid) on one vertex x of degree
// <= HC / 2, with the team's table (clean before and after, as sh.nused) and
// hardware barrier.  Returns (on thread 0) whether the vertex must be
// appended to the movers list.
template <int HC, typename V, bool kConv, class L, int TW = kCtaWarps>
__device__ __forceinline__ bool CtaStep(const BMArgs& a, const RoundView& rv, const VertexCtx& x, V* vals,
                                        uint32_t* keys, uint16_t* used, CtaShared<V, TW>& sh, unsigned tid,
                                        unsigned bar, bool replay) {
  constexpr int BT = TW * 32;
  const unsigned lane = tid & 31, warp = tid >> 5;
  bool append = false;
  for (uint32_t e0 = 0; e0 < x.d; e0 += BT * kCertUnroll) {
    uint32_t uu[kCertUnroll], cc[kCertUnroll];
    float ww[kCertUnroll];
#pragma unroll
    for (int k = 0; k < kCertUnroll; ++k) {
      const uint32_t e = e0 + BT * k + tid;
      uu[k] = x.v;
      ww[k] = 0.f;
      if (e < x.d) {
        uu[k] = a.nbr[x.b + e];
        ww[k] = a.w ? a.w[x.b + e] : 1.0f;
      }
    }
#pragma unroll
    for (int k = 0; k < kCertUnroll; ++k) cc[k] = uu[k] != x.v ? L::C(a.C + uu[k]) : kNone;
#pragma unroll
    for (int k = 0; k < kCertUnroll; ++k) {
      if (e0 + BT * k + 32 * warp >= x.d) break;  // uniform over the warp
      const bool cand = uu[k] != x.v;
      const uint32_t cu = cc[k];
      uint32_t slot = kNone;
      bool ins = false;
      if (cand) {
        slot = FindOrInsertT<false>(keys, HC, cu, &ins);
        if (slot == kNone) atomicExch(&a.ctr->error, kErrHashFull);
      }
      const unsigned im = __ballot_sync(kFull, ins);
      if (im) {
        const int first = __ffs(im) - 1;
        uint32_t base = 0;
        if (int(lane) == first) base = atomicAdd(&sh.nused, uint32_t(__popc(im)));
        base = __shfl_sync(kFull, base, first);
        if (ins) used[base + __popc(im & LaneMaskLt())] = static_cast<uint16_t>(slot);
      }
      const V xi = cand ? EntryUnits<V, kConv>(a, ww[k]) : V(0);
      if (slot != kNone) SharedAdd(&vals[slot], xi);
    }
  }
  TeamSync<BT>(bar);  // table complete
  const uint32_t nused = sh.nused;
  V T = 0;
  {
    const uint32_t slot = FindT<false>(keys, HC, x.c);
    if (slot != kNone) T = vals[slot];
  }
  const float k32 = a.kf[x.v];
  const ChangeApproxT<V> ca = ApproxChange<V>(Res32Of(a, x.v), a.int_nw != 0, k32, a.Kf[x.c], T);
  const float cabs = ChangeAbsBound(ca);
  V vmax = sizeof(V) == 4 ? V(INT_MIN) : V(LLONG_MIN);
  for (uint32_t i = tid; i < nused; i += BT) vmax = max(vmax, vals[used[i]]);
  vmax = WarpMaxV<V>(vmax);
  if (lane == 0) sh.max[warp] = vmax;
  TeamSync<BT>(bar);
  V smax = sh.max[0];
#pragma unroll
  for (int w = 1; w < TW; ++w) smax = max(smax, sh.max[w]);
  float U = -CUDART_INF_F;
  float hi1 = -CUDART_INF_F, hi2 = -CUDART_INF_F;  // KeepTop2 of this thread's candidates
  uint32_t i1 = kNone;
  for (uint32_t i = tid; i < nused; i += BT) {
    const uint32_t slot = used[i];
    const FilterVal f = FilterOf<V>(Res32Of(a, x.v), k32, a.Kf[keys[slot]], vals[slot], smax, cabs);
    if (f.sane) U = fmaxf(U, __fsub_rn(f.Y, f.e));
    KeepTop2(hi1, hi2, i1, f.sane ? __fadd_rn(f.Y, f.e) : CUDART_INF_F, i);
  }
  U = WarpMaxFinite(U);
  if (lane == 0) sh.u[warp] = U;
  TeamSync<BT>(bar);
  U = sh.u[0];
#pragma unroll
  for (int w = 1; w < TW; ++w) U = fmaxf(U, sh.u[w]);
  LexKeyT<V> lead, tail;
  // The contenders are the candidates with Y + e >= U (all when U = -inf);
  // when this thread's runner-up is below U, at most its candidate i1 is
  // one, and the others are cleared and marked without a second
  // evaluation.
  const bool rescan = !(hi2 < U);
  if (!rescan) {
    for (uint32_t i = tid; i < nused; i += BT) {
      const uint32_t slot = used[i];
      if (i == i1 && !(hi1 < U)) {
        const uint32_t key = keys[slot];
        const V S = vals[slot];
        const unsigned long long ko = KOrder(L::K(a.K + key));
        lead.Keep(S, ko, key);
        tail.Keep(-S, ~ko, key);
        continue;
      }
      keys[slot] = kNone;
      vals[slot] = 0;
      used[i] = 0xFFFFu;
    }
  }
  for (uint32_t i = tid; i < (rescan ? nused : 0u); i += BT) {
    const uint32_t slot = used[i];
    const uint32_t key = keys[slot];
    const FilterVal f = FilterOf<V>(Res32Of(a, x.v), k32, a.Kf[key], vals[slot], smax, cabs);
    if (f.sane && __fadd_rn(f.Y, f.e) < U) {
      keys[slot] = kNone;  // not a contender: cleared now, skipped later
      vals[slot] = 0;
      used[i] = 0xFFFFu;
      continue;
    }
    const unsigned long long ko = KOrder(L::K(a.K + key));
    const V S = vals[slot];
    lead.Keep(S, ko, key);
    tail.Keep(-S, ~ko, key);
  }
  LexWarpLeader<V>(lead);
  LexWarpLeader<V>(tail);
  if (lane == 0) {
    sh.ls[warp] = lead.S;
    sh.lk[warp] = lead.K;
    sh.li[warp] = lead.id;
    sh.ts[warp] = tail.S;
    sh.tk[warp] = tail.K;
    sh.ti[warp] = tail.id;
  }
  TeamSync<BT>(bar);
  if (warp == 0) {
    LexKeyT<V> top, low;
#pragma unroll
    for (int w = 0; w < TW; ++w) {
      top.Keep(sh.ls[w], sh.lk[w], sh.li[w]);
      low.Keep(sh.ts[w], sh.tk[w], sh.ti[w]);
    }
    // One (S, K) class among the contenders iff the lowest-ranked one
    // (low: smallest S, then largest K) is in the leader's class.
    const bool single = top.id == kNone || (-low.S == top.S && ~low.K == top.K);
    int cres = kUncertain;
    uint32_t ctarget = kNone;
    if (single) {
      const float KfA = top.id != kNone ? a.Kf[top.id] : 0.f;
      cres = CertifyDecision<V>(ca, Res32Of(a, x.v), k32, top.id != kNone, top.S, KfA, top.id, a.n, &ctarget);
    }
    const uint32_t cmove = cres == kUncertain ? kNone : CertifiedMove(a, x, ctarget, cres == kCertMove);
    if (TW > kCtaWarps && nused == 0) {
      // A hub whose entries are all self-loops: the reduce identity (0, 0.0).
      if (lane == 0) append = Decide<false>(a, x, 0.0, 0, ChangeOf(a, x, 0.0), rv.stamp);
    } else if (replay || cres == kUncertain) {
      append = WarpExact<HC, V>(a, x, T, keys, vals, used, nused, replay, cres, cmove, rv.stamp);
    } else if (lane == 0) {
      append = ApplyCertified(a, x, cmove, rv.stamp);
    }
  }
  TeamSync<BT>(bar);  // the table is read by WarpExact up to here
  for (uint32_t i = tid; i < nused; i += BT) {
    const uint32_t slot = used[i];
    if (slot != 0xFFFFu) {
      keys[slot] = kNone;
      vals[slot] = 0;
    }
  }
  if (tid == 0) sh.nused = 0;
  TeamSync<BT>(bar);
  return append;
}

}  // namespace
}  // namespace pcc
