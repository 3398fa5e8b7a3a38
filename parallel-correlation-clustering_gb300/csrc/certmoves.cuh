// certmoves.cuh -- the certified best move of a vertex (INT mode, synchronous
// rounds), by a lane group, a warp or a team of warps: the bodies shared by
// the degree-binned kernels (bestmove.cu) and the kernel that runs a whole
// level's rounds (roundloop.cu).
//
// A lane-group vertex (degree <= 32) is handled in two parts.  The scan gathers
// its entries, sums them per neighbour cluster and filters the candidates in
// FP32; the next step's rows are loaded meanwhile.  What is left of it, the
// together-sum and the leading class's sum and lowest id, waits in the lane of
// a Pending record.  The decision (certify.cuh: change, bounds, singleton
// rule, move) is then taken for up to 32 vertices at once, one per lane: taken
// vertex by vertex by the whole warp, that scalar part was about half of the
// 490 warp instructions that a vertex of degree 17-32 cost.  Lane-group kernels
// of a clustering: RMAT-22 21.8 -> 16.2 ms, 128 block models 26.8 -> 18.9,
// RMAT-20 correlation 19.0 -> 16.3.
// Vertices that the bounds do not decide although their leading class is known
// (5-10% of a correlation clustering's: moves of value 0) take their two FP64
// values in their lane; those whose contenders are of several (S, K) classes
// (below 1%) are scanned again and decided from every candidate's exact value.
#pragma once

#include <cmath>

#include "certify.cuh"
#include "moves.cuh"

namespace pcc {
namespace {

constexpr int kCertUnroll = 4;  // chunks of 32 entries loaded together
constexpr int kCertRegRounds = 1;  // candidates per lane held in registers
constexpr int kCtaWarps = 4;  // warps of a team on a vertex of degree 257-1000

template <typename V>
__device__ __forceinline__ V WarpAddV(V x) {
  if constexpr (sizeof(V) == 4) {
    return __reduce_add_sync(kFull, x);
  } else {
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) x += __shfl_xor_sync(kFull, x, o);
    return x;
  }
}

template <typename V>
__host__ __device__ constexpr V LowestV() {
  return sizeof(V) == 4 ? V(INT_MIN) : V(LLONG_MIN);
}
template <typename V>
__device__ __forceinline__ V WarpMaxV(V x) {
  if constexpr (sizeof(V) == 4) {
    return __reduce_max_sync(kFull, x);
  } else {
    return WarpMaxLL(x);
  }
}

// ---------------------------------------------------------------------------
// The filter.  A candidate's value is ordered by Y = (S - M) - R, R = res * kv
// * K, with M the largest sum: an exact integer difference, so that candidates
// of equal S are told apart by R alone (modularity's R is 1e-7 of S).  It is
// known in FP32 within
//   e = 2^-18 (|R| + |Y|) + base,  base = 2^-48 (|change| + |M|) and more:
// FilterBound (moves.cuh) with |S| <= |Y| + |R| + |M|, whose first two terms
// disappear in the margin of the first one.  Kf is FilterF32(K), so it is 0, in
// [2^-100, 2^100] or NaN; R outside that range (or NaN) makes the candidate
// a contender in any case.
// ---------------------------------------------------------------------------
struct VertexFilter {
  float r32, k32, base;
  bool ok;       // base is finite
  bool int_nw;
};

template <typename V>
__device__ __forceinline__ VertexFilter FilterFor(const BMArgs& a, uint32_t v, uint32_t c, V T, V M) {
  VertexFilter f;
  f.r32 = Res32Of(a, v);
  f.k32 = a.kf[v];
  const float kc = a.Kf[c];
  const float m = __fmul_rn(fabsf(__fmul_rn(f.r32, f.k32)), __fadd_rn(fabsf(kc), fabsf(f.k32)));
  f.base = __fmul_rn(3.6e-15f /* 1.01 * 2^-48 */, __fadd_rn(m, __fadd_rn(fabsf(I2F(T)), fabsf(I2F(M)))));
  f.ok = f.base <= 3.0e38f;  // false for NaN
  f.int_nw = a.int_nw != 0;
  return f;
}

// Upper and lower end of a candidate's Y (+inf, -inf when unknown).
template <typename V>
__device__ __forceinline__ void FilterEnds(const VertexFilter& f, V S, V M, float Kf, float* hi, float* lo) {
  const float R = __fmul_rn(f.r32, __fmul_rn(f.k32, Kf));
  const float aR = fabsf(R);
  const float Y = __fsub_rn(I2F(static_cast<V>(S - M)), R);
  const float e = __fadd_rn(__fmul_rn(3.814697265625e-06f /* 2^-18 */, __fadd_rn(aR, fabsf(Y))), f.base);
  const bool sane = f.ok && aR <= 1.2676506002282294e30f /* 2^100 */ &&
                    (aR >= 7.888609052210118e-31f /* 2^-100 */ || aR == 0.0f);
  *hi = sane ? __fadd_rn(Y, e) : CUDART_INF_F;
  *lo = sane ? __fsub_rn(Y, e) : -CUDART_INF_F;
}

// Whether two clusters with equal FP32 weights have equal weights: integers
// below 2^24 are exact in FP32, others are compared in FP64.
template <class L>
__device__ __forceinline__ bool SameK(const BMArgs& a, const VertexFilter& f, float Kf, uint32_t i, uint32_t j) {
  return (f.int_nw && fabsf(Kf) < kTwo24) || L::K(a.K + i) == L::K(a.K + j);
}

// ---------------------------------------------------------------------------
// Scanned vertices waiting for their decision, one per lane.
// ---------------------------------------------------------------------------
template <typename V>
struct Pending {
  uint32_t v = kNone;   // kNone: no vertex in this lane
  uint32_t id = kNone;  // leading class: lowest id (kNone: no candidate) ...
  V T = 0, S = 0;       // together-sum; the leading class's sum
  bool single = false;  // every contender is of the leading class
  uint32_t n = 0;       // lanes in use (warp-uniform)
};

// The decision from the exact values of the leading class (S, id) and of the
// new cluster, each lane for itself.  (Not inlined, as every exact function.)
template <typename V, class L>
__device__ __noinline__ bool DecideClass(const BMArgs& a, uint32_t v, uint32_t id, V T, V S, uint32_t stamp) {
  const VertexCtx x = LoadVertexAs<L>(a, v);
  const double change = ChangeOf(a, x, UnitsToDouble<V>(a, T));
  double val = -CUDART_INF;
  if (id != kNone) val = ValOf(a, x, change, UnitsToDouble<V>(a, S), L::K(a.K + id));
  return Decide<false>(a, x, val, id, change, stamp);
}

// The decision of the calling lane's vertex v (kNone: none) from its scan; the
// certified ones are applied.  Not inlined: it runs once per 32 vertices, and
// its bounds would otherwise hold registers in the scan loops.
struct LaneDecision {
  uint32_t cmove;   // certified move (kNone: none)
  int cres;
  bool append;      // to be appended to the movers list
  bool redo;        // several classes, or replayed: decide from exact values
};
template <typename V, class L>
__device__ __noinline__ LaneDecision DecideLane(const BMArgs& a, uint32_t stamp, uint32_t v, uint32_t id, V T, V S,
                                                bool single, bool replay) {
  LaneDecision d{kNone, kUncertain, false, false};
  if (v == kNone) return d;
  VertexCtx x{};
  x.v = v;
  x.c = L::C(a.C + v);
  const float r32 = Res32Of(a, v), k32 = a.kf[v];
  if (single) {
    const ChangeApproxT<V> ca = ApproxChange<V>(r32, a.int_nw != 0, k32, a.Kf[x.c], T);
    const float KfA = id != kNone ? a.Kf[id] : 0.f;
    uint32_t target = kNone;
    d.cres = CertifyDecision<V>(ca, r32, k32, id != kNone, S, KfA, id, a.n, &target);
    if (d.cres != kUncertain) d.cmove = CertifiedMove(a, x, target, d.cres == kCertMove);
  }
  d.redo = replay || !single;
  if (d.redo) return d;
  d.append = d.cres == kUncertain ? DecideClass<V, L>(a, v, id, T, S, stamp) : ApplyCertified(a, x, d.cmove, stamp);
  return d;
}

// Decides the pending vertices and empties the record (every lane of the warp
// calls).  exact(v, cres, cmove): the whole warp decides v from exact values
// and returns (lane 0) whether it must be appended to the movers list.
// Replay decides every vertex exactly and checks the certified decision.
template <typename V, class L, class F>
__device__ __forceinline__ void DecidePending(const BMArgs& a, const RoundView& rv, Pending<V>& p, bool replay,
                                              WarpMoverBuffer& mb, uint32_t* movers, F exact) {
  if (p.n == 0) return;
  const uint32_t pv = LaneId() < p.n ? p.v : kNone;
  const LaneDecision d = DecideLane<V, L>(a, rv.stamp, pv, p.id, p.T, p.S, p.single, replay);
  mb.Add(movers, a.movers, d.append, pv);
  for (unsigned m = __ballot_sync(kFull, d.redo); m; m &= m - 1) {
    const int j = __ffs(m) - 1;
    const uint32_t v = __shfl_sync(kFull, pv, j);
    const int cr = __shfl_sync(kFull, d.cres, j);
    const uint32_t cm = __shfl_sync(kFull, d.cmove, j);
    const bool app = exact(v, cr, cm);
    mb.Add(movers, a.movers, app, v);
  }
  p.n = 0;
}

// The warp's best (value, id) and its decision; in replay also the check of
// the certified decision.  Returns (lane 0) whether the vertex must be
// appended to the movers list.
__device__ __forceinline__ bool DecideExact(const BMArgs& a, const RoundView& rv, const VertexCtx& x, double best,
                                            uint32_t bid, double change, int cres, uint32_t cmove) {
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
  if (LaneId() == 0) {
    append = Decide<false>(a, x, best, bid, change, rv.stamp);
    if (cres != kUncertain && a.out_moves && a.out_moves[x.v] != cmove) atomicExch(&a.ctr->error, kErrCertMismatch);
  }
  return append;
}

// ---------------------------------------------------------------------------
// Lane groups of G lanes, one vertex (degree <= G) per group.
// ---------------------------------------------------------------------------
// A vertex of degree <= 32 from exact FP64 values, by the warp.  A separate
// non-inlined function (as the other exact ones), so that the compiler cannot
// hoist its FP64 arithmetic onto the certified path: an FP64 warp instruction
// costs ~19 SM cycles on this GPU.
template <typename V, class L>
__device__ __noinline__ bool GroupExact(const BMArgs& a, const RoundView& rv, uint32_t v, int cres, uint32_t cmove) {
  const unsigned lane = LaneId();
  const VertexCtx x = LoadVertexAs<L>(a, v);
  const bool has = lane < x.d;
  const uint32_t u = has ? a.nbr[x.b + lane] : v;
  const bool cand = u != v;
  const V xi = cand ? EntryUnits<V, true>(a, a.w ? a.w[x.b + lane] : 1.0f) : V(0);
  const uint32_t cu = cand ? L::C(a.C + u) : kNone;
  const unsigned peers = __match_any_sync(kFull, cand ? cu : LaneSentinel(lane));
  V S = 0;
  for (unsigned mm = peers; mm; mm &= mm - 1) S += __shfl_sync(peers, xi, __ffs(mm) - 1);
  const bool leader = cand && int(lane) == __ffs(peers) - 1;
  const V T = WarpAddV<V>(cand && cu == x.c ? xi : V(0));
  const double change = ChangeOf(a, x, UnitsToDouble<V>(a, T));
  double val = -CUDART_INF;
  if (leader) val = ValOf(a, x, change, UnitsToDouble<V>(a, S), L::K(a.K + cu));
  return DecideExact(a, rv, x, val, leader ? cu : kNone, change, cres, cmove);
}

// A lane's part of a group vertex, loaded ahead of its turn: first the row's
// bounds, cluster and frontier mark, then the lane's entry.
struct GroupRow {
  uint32_t v = 0, d = 0, c = 0, u = 0;
  uint64_t b = 0;
  float w = 0.f;
  bool in = false;
};
template <class L>
__device__ __forceinline__ void GroupHead(const BMArgs& a, const RoundView& rv, bool in, uint32_t v, GroupRow& r) {
  r.v = v;
  r.d = 0;
  r.in = in && InFront(a, rv, v);
  if (in) {
    r.b = a.off[v];
    r.d = uint32_t(a.off[v + 1] - r.b);
    r.c = L::C(a.C + v);
  }
}
template <int G>
__device__ __forceinline__ void GroupEntry(const BMArgs& a, GroupRow& r) {
  const unsigned gl = LaneId() % G;
  r.u = r.v;
  if (r.in && gl < r.d) {
    r.u = a.nbr[r.b + gl];
    r.w = a.w ? a.w[r.b + gl] : 1.0f;
  }
}

// Scans the groups' vertices r into p, which must have room for the warp's
// 32 / G vertices.  stage: 32 values of the calling warp.  ahead() is called
// while the scan waits for no load of its own: it loads the next row.  V: int
// when every sum of a row fits in 32 bits, else long long.
template <int G, typename V, class L, class F>
__device__ __forceinline__ void GroupScan(const BMArgs& a, const GroupRow& r, V* stage, Pending<V>& p,
                                          uint32_t& fam_e, uint32_t& fam_v, F ahead) {
  constexpr unsigned kVpw = 32 / G;
  const unsigned lane = LaneId();
  const unsigned g = lane / G, gl = lane % G;
  const unsigned gmask = G == 32 ? kFull : (((1u << G) - 1u) << (g * G));
  const uint32_t vid = r.v, c = r.c;
  const bool in = r.in;
  if (__ballot_sync(kFull, in) == 0) {  // no frontier vertex in this warp
    ahead();
    return;
  }
  if (in && gl == 0) {
    fam_e += r.d;
    fam_v += 1;
  }
  const bool cand = r.u != vid;
  const uint32_t cu = cand ? L::C(a.C + r.u) : kNone;
  ahead();
  float Kf = cand ? a.Kf[cu] : 0.f;  // (every entry's: the load overlaps the grouping)
  const unsigned peers = __match_any_sync(kFull, cand ? cu : LaneSentinel(lane)) & gmask;
  const bool leader = cand && int(lane) == __ffs(peers) - 1;
  const V xi = cand ? EntryUnits<V, true>(a, r.w) : V(0);
  const V S = GroupSumInt<V>(peers, xi, a.w == nullptr, leader, stage);
  const unsigned tmask = __ballot_sync(kFull, leader && cu == c) & gmask;
  const V Tsh = __shfl_sync(kFull, S, tmask ? __ffs(tmask) - 1 : int(lane));
  const V T = tmask ? Tsh : V(0);
  V M = leader ? S : LowestV<V>();
  if constexpr (G == 32) {
    M = WarpMaxV<V>(M);
  } else {
#pragma unroll
    for (int o = G / 2; o >= 1; o >>= 1) M = max(M, __shfl_xor_sync(kFull, M, o));
  }
  float hi = -CUDART_INF_F, U = -CUDART_INF_F;
  VertexFilter f{};
  if (leader) {
    f = FilterFor<V>(a, vid, c, T, M);
    FilterEnds<V>(f, S, M, Kf, &hi, &U);
  }
  if constexpr (G == 32) {
    U = WarpMaxFinite(U);
  } else {
#pragma unroll
    for (int o = G / 2; o >= 1; o >>= 1) U = fmaxf(U, __shfl_xor_sync(kFull, U, o));
  }
  const bool cont = leader && hi >= U;
  const unsigned m = __ballot_sync(kFull, cont) & gmask;
  // The group's representative contender; with several, all must be of its
  // (S, K) class and the lowest id leads.
  const int j = m ? __ffs(m) - 1 : int(lane);
  V lS = __shfl_sync(kFull, S, j);
  uint32_t id = __shfl_sync(kFull, cu, j);
  if (!m) id = kNone;
  bool single = true;
  if (__ballot_sync(kFull, (m & (m - 1)) != 0)) {
    const float lK = __shfl_sync(kFull, Kf, j);
    const bool diff = cont && (S != lS || !(Kf == lK) || !SameK<L>(a, f, Kf, cu, id));
    single = (__ballot_sync(kFull, diff) & gmask) == 0;
    uint32_t low = cont ? cu : kNone;
    if constexpr (G == 32) {
      low = __reduce_min_sync(kFull, low);
    } else {
#pragma unroll
      for (int o = G / 2; o >= 1; o >>= 1) low = min(low, __shfl_xor_sync(kFull, low, o));
    }
    id = low;
  }
  // Lane p.n + i takes group i's result.
  const unsigned slot = lane - p.n;
  const int src = int((slot % kVpw) * G);
  const uint32_t sv = __shfl_sync(kFull, in ? vid : kNone, src);
  const uint32_t sid = __shfl_sync(kFull, id, src);
  const V sT = __shfl_sync(kFull, T, src);
  const V sS = __shfl_sync(kFull, lS, src);
  const unsigned sing = __ballot_sync(kFull, single);
  if (slot < kVpw) {
    p.v = sv;
    p.id = sid;
    p.T = sT;
    p.S = sS;
    p.single = (sing >> src) & 1u;
  }
  p.n += kVpw;
}

// ---------------------------------------------------------------------------
// One warp or one team of warps per vertex, decided at once.  (Deferring these
// decisions as the lane groups do, with one pass over the candidates, measured
// slower: RMAT-22's warps 33 -> 53 ms.  Their time is the table's and the
// gathers' latency, and the pending record and the lanes' running classes cost
// registers, so warps in flight.)
// ---------------------------------------------------------------------------
// Exact FP64 fallback.  Returns (lane 0) whether the vertex must be appended
// to the movers list; in replay mode it also runs the self-check.
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
  if (replay || !single) {
    append = WarpExact<HC, V>(a, x, T, keys, vals, used, nused, replay, cres, cmove, rv.stamp);
  } else if (lane == 0) {
    append = cres == kUncertain ? DecideClass<V, L>(a, x.v, lead.id, T, lead.S, rv.stamp)
                                : ApplyCertified(a, x, cmove, rv.stamp);
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
  uint32_t exact;  // the vertex goes to TeamExact, with:
  int cres;
  uint32_t cmove;
  double change;
  double bv[TW];
  uint32_t bi[TW];
};

// WarpExact by a whole team: FP64 values of the contenders on the used list,
// cleared as they are read.  (One warp over the 12,288 slots that a hub can
// use took longer than the rest of its CTA's work.)
template <typename V, int TW>
__device__ __noinline__ bool TeamExact(const BMArgs& a, const VertexCtx& x, V* vals, uint32_t* keys,
                                       const uint16_t* used, uint32_t nused, CtaShared<V, TW>& sh, unsigned tid,
                                       unsigned bar, bool replay, uint32_t stamp) {
  const double change = sh.change;
  double best = -CUDART_INF;
  uint32_t bid = kNone;
  for (uint32_t i = tid; i < nused; i += TW * 32) {
    const uint32_t slot = used[i];
    if (slot == 0xFFFFu) continue;
    const uint32_t key = keys[slot];
    const double val = ValOf(a, x, change, UnitsToDouble<V>(a, vals[slot]), a.K[key]);
    keys[slot] = kNone;
    vals[slot] = 0;
    if (Better(val, key, best, bid)) {
      best = val;
      bid = key;
    }
  }
  if (__any_sync(kFull, bid != kNone)) {
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
      const double ov = __shfl_xor_sync(kFull, best, o);
      const uint32_t oid = __shfl_xor_sync(kFull, bid, o);
      if (Better(ov, oid, best, bid)) {
        best = ov;
        bid = oid;
      }
    }
  }
  if ((tid & 31) == 0) {
    sh.bv[tid >> 5] = best;
    sh.bi[tid >> 5] = bid;
  }
  TeamSync<TW * 32>(bar);
  bool append = false;
  if (tid == 0) {
    for (int w = 1; w < TW; ++w)
      if (Better(sh.bv[w], sh.bi[w], best, bid)) {
        best = sh.bv[w];
        bid = sh.bi[w];
      }
    append = Decide<false>(a, x, best, bid, change, stamp);
    if (replay && sh.cres != kUncertain && a.out_moves && a.out_moves[x.v] != sh.cmove)
      atomicExch(&a.ctr->error, kErrCertMismatch);
  }
  return append;
}

// A team of TW warps (its thread index tid) on one vertex x of degree below
// HC (the table must not fill: up to HC / 2 for the teams and small hubs, 3/4 HC
// for the hubs of one partition), with the team's table (clean before and after,
// as sh.nused), a `used` list of at least degree entries, and its hardware
// barrier.  Returns (on thread 0) whether the vertex must be
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
    if (lane == 0) sh.exact = 0;
    if (TW > kCtaWarps && nused == 0) {
      // A hub whose entries are all self-loops: the reduce identity (0, 0.0).
      if (lane == 0) append = Decide<false>(a, x, 0.0, 0, ChangeOf(a, x, 0.0), rv.stamp);
    } else if (replay || !single) {
      if (lane == 0) {
        sh.exact = 1;
        sh.cres = cres;
        sh.cmove = cmove;
        sh.change = ChangeOf(a, x, UnitsToDouble<V>(a, T));
      }
    } else if (lane == 0) {
      append = cres == kUncertain ? DecideClass<V, L>(a, x.v, top.id, T, top.S, rv.stamp)
                                  : ApplyCertified(a, x, cmove, rv.stamp);
    }
  }
  TeamSync<BT>(bar);
  if (sh.exact) {
    append = TeamExact<V, TW>(a, x, vals, keys, used, nused, sh, tid, bar, replay, rv.stamp);
  } else {
    for (uint32_t i = tid; i < nused; i += BT) {
      const uint32_t slot = used[i];
      if (slot != 0xFFFFu) {
        keys[slot] = kNone;
        vals[slot] = 0;
      }
    }
  }
  if (tid == 0) sh.nused = 0;
  TeamSync<BT>(bar);
  return append;
}

}  // namespace
}  // namespace pcc
