// hubeval.cuh -- a hub CTA's row scan, reductions and table evaluation,
// shared by the hub kernels (hubs.cu) and the kernel that runs a whole level's
// rounds (roundloop.cu).  The scheme is in hubs.cuh.
#pragma once

#include <type_traits>

#include "certify.cuh"
#include "hubs.cuh"
#include "moves.cuh"

namespace pcc {
namespace {

constexpr int kHubUnroll = 4;              // entries per thread in flight
constexpr uint32_t kHubMaxSub = 1u << 12;  // sub-partitions before giving up
constexpr uint32_t kMaxCont = 256;         // contender list per CTA
constexpr int kEvalBatch = 4;              // table slots per thread in flight (EvalTable)

// MurmurHash3's 32-bit finalizer (a bijection; every output bit depends on
// every input bit).  The product with the capacity's high half picks the
// slot, bits 8..19 the sub-partition, the top bits (again through a
// product) the partition.
__device__ __forceinline__ uint32_t Mix32(uint32_t x) {
  x ^= x >> 16;
  x *= 0x85EBCA6Bu;
  x ^= x >> 13;
  x *= 0xC2B2AE35u;
  x ^= x >> 16;
  return x;
}

__device__ __forceinline__ uint32_t SlotHash(uint32_t cu) {
  // A second mix so that the slot is independent of the partition bits.
  return Mix32(cu ^ 0x9E3779B9u);
}

__device__ __forceinline__ void KeepBest(double& bv, uint32_t& bi, double v, uint32_t i) {
  if (i == kNone) return;
  if (bi == kNone || v > bv || (v == bv && i < bi)) {
    bv = v;
    bi = i;
  }
}

// Value types of the tables: int (narrow INT sums), long long (INT sums),
// double (FP64 sums).
template <typename V>
__device__ __forceinline__ V AtomicAddV(V* p, V x) {
  if constexpr (std::is_same<V, int>::value) {
    return atomicAdd(p, x);
  } else if constexpr (std::is_same<V, long long>::value) {
    return static_cast<long long>(atomicAdd(reinterpret_cast<unsigned long long*>(p),
                                            static_cast<unsigned long long>(x)));
  } else {
    return atomicAdd(p, x);
  }
}

// Shared scratch of a hub CTA of BT threads besides its table.  The
// reduction arrays hold one partial per warp; their last element carries a
// result that warp 0 publishes (wide CTAs, HubChangeSmax).
template <int BT>
struct HubShared {
  static constexpr int kW = BT / 32;
  long long red_ll[kW + 1];
  long long red_mx[kW + 1];
  unsigned long long red_k[kW + 1];
  double red_d[kW];
  float red_f[kW + 1];
  uint32_t red_i[kW + 1];
  uint32_t cont_key[kMaxCont];
  long long cont_S[kMaxCont];
  uint32_t ncont;
  uint32_t overflow;
  uint32_t nkeys;
  uint32_t last;  // global path: this CTA evaluated the hub's last slice
  long long together;  // INT mode: the hub's own-cluster sum
  double change;
  float change32;
};

// Block reductions; every thread receives the result.  In wide CTAs (512
// threads and more) warp 0 combines the warps' partials and publishes the
// result in red[BT / 32], so that the other threads read one value instead
// of BT / 32; the combines here (max, integer sum, lexicographic and
// (value, id) selections) give the same result in any order.
template <int BT>
constexpr bool kWideBlock = BT >= 512;

template <int BT>
__device__ __forceinline__ long long BlockMaxLL(long long x, long long* red) {
#pragma unroll
  for (int o = 16; o; o >>= 1) x = max(x, __shfl_xor_sync(kFull, x, o));
  if (LaneId() == 0) red[threadIdx.x >> 5] = x;
  __syncthreads();
  if constexpr (kWideBlock<BT>) {
    if (threadIdx.x < 32) {
      long long r = threadIdx.x < BT / 32 ? red[threadIdx.x] : LLONG_MIN;
#pragma unroll
      for (int o = 16; o; o >>= 1) r = max(r, __shfl_xor_sync(kFull, r, o));
      if (threadIdx.x == 0) red[BT / 32] = r;
    }
    __syncthreads();
    return red[BT / 32];
  }
  long long r = red[0];
#pragma unroll
  for (int w = 1; w < BT / 32; ++w) r = max(r, red[w]);
  __syncthreads();
  return r;
}

template <int BT>
__device__ __forceinline__ float BlockMaxF(float x, float* red) {
#pragma unroll
  for (int o = 16; o; o >>= 1) x = fmaxf(x, __shfl_xor_sync(kFull, x, o));
  if (LaneId() == 0) red[threadIdx.x >> 5] = x;
  __syncthreads();
  if constexpr (kWideBlock<BT>) {
    if (threadIdx.x < 32) {
      float r = threadIdx.x < BT / 32 ? red[threadIdx.x] : -CUDART_INF_F;
#pragma unroll
      for (int o = 16; o; o >>= 1) r = fmaxf(r, __shfl_xor_sync(kFull, r, o));
      if (threadIdx.x == 0) red[BT / 32] = r;
    }
    __syncthreads();
    return red[BT / 32];
  }
  float r = red[0];
#pragma unroll
  for (int w = 1; w < BT / 32; ++w) r = fmaxf(r, red[w]);
  __syncthreads();
  return r;
}

// Deterministic sum: butterfly inside warps, then the warps in order.
template <int BT, class T>
__device__ __forceinline__ T BlockSum(T x, T* red) {
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    if constexpr (std::is_floating_point<T>::value) {
      x = Dadd(x, __shfl_xor_sync(kFull, x, o));
    } else {
      x += __shfl_xor_sync(kFull, x, o);
    }
  }
  if (LaneId() == 0) red[threadIdx.x >> 5] = x;
  __syncthreads();
  if constexpr (kWideBlock<BT> && std::is_integral<T>::value) {
    if (threadIdx.x < 32) {
      T r = threadIdx.x < BT / 32 ? red[threadIdx.x] : T(0);
#pragma unroll
      for (int o = 16; o; o >>= 1) r += __shfl_xor_sync(kFull, r, o);
      if (threadIdx.x == 0) red[BT / 32] = r;
    }
    __syncthreads();
    return red[BT / 32];
  }
  T r = red[0];
#pragma unroll
  for (int w = 1; w < BT / 32; ++w) {
    if constexpr (std::is_floating_point<T>::value) {
      r = Dadd(r, red[w]);
    } else {
      r += red[w];
    }
  }
  __syncthreads();
  return r;
}

// Argmax over (value desc, id asc) with integer compares: the values are
// mapped to order-preserving 64-bit images (no FP64 instruction; the values
// here are never -0, the only case where the image order and IEEE equality
// differ).
__device__ __forceinline__ unsigned long long ValBits(double d) {
  const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(d));
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double BitsVal(unsigned long long k) {
  const unsigned long long b = (k >> 63) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k;
  return __longlong_as_double(static_cast<long long>(b));
}
__device__ __forceinline__ void KeepBits(unsigned long long& bo, uint32_t& bi, unsigned long long o, uint32_t i) {
  if (i == kNone) return;
  if (bi == kNone || o > bo || (o == bo && i < bi)) {
    bo = o;
    bi = i;
  }
}

template <int BT>
__device__ __forceinline__ void BlockArgmax(double& v, uint32_t& id, unsigned long long* redv, uint32_t* redi) {
  unsigned long long o = ValBits(v);
#pragma unroll
  for (int off = 16; off; off >>= 1) {
    const unsigned long long oo = __shfl_xor_sync(kFull, o, off);
    const uint32_t oi = __shfl_xor_sync(kFull, id, off);
    KeepBits(o, id, oo, oi);
  }
  if (LaneId() == 0) {
    redv[threadIdx.x >> 5] = o;
    redi[threadIdx.x >> 5] = id;
  }
  __syncthreads();
  if constexpr (kWideBlock<BT>) {
    if (threadIdx.x < 32) {
      const bool in = threadIdx.x < BT / 32;
      unsigned long long wo = redv[in ? threadIdx.x : 0];
      uint32_t wi = in ? redi[threadIdx.x] : kNone;
#pragma unroll
      for (int off = 16; off; off >>= 1) {
        const unsigned long long oo = __shfl_xor_sync(kFull, wo, off);
        const uint32_t oi = __shfl_xor_sync(kFull, wi, off);
        KeepBits(wo, wi, oo, oi);
      }
      if (threadIdx.x == 0) {
        redv[BT / 32] = wo;
        redi[BT / 32] = wi;
      }
    }
    __syncthreads();
    v = BitsVal(redv[BT / 32]);
    id = redi[BT / 32];
    return;
  }
  unsigned long long ro = redv[0];
  uint32_t ri = redi[0];
#pragma unroll
  for (int w = 1; w < BT / 32; ++w) KeepBits(ro, ri, redv[w], redi[w]);
  __syncthreads();
  v = BitsVal(ro);
  id = ri;
}

template <int BT, typename I>
__device__ __forceinline__ LexKeyT<I> BlockLex(LexKeyT<I> x, long long* rs, unsigned long long* rk, uint32_t* ri) {
  LexGroupReduce<32, I>(x);
  if (LaneId() == 0) {
    rs[threadIdx.x >> 5] = x.S;
    rk[threadIdx.x >> 5] = x.K;
    ri[threadIdx.x >> 5] = x.id;
  }
  __syncthreads();
  if constexpr (kWideBlock<BT>) {
    if (threadIdx.x < 32) {
      LexKeyT<I> w;
      if (threadIdx.x < BT / 32) w.Keep(static_cast<I>(rs[threadIdx.x]), rk[threadIdx.x], ri[threadIdx.x]);
      LexGroupReduce<32, I>(w);
      if (threadIdx.x == 0) {
        rs[BT / 32] = w.S;
        rk[BT / 32] = w.K;
        ri[BT / 32] = w.id;
      }
    }
    __syncthreads();
    LexKeyT<I> r;
    r.Keep(static_cast<I>(rs[BT / 32]), rk[BT / 32], ri[BT / 32]);
    return r;
  }
  LexKeyT<I> r;
#pragma unroll
  for (int w = 0; w < BT / 32; ++w) r.Keep(static_cast<I>(rs[w]), rk[w], ri[w]);
  __syncthreads();
  return r;
}

// Block leader of `lead` and the class test over `tail` (the two BlockLex
// calls and the (S, K) comparison) with 32-bit sums: warp leaders by REDUX,
// the warps' leaders combined by every thread, the test by one barrier with
// a predicate.
template <int BT>
__device__ __forceinline__ bool BlockLexLeadInt(LexKeyT<int>& lead, const LexKeyT<int>& tail, long long* rs,
                                                unsigned long long* rk, uint32_t* ri) {
  LexWarpLeaderInt(lead);
  if (LaneId() == 0) {
    rs[threadIdx.x >> 5] = lead.S;
    rk[threadIdx.x >> 5] = lead.K;
    ri[threadIdx.x >> 5] = lead.id;
  }
  __syncthreads();
  LexKeyT<int> r;
  if constexpr (kWideBlock<BT>) {
    if (threadIdx.x < 32) {
      LexKeyT<int> w;
      if (threadIdx.x < BT / 32) w.Keep(static_cast<int>(rs[threadIdx.x]), rk[threadIdx.x], ri[threadIdx.x]);
      LexWarpLeaderInt(w);
      if (threadIdx.x == 0) {
        rs[BT / 32] = w.S;
        rk[BT / 32] = w.K;
        ri[BT / 32] = w.id;
      }
    }
    __syncthreads();
    r.Keep(static_cast<int>(rs[BT / 32]), rk[BT / 32], ri[BT / 32]);
  } else {
#pragma unroll
    for (int w = 0; w < BT / 32; ++w) r.Keep(static_cast<int>(rs[w]), rk[w], ri[w]);
  }
  lead = r;
  const bool diff = r.id != kNone && tail.id != kNone && (-tail.S != r.S || ~tail.K != r.K);
  return !__syncthreads_or(diff);  // also orders the reads of rs/rk/ri before their next use
}

// Finds or inserts `key` in a table of `cap` slots (any capacity), probing
// linearly from the slot the hash picks; kNone when the table is full.
__device__ __forceinline__ uint32_t HubInsert(uint32_t* keys, uint32_t cap, uint32_t hsh, uint32_t key,
                                              bool* ins) {
  uint32_t s = __umulhi(hsh, cap);
  *ins = false;
  for (uint32_t pr = 0; pr < cap; ++pr) {
    const uint32_t k = *reinterpret_cast<volatile uint32_t*>(keys + s);
    if (k == key) return s;
    if (k == kNone) {
      const uint32_t old = atomicCAS(keys + s, kNone, key);
      if (old == kNone) {
        *ins = true;
        return s;
      }
      if (old == key) return s;
    }
    s = s + 1 == cap ? 0 : s + 1;
  }
  return kNone;
}

// Entry contribution w - offset: integer in INT mode, the reference hub
// path's float-rounded value in FP64 mode.
template <bool kInt, typename V>
__device__ __forceinline__ void EntryWeight(const BMArgs& a, float wt, V* xi, double* xd) {
  if constexpr (kInt) {
    *xi = EntryUnits<V, true>(a, wt);
  } else {
    *xd = static_cast<double>(static_cast<float>(Dsub(static_cast<double>(wt), a.offset)));
  }
}

// Warp-aggregated FP64 sum of the entry weights of each match group, in lane
// order (for the group's leader).
template <int BT>
__device__ __forceinline__ double GroupWeights(unsigned peers, bool leader, double xd) {
  __shared__ double stage_d[BT / 32][32];
  const unsigned warp = threadIdx.x >> 5, lane = LaneId();
  stage_d[warp][lane] = xd;
  __syncwarp();
  double acc = 0.0;
  if (leader) {
    unsigned mm = peers;
    while (mm) {
      acc = Dadd(acc, stage_d[warp][__ffs(mm) - 1]);
      mm &= mm - 1;
    }
  }
  __syncwarp();
  return acc;
}

// Evaluates the CTA's table: returns (to every thread) the best (exact FP64
// value, id) of its keys and clears the table.  INT sync mode: FP32
// pre-filter, then FP64 only for the survivors outside the leading (S, K)
// class, whose members share one FP64 value (evaluated once).
template <int BT, bool kInt, bool kAsync, typename V>
__device__ void EvalTable(const BMArgs& a, const VertexCtx& x, float k32, double change, long long smax_ll,
                          uint32_t* skeys, V* svals, uint32_t cap, HubShared<BT>& sh, double* out_v,
                          uint32_t* out_id) {
  // Integer type of the sums: int for narrow tables (32-bit conversions).
  using I = typename std::conditional<std::is_same<V, int>::value, int, long long>::type;
  const unsigned tid = threadIdx.x;
  constexpr bool kFilter = kInt && !kAsync;
  double lv = 0.0;
  uint32_t lid = kNone;
  // Slots are read kEvalBatch at a time per thread, so that the gathers of
  // their cluster weights are in flight together.
  constexpr int kB = kEvalBatch;
  if (kFilter) {
    const I smax = static_cast<I>(smax_ll);
    const float c32 = __fmul_rn(sh.change32, a.wscale);  // in the units of the sums
    const float r32 = Res32Of(a, x.v);
    float U = -CUDART_INF_F;
    // The two largest upper ends (Y + e; +inf for a candidate outside the
    // error model) among this thread's slots, and the slot of the largest:
    // when the second is below the block's U, no other slot of the thread
    // can be a contender and the second pass need not re-evaluate them.
    float hi1 = -CUDART_INF_F, hi2 = -CUDART_INF_F;
    uint32_t slot1 = kNone;
    for (uint32_t s0 = tid; s0 < cap; s0 += BT * kB) {
      uint32_t kk[kB];
      I ss[kB];
      float kf[kB];
#pragma unroll
      for (int j = 0; j < kB; ++j) {
        const uint32_t s = s0 + j * BT;
        kk[j] = s < cap ? skeys[s] : kNone;
        ss[j] = s < cap ? static_cast<I>(svals[s]) : I(0);
      }
#pragma unroll
      for (int j = 0; j < kB; ++j) kf[j] = kk[j] != kNone ? a.Kf[kk[j]] : 0.f;
#pragma unroll
      for (int j = 0; j < kB; ++j) {
        if (kk[j] == kNone) continue;
        const FilterVal f = FilterOf<I>(r32, k32, kf[j], ss[j], smax, c32);
        if (f.sane) U = fmaxf(U, __fsub_rn(f.Y, f.e));
        KeepTop2(hi1, hi2, slot1, f.sane ? __fadd_rn(f.Y, f.e) : CUDART_INF_F, s0 + j * BT);
      }
    }
    if (tid == 0) sh.ncont = 0;
    U = BlockMaxF<BT>(U, sh.red_f);
    LexKeyT<I> lead, tail;
    // The contenders are the slots with hi >= U (every slot when U = -inf).
    const bool rescan = !(hi2 < U);
    if (!rescan) {
      // At most slot1 is a contender; the thread's other slots are cleared.
      if (slot1 != kNone && !(hi1 < U)) {
        const uint32_t key = skeys[slot1];
        const I S = static_cast<I>(svals[slot1]);
        const double KD = a.K[key];
        const unsigned long long ko = KOrder(KD);
        lead.Keep(S, ko, key);
        tail.Keep(-S, ~ko, key);
        const uint32_t pos = atomicAdd(&sh.ncont, 1u);
        if (pos < kMaxCont) {
          sh.cont_key[pos] = key;
          sh.cont_S[pos] = S;
        } else {
          KeepBest(lv, lid, ValOf(a, x, change, UnitsToDouble<I>(a, S), KD), key);  // list full: now
        }
      }
      for (uint32_t s = tid; s < cap; s += BT) {
        if (skeys[s] != kNone) {
          skeys[s] = kNone;
          svals[s] = V(0);
        }
      }
    }
    for (uint32_t s0 = rescan ? tid : cap; s0 < cap; s0 += BT * kB) {
      uint32_t kk[kB];
      I ss[kB];
      float kf[kB];
#pragma unroll
      for (int j = 0; j < kB; ++j) {
        const uint32_t s = s0 + j * BT;
        kk[j] = kNone;
        ss[j] = I(0);
        if (s < cap) {
          kk[j] = skeys[s];
          if (kk[j] != kNone) {
            ss[j] = static_cast<I>(svals[s]);
            skeys[s] = kNone;
            svals[s] = V(0);
          }
        }
      }
#pragma unroll
      for (int j = 0; j < kB; ++j) kf[j] = kk[j] != kNone ? a.Kf[kk[j]] : 0.f;
#pragma unroll
      for (int j = 0; j < kB; ++j) {
        const uint32_t key = kk[j];
        if (key == kNone) continue;
        const I S = ss[j];
        const FilterVal f = FilterOf<I>(r32, k32, kf[j], S, smax, c32);
        if (f.sane && __fadd_rn(f.Y, f.e) < U) continue;
        const double KD = a.K[key];
        const unsigned long long ko = KOrder(KD);
        lead.Keep(S, ko, key);
        tail.Keep(-S, ~ko, key);
        const uint32_t pos = atomicAdd(&sh.ncont, 1u);
        if (pos < kMaxCont) {
          sh.cont_key[pos] = key;
          sh.cont_S[pos] = S;
        } else {
          KeepBest(lv, lid, ValOf(a, x, change, UnitsToDouble<I>(a, S), KD), key);  // list full: now
        }
      }
    }
    bool single;
    if constexpr (std::is_same<I, int>::value) {
      single = BlockLexLeadInt<BT>(lead, tail, sh.red_ll, sh.red_k, sh.red_i);
    } else {
      lead = BlockLex<BT, I>(lead, sh.red_ll, sh.red_k, sh.red_i);
      tail = BlockLex<BT, I>(tail, sh.red_ll, sh.red_k, sh.red_i);
      single = lead.id == kNone || (-tail.S == lead.S && ~tail.K == lead.K);
    }
    const uint32_t nc = min(sh.ncont, kMaxCont);
    if (!single) {
      for (uint32_t i = tid; i < nc; i += BT) {
        const uint32_t key = sh.cont_key[i];
        const I S = static_cast<I>(sh.cont_S[i]);
        const double KD = a.K[key];
        if (S == lead.S && KOrder(KD) == lead.K) continue;  // the leading class
        KeepBest(lv, lid, ValOf(a, x, change, UnitsToDouble<I>(a, S), KD), key);
      }
    }
    if (tid == 0 && lead.id != kNone)
      KeepBest(lv, lid, ValOf(a, x, change, UnitsToDouble<I>(a, lead.S), a.K[lead.id]), lead.id);
  } else {
    for (uint32_t s0 = tid; s0 < cap; s0 += BT * kB) {
      uint32_t kk[kB];
      V sv[kB];
      double kd[kB];
#pragma unroll
      for (int j = 0; j < kB; ++j) {
        const uint32_t s = s0 + j * BT;
        kk[j] = kNone;
        sv[j] = V(0);
        if (s < cap) {
          kk[j] = skeys[s];
          if (kk[j] != kNone) {
            sv[j] = svals[s];
            skeys[s] = kNone;
            svals[s] = V(0);
          }
        }
      }
#pragma unroll
      for (int j = 0; j < kB; ++j) kd[j] = kk[j] != kNone ? LdK<kAsync>(a.K + kk[j]) : 0.0;
#pragma unroll
      for (int j = 0; j < kB; ++j)
        if (kk[j] != kNone) KeepBest(lv, lid, ValOf(a, x, change, kInt ? UnitsToDouble<I>(a, static_cast<I>(sv[j])) : static_cast<double>(sv[j]), kd[j]),
                   kk[j]);
    }
  }
  BlockArgmax<BT>(lv, lid, sh.red_k, sh.red_i);
  *out_v = lv;
  *out_id = lid;
}

template <bool kAsync>
__device__ __forceinline__ void HubDecide(const BMArgs& a, const VertexCtx& x, double bv, uint32_t bi,
                                          double change, uint32_t stamp, uint32_t* movers) {
  if (bi == kNone) {  // no entries: the reduce identity (0, 0.0)
    bv = 0.0;
    bi = 0;
  }
  const bool append = Decide<kAsync>(a, x, bv, bi, change, stamp);
  if (!kAsync && append) a.movers[atomicAdd(movers, 1u)] = x.v;
}

// One CTA's scan of a hub row: the entries whose cluster falls in partition
// p / sub-partition q are added into the CTA's table; "together" (the hub's
// own cluster) accumulates when want_T.  Returns the largest running sum seen
// (32-bit sums) through *smax: the pre-filter's shift, which any value near the
// largest sums serves.  64-bit sums leave it and take the together-sum
// instead: an atomic that returns the old sum costs twice the one that does
// not.
template <int BT, bool kInt, bool kAsync, typename V, class L = ConstLoads>
__device__ __forceinline__ void ScanRow(const BMArgs& a, const VertexCtx& x, uint32_t P, uint32_t p, uint32_t Q,
                                        uint32_t q, bool want_T, uint32_t* skeys, V* svals, uint32_t cap,
                                        uint32_t maxkeys, HubShared<BT>& sh, long long* t_int, double* t_dbl,
                                        long long* smax) {
  const unsigned tid = threadIdx.x, lane = LaneId();
  const uint32_t v = x.v;
  for (uint32_t e0 = 0; e0 < x.d; e0 += BT * kHubUnroll) {
    uint32_t uu[kHubUnroll], cc[kHubUnroll];
    float ww[kHubUnroll];
#pragma unroll
    for (int k = 0; k < kHubUnroll; ++k) {
      const uint32_t e = e0 + k * BT + tid;
      uu[k] = v;
      ww[k] = 0.f;
      if (e < x.d) {
        uu[k] = a.nbr[x.b + e];
        ww[k] = a.w ? a.w[x.b + e] : 1.0f;
      }
    }
#pragma unroll
    for (int k = 0; k < kHubUnroll; ++k) cc[k] = uu[k] == v ? kNone : kAsync ? LdC<true>(a.C + uu[k]) : L::C(a.C + uu[k]);
#pragma unroll
    for (int k = 0; k < kHubUnroll; ++k) {
      if (e0 + k * BT >= x.d) break;  // uniform over the CTA
      const bool cand = uu[k] != v;
      const uint32_t cu = cc[k];
      V xi = 0;
      double xd = 0.0;
      if (cand) EntryWeight<kInt, V>(a, ww[k], &xi, &xd);
      if (want_T && cand && cu == x.c) {
        if (kInt)
          *t_int += xi;
        else
          *t_dbl = Dadd(*t_dbl, xd);
      }
      bool mine = cand;
      if (P > 1 || Q > 1) {
        const uint32_t hp = Mix32(cu);
        mine = mine && __umulhi(hp, P) == p && ((hp >> 8) & (Q - 1)) == q;
      }
      // INT mode: every entry adds its own integer weight (exact in any
      // order); FP64 mode: equal clusters of the warp are summed in lane
      // order first, one atomic per cluster.
      unsigned peers = 0;
      bool leader = mine;
      double Sd = 0.0;
      if constexpr (!kInt) {
        peers = __match_any_sync(kFull, mine ? cu : LaneSentinel(lane));
        leader = mine && int(lane) == __ffs(peers) - 1;
        Sd = GroupWeights<BT>(peers, leader, xd);
      }
      if (leader && *reinterpret_cast<volatile uint32_t*>(&sh.overflow) == 0) {
        bool ins;
        const uint32_t slot = HubInsert(skeys, cap, SlotHash(cu), cu, &ins);
        if (slot == kNone) {
          sh.overflow = 1;
        } else {
          if (ins && atomicAdd(&sh.nkeys, 1u) + 1 > maxkeys) sh.overflow = 1;
          if constexpr (std::is_same<V, long long>::value) {
            SharedAdd(svals + slot, xi);
          } else if constexpr (kInt) {
            const V old = AtomicAddV<V>(svals + slot, xi);
            *smax = max(*smax, static_cast<long long>(old) + static_cast<long long>(xi));
          } else {
            AtomicAddV<V>(svals + slot, static_cast<V>(Sd));
          }
        }
      }
    }
  }
}

// The hub's "together" and change, once per item (FP64 by one thread).
template <int BT, bool kInt>
__device__ __forceinline__ double HubChange(const BMArgs& a, const VertexCtx& x, long long t_int, double t_dbl,
                                            HubShared<BT>& sh) {
  double T;
  if constexpr (kInt) {
    const long long t = BlockSum<BT, long long>(t_int, sh.red_ll);
    T = UnitsToDouble<long long>(a, t);
    if (threadIdx.x == 0) sh.together = t;
  } else {
    T = BlockSum<BT, double>(t_dbl, sh.red_d);
  }
  if (threadIdx.x == 0) {
    sh.change = ChangeOf(a, x, T);
    sh.change32 = static_cast<float>(sh.change);
  }
  __syncthreads();
  return sh.change;
}

// HubChange and, in INT mode, the block maximum of the running sums.  Wide
// CTAs take both in one reduction: warp 0 combines the warps' (sum, max)
// partials and its lane 0 computes the change, so that the table scan's end
// costs two barriers.
template <int BT, bool kInt>
__device__ __forceinline__ double HubChangeSmax(const BMArgs& a, const VertexCtx& x, long long t_int, double t_dbl,
                                                long long* smax, HubShared<BT>& sh) {
  if constexpr (!kWideBlock<BT>) {
    __syncthreads();
    const double change = HubChange<BT, kInt>(a, x, t_int, t_dbl, sh);
    if (kInt) *smax = BlockMaxLL<BT>(*smax, sh.red_ll);
    if (kInt && *smax == LLONG_MIN) *smax = sh.together;
    return change;
  } else if constexpr (!kInt) {
    return HubChange<BT, kInt>(a, x, t_int, t_dbl, sh);
  } else {
    constexpr int kW = BT / 32;
    long long t = t_int, m = *smax;
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      t += __shfl_xor_sync(kFull, t, o);
      m = max(m, __shfl_xor_sync(kFull, m, o));
    }
    if (LaneId() == 0) {
      sh.red_ll[threadIdx.x >> 5] = t;
      sh.red_mx[threadIdx.x >> 5] = m;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      long long wt = threadIdx.x < kW ? sh.red_ll[threadIdx.x] : 0;
      long long wm = threadIdx.x < kW ? sh.red_mx[threadIdx.x] : LLONG_MIN;
#pragma unroll
      for (int o = 16; o; o >>= 1) {
        wt += __shfl_xor_sync(kFull, wt, o);
        wm = max(wm, __shfl_xor_sync(kFull, wm, o));
      }
      if (threadIdx.x == 0) {
        sh.change = ChangeOf(a, x, UnitsToDouble<long long>(a, wt));
        sh.change32 = static_cast<float>(sh.change);
        sh.red_mx[kW] = wm == LLONG_MIN ? wt : wm;
      }
    }
    __syncthreads();
    *smax = sh.red_mx[kW];
    return sh.change;
  }
}

}  // namespace
}  // namespace pcc
