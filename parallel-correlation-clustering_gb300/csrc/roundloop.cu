// roundloop.cu -- the best-move rounds of a level (IterateBestMoves,
// parallel-correlation-clusterer.cc:340-365) in one cooperative kernel: best
// moves, MoveNodesToCluster, the FP32 images and the next frontier of every
// round, with grid-wide barriers between the phases.
//
// Why: a round of a small or middle level is microseconds of work per kernel,
// but took 12-33 kernel nodes of a device-side graph loop, 3-4 us each with
// their launch and drain, and a level's degree bins ran as separate kernels
// whose tails and serial chains left most of the GPU idle.  Here a round costs
// its work plus grid barriers of 1-2 us: two when no vertex moves, three when
// some do, three more when clusters are opened, and one more on levels with rows
// above 4096.  Per round, before and after: 576 entries 45 -> 34 us, 4,686
// entries 49 -> 27 us, 1M entries 147 -> 77 us, 5.6M entries with a 147,524-entry
// row 430 -> 270 us.  Every kind of work item goes through one queue, largest
// items first, so a CTA that runs out of one kind goes on with the next:
//   stage 0  CTA items: chunks of the rows above degree 4096 (summed into
//            per-hub tables in HBM), then hubs of degree 1001-4096 (one CTA,
//            table in shared memory)
//   stage 1  teams of four warps: degree 257-1000 (129-1000 with 64-bit sums)
//   stage 2  warps: degree 33-256 (33-128)
//   stage 3  lane groups: degree <= 32
// Rows above degree 4096 are then evaluated slice by slice.
//
// Every wait is a grid barrier of a cooperative launch (all CTAs resident),
// with an iteration limit after which the kernel reports kErrBarrier and
// returns.
#include <algorithm>
#include <cstddef>
#include <cstring>

#include "barrier.h"
#include "certmoves.cuh"
#include "hubeval.cuh"
#include "roundloop.cuh"

namespace pcc {
namespace {

constexpr int kLT = 512;           // threads of a CTA
constexpr int kLW = kLT / 32;      // warps
constexpr int kTeams = kLW / kCtaWarps;
constexpr int kLoopUnroll = 4;
constexpr int kMaskWords = 4;      // ids per thread of the empty-id scan, / 32

struct LoopShared {
  union {
    uint32_t mover_buf[kLW][64];  // best-move stages
    HubShared<kLT> hub;           // table slices, after every buffer's flush
  };
  uint32_t bin_start[kNumBins + 1];
  uint32_t push_start[kNumBins + 1];
  unsigned long long fam_e[kNumFamilies], fam_v[kNumFamilies];
  unsigned long long red64[kLW + 1];
  uint32_t red_a[kLW], red_b[kLW];
  uint32_t item;
  uint32_t team_item[kTeams];
  uint32_t ok;
};

// Grid-wide barrier: waits until `target` arrivals are counted (modulo 2^32).
// Release and acquire at GPU scope: the writes before it are visible after it,
// and the L1 lines read before it are dropped.  False: given up after `polls`
// looks.  The CTA then leaves without arriving again, so no other one passes
// the next barrier: what runs meanwhile reads only what was complete here.
__device__ __forceinline__ bool GridSync(LoopShared& sh, uint32_t* count, uint32_t target, uint32_t polls) {
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t ok = 1;
    if (gridDim.x > 1) {
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
      uint32_t c = 0;
      ok = 0;
      for (uint32_t t = 0; t < polls; ++t) {
        asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(c) : "l"(count) : "memory");
        if (BarrierReached(c, target)) {
          ok = 1;
          break;
        }
      }
    }
    sh.ok = ok;
  }
  __syncthreads();
  return sh.ok != 0;
}

// Sum of x over the block (every thread gets it).
__device__ __forceinline__ uint32_t BlockSum32(uint32_t x, uint32_t* red) {
  x = __reduce_add_sync(kFull, x);
  if (LaneId() == 0) red[threadIdx.x >> 5] = x;
  __syncthreads();
  uint32_t r = 0;
#pragma unroll
  for (int w = 0; w < kLW; ++w) r += red[w];
  __syncthreads();
  return r;
}

// The next frontier: u is stamped; the thread that stamps it first counts it.
struct Pusher {
  uint32_t* next;
  const uint64_t* off;
  uint32_t stamp;
  uint32_t cnt = 0;
  unsigned long long deg = 0;
  __device__ __forceinline__ void Mark(uint32_t u, uint32_t cur) {
    if (cur != stamp && atomicExch(&next[u], stamp) != stamp) {
      cnt += 1;
      deg += off[u + 1] - off[u];
    }
  }
};

template <typename V, bool kConv>
__global__ void __launch_bounds__(kLT, 2) RoundLoopKernel(const __grid_constant__ RoundLoopArgs l) {
  extern __shared__ __align__(16) unsigned char loop_smem[];
  __shared__ LoopShared sh;
  __shared__ CtaShared<V> team_sh[kTeams];
  __shared__ CtaShared<V, kLW> cta_sh;
  const BMArgs& a = l.a;
  const uint32_t slots = l.table_slots;
  uint32_t* keys = reinterpret_cast<uint32_t*>(loop_smem);
  V* vals = reinterpret_cast<V*>(loop_smem + size_t(slots) * 4);
  unsigned char* extra = loop_smem + size_t(slots) * (4 + sizeof(V));  // slots bytes, dirty
  const unsigned tid = threadIdx.x, lane = LaneId(), warp = tid >> 5, team = warp / kCtaWarps;
  const uint32_t G = gridDim.x;
  // This warp's and this team's parts of the tables and of `extra`.
  const uint32_t wslots = slots / kLW, tslots = slots / kTeams;
  uint32_t* wkeys = keys + warp * wslots;
  V* wvals = vals + warp * wslots;
  uint16_t* wused = reinterpret_cast<uint16_t*>(extra + size_t(warp) * wslots);
  uint32_t* tkeys = keys + team * tslots;
  V* tvals = vals + team * tslots;
  uint16_t* tused = reinterpret_cast<uint16_t*>(extra + size_t(team) * tslots);
  V* wstage = reinterpret_cast<V*>(extra + size_t(warp) * wslots);  // 32 values

  for (uint32_t i = tid; i < slots; i += kLT) {
    keys[i] = kNone;
    vals[i] = V(0);
  }
  if (tid <= kNumBins) {
    sh.bin_start[tid] = l.starts[tid];
    sh.push_start[tid] = l.push_starts[tid];
  }
  if (tid < kNumFamilies) sh.fam_e[tid] = sh.fam_v[tid] = 0;
  if (tid < kTeams) team_sh[tid].nused = 0;
  if (tid == 0) cta_sh.nused = 0;
  __syncthreads();

  RoundView rv;
  const RoundState rs = l.st->head.rs;
  rv.stamp = rs.stamp + 1;
  rv.front_val = rs.front_val;
  rv.all = rs.front_all != 0;
  unsigned long long front_edges = rs.front_edges, front_size = rs.front_size, visited = rs.visited;
  const uint32_t n = a.n;
  uint32_t* count = &l.st->barrier;
  uint32_t arrivals = kBarrierStart;
  const bool all_move = l.move_method == PCC_ALL_MOVE;
  WarpMoverBuffer mb{sh.mover_buf[warp]};
  // Degree bins of the teams: 257-1000, with 64-bit sums (two table words
  // more per entry) 129-1000.
  constexpr int kTeamLow = sizeof(V) == 4 ? kBinW512 : kBinW256;
  Pending<V> pend;

  for (uint32_t round = 0; round < l.num_inner; ++round) {
    LoopCounters* ctr = &l.st->ctr[round % 3];
    uint32_t* movers = &ctr->movers;

    // ---- Best moves -------------------------------------------------------
    // Stage 0: CTA items.  The next item is taken while this one runs.
    {
      unsigned long long fe_s = 0, fv_s = 0, fe_b = 0, fv_b = 0;  // thread 0
      const uint32_t items = l.num_chunks + l.num_small;
      uint32_t item = blockIdx.x;
      while (item < items) {
        uint32_t next = 0;
        if (tid == 0) next = G + atomicAdd(&ctr->queue[0], 1u);
        if (item < l.num_chunks) {
          const uint32_t hb = l.chunk_hub[item];
          const uint32_t v = l.big_v[hb];
          if (InFront(a, rv, v)) {  // uniform over the CTA
            const VertexCtx x = LoadVertexAs<LiveLoads>(a, v);
            const uint32_t e_begin = l.chunk_start[item];
            const uint32_t e_end = min(x.d, e_begin + kLoopChunk);
            uint32_t* gk = l.gkeys + l.big_base[hb];
            V* gv = reinterpret_cast<V*>(l.gvals) + l.big_base[hb];
            const uint32_t cap = l.big_cap[hb];
            if (tid == 0 && e_begin == 0) {
              fe_b += x.d;
              fv_b += 1;
            }
            long long t_int = 0;
            uint32_t uu[kLoopUnroll], cc[kLoopUnroll];
            float ww[kLoopUnroll];
#pragma unroll
            for (int k = 0; k < kLoopUnroll; ++k) {
              const uint32_t e = e_begin + k * kLT + tid;
              uu[k] = v;
              ww[k] = 0.f;
              if (e < e_end) {
                uu[k] = a.nbr[x.b + e];
                ww[k] = a.w ? a.w[x.b + e] : 1.0f;
              }
            }
#pragma unroll
            for (int k = 0; k < kLoopUnroll; ++k) cc[k] = uu[k] != v ? a.C[uu[k]] : kNone;
#pragma unroll
            for (int k = 0; k < kLoopUnroll; ++k) {
              if (cc[k] == kNone) continue;
              const V xi = EntryUnits<V, true>(a, ww[k]);
              if (cc[k] == x.c) t_int += xi;
              bool ins;
              const uint32_t slot = HubInsert(gk, cap, SlotHash(cc[k]), cc[k], &ins);
              if (slot == kNone) {
                atomicExch(&a.ctr->error, kErrHashFull);  // cannot happen: 2 * degree + 2 slots
              } else {
                AtomicAddV<V>(gv + slot, xi);
              }
            }
            const long long t = BlockSum<kLT, long long>(t_int, reinterpret_cast<long long*>(sh.red64));
            if (tid == 0 && t)
              atomicAdd(reinterpret_cast<unsigned long long*>(l.gt_int + hb), static_cast<unsigned long long>(t));
          }
        } else {
          const uint32_t v = l.small_v[item - l.num_chunks];
          if (InFront(a, rv, v)) {  // uniform over the CTA
            const VertexCtx x = LoadVertexAs<LiveLoads>(a, v);
            if (tid == 0) {
              fe_s += x.d;
              fv_s += 1;
            }
            const bool append = CtaStep<2 * kHubSmallMax, V, kConv, LiveLoads, kLW>(
                a, rv, x, vals, keys, reinterpret_cast<uint16_t*>(extra), cta_sh, tid, 0, false);
            if (warp == 0) mb.Add(movers, a.movers, append, v);
          }
        }
        if (tid == 0) sh.item = next;
        __syncthreads();
        item = sh.item;
        __syncthreads();
      }
      if (tid == 0) {
        sh.fam_e[kFamHubSmall] += fe_s;
        sh.fam_v[kFamHubSmall] += fv_s;
        sh.fam_e[kFamHubBig] += fe_b;
        sh.fam_v[kFamHubBig] += fv_b;
      }
    }
    unsigned long long fam_e = 0, fam_v = 0;
    // Stage 1: teams.
    {
      const uint32_t first = sh.bin_start[kTeamLow];
      const uint32_t items = sh.bin_start[kBinW1000 + 1] - first;
      const uint32_t* tl = l.list + first;
      uint32_t item = blockIdx.x * kTeams + team;
      const unsigned tt = tid & (kCtaWarps * 32 - 1);
      while (item < items) {
        uint32_t next = 0;
        if (tt == 0) next = G * kTeams + atomicAdd(&ctr->queue[1], 1u);
        // Largest degrees first (the bins are in ascending order).
        const uint32_t v = tl[items - 1 - item];
        if (InFront(a, rv, v)) {  // uniform over the team
          const VertexCtx x = LoadVertexAs<LiveLoads>(a, v);
          if (tt == 0) {
            fam_e += x.d;
            fam_v += 1;
          }
          const bool append = CtaStep<2048, V, kConv, LiveLoads>(a, rv, x, tvals, tkeys, tused, team_sh[team], tt,
                                                                 1 + team, false);
          if (tt < 32) mb.Add(movers, a.movers, append, v);
        }
        if (tt == 0) sh.team_item[team] = next;
        TeamSync<kCtaWarps * 32>(1 + team);
        item = sh.team_item[team];
        TeamSync<kCtaWarps * 32>(1 + team);
      }
    }
    // Stage 2: warps, runs of consecutive vertices.
    {
      const uint32_t first = sh.bin_start[kBinW128];
      const uint32_t items = sh.bin_start[kTeamLow] - first;
      const uint32_t split = sh.bin_start[kBinW256] - first;  // vertices of degree <= 128 come first
      const uint32_t run = min(4u, max(1u, items / (G * kLW * 8)));
      const uint32_t runs = (items + run - 1) / run;
      const uint32_t* wl = l.list + first;
      uint32_t r = blockIdx.x * kLW + warp;
      while (r < runs) {
        uint32_t next = 0;
        if (lane == 0) next = G * kLW + atomicAdd(&ctr->queue[2], 1u);
        const uint32_t e = items - r * run, b = e > run ? e - run : 0;
        uint32_t vid = wl[e - 1];
        for (uint32_t i = e; i > b; --i) {
          const uint32_t v = vid;
          if (i - 1 > b) vid = wl[i - 2];
          if (!InFront(a, rv, v)) continue;
          const VertexCtx x = LoadVertexAs<LiveLoads>(a, v);
          if (lane == 0) {
            fam_e += x.d;
            fam_v += 1;
          }
          bool append;
          if (sizeof(V) == 4 && i - 1 >= split)
            append = WarpStep<512, V, kConv, LiveLoads>(a, rv, x, wvals, wkeys, wused, false);
          else
            append = WarpStep<256, V, kConv, LiveLoads>(a, rv, x, wvals, wkeys, wused, false);
          mb.Add(movers, a.movers, append, v);
        }
        r = __shfl_sync(kFull, next, 0);
      }
    }
    if (fam_v) {
      atomicAdd(&sh.fam_e[kFamWarp], fam_e);
      atomicAdd(&sh.fam_v[kFamWarp], fam_v);
    }
    fam_e = fam_v = 0;
    // Stage 3: lane groups, runs of warp steps over the four bins.
    {
      const uint32_t s0 = sh.bin_start[kBinG4], s1 = sh.bin_start[kBinG8], s2 = sh.bin_start[kBinG16],
                     s3 = sh.bin_start[kBinG32], s4 = sh.bin_start[kBinW128];
      auto exact = [&](uint32_t v, int cres, uint32_t cmove) {
        return GroupExact<V, LiveLoads>(a, rv, v, cres, cmove);
      };
      const uint32_t n32 = s4 - s3, n16 = (s3 - s2 + 1) / 2, n8 = (s2 - s1 + 3) / 4, n4 = (s1 - s0 + 7) / 8;
      const uint32_t steps = n32 + n16 + n8 + n4;
      const uint32_t run = min(8u, max(1u, steps / (G * kLW * 8)));
      const uint32_t runs = (steps + run - 1) / run;
      uint32_t r = blockIdx.x * kLW + warp, got = 0, i = 0, end = 0;
      // The next step (kNone: none), as for the warps.
      auto take = [&]() -> uint32_t {
        if (i == end) {
          if (end) r = __shfl_sync(kFull, got, 0);
          if (r >= runs) return kNone;
          if (lane == 0) got = G * kLW + atomicAdd(&ctr->queue[3], 1u);
          i = r * run;
          end = min(steps, i + run);
        }
        return i++;
      };
      // Lanes per vertex of a step, and the vertex of the calling lane.
      auto width = [&](uint32_t s) { return s < n32 ? 32u : s < n32 + n16 ? 16u : s < n32 + n16 + n8 ? 8u : 4u; };
      auto head = [&](uint32_t s, GroupRow& row) {
        uint32_t p, e;
        if (s < n32) {
          p = s3 + s;
          e = s4;
        } else if (s < n32 + n16) {
          p = s2 + (s - n32) * 2 + lane / 16;
          e = s3;
        } else if (s < n32 + n16 + n8) {
          p = s1 + (s - n32 - n16) * 4 + lane / 8;
          e = s2;
        } else {
          p = s0 + (s - n32 - n16 - n8) * 8 + lane / 4;
          e = s1;
        }
        const bool in = s != kNone && p < e;
        GroupHead<LiveLoads>(a, rv, in, in ? l.list[p] : 0u, row);
      };
      auto entry = [&](unsigned g, GroupRow& row) {
        const unsigned gl = lane & (g - 1);
        row.u = row.v;
        if (row.in && gl < row.d) {
          row.u = a.nbr[row.b + gl];
          row.w = a.w ? a.w[row.b + gl] : 1.0f;
        }
      };
      uint32_t gf_e = 0, gf_v = 0;
      GroupRow row, ahead;
      uint32_t step = take();
      if (step != kNone) {
        unsigned g = width(step);
        head(step, row);
        entry(g, row);
        while (true) {
          step = take();
          const bool more = step != kNone;
          const unsigned gn = width(step);
          head(step, ahead);
          auto load = [&] { entry(gn, ahead); };
          if (pend.n + 32 / g > 32) DecidePending<V, LiveLoads>(a, rv, pend, false, mb, movers, exact);
          if (g == 32)
            GroupScan<32, V, LiveLoads>(a, row, wstage, pend, gf_e, gf_v, load);
          else if (g == 16)
            GroupScan<16, V, LiveLoads>(a, row, wstage, pend, gf_e, gf_v, load);
          else if (g == 8)
            GroupScan<8, V, LiveLoads>(a, row, wstage, pend, gf_e, gf_v, load);
          else
            GroupScan<4, V, LiveLoads>(a, row, wstage, pend, gf_e, gf_v, load);
          if (!more) break;
          row = ahead;
          g = gn;
        }
        DecidePending<V, LiveLoads>(a, rv, pend, false, mb, movers, exact);
      }
      fam_e += gf_e;
      fam_v += gf_v;
    }
    mb.Flush(movers, a.movers);
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
      fam_e += __shfl_xor_sync(kFull, fam_e, o);
      fam_v += __shfl_xor_sync(kFull, fam_v, o);
    }
    if (lane == 0 && fam_v) {
      atomicAdd(&sh.fam_e[kFamGroup], fam_e);
      atomicAdd(&sh.fam_v[kFamGroup], fam_v);
    }
    if (!GridSync(sh, count, arrivals += G, l.polls)) break;

    // ---- Rows above degree 4096: their tables, slice by slice --------------
    if (l.num_slices) {
      for (uint32_t item = blockIdx.x; item < l.num_slices; item += G) {
        const uint32_t hb = l.slice_hub[item];
        const uint32_t v = l.big_v[hb];
        if (!InFront(a, rv, v)) continue;  // uniform over the CTA
        const VertexCtx x = LoadVertexAs<LiveLoads>(a, v);
        const uint32_t s0 = l.slice_start[item];
        const uint32_t len = min(kLoopSlice, l.big_cap[hb] - s0);
        const long long T = l.gt_int[hb];
        if (tid == 0) {
          sh.hub.change = ChangeOf(a, x, UnitsToDouble<long long>(a, T));
          sh.hub.change32 = static_cast<float>(sh.hub.change);
        }
        __syncthreads();
        const double change = sh.hub.change;
        double bv;
        uint32_t bi;
        const unsigned long long base = l.big_base[hb] + s0;
        EvalTable<kLT, true, false, V>(a, x, a.kf[v], change, T, l.gkeys + base,
                                       reinterpret_cast<V*>(l.gvals) + base, len, sh.hub, &bv, &bi);
        const uint32_t sb = l.big_sbase[hb], ns = l.big_nslices[hb];
        if (tid == 0) {
          l.gpart_val[sb + s0 / kLoopSlice] = bv;
          l.gpart_id[sb + s0 / kLoopSlice] = bi;
          __threadfence();
          sh.hub.last = atomicAdd(&l.gdone[hb], 1u) == ns - 1 ? 1u : 0u;
        }
        __syncthreads();
        if (sh.hub.last) {  // uniform: the CTA of the hub's last slice combines the bests
          __threadfence();
          double cv = 0.0;
          uint32_t ci = kNone;
          for (uint32_t j = tid; j < ns; j += kLT)
            KeepBest(cv, ci, __ldcg(l.gpart_val + sb + j), __ldcg(l.gpart_id + sb + j));
          BlockArgmax<kLT>(cv, ci, sh.hub.red_k, sh.hub.red_i);
          if (tid == 0) {
            HubDecide<false>(a, x, cv, ci, change, rv.stamp, movers);
            l.gdone[hb] = 0;
            l.gt_int[hb] = 0;
          }
        }
        __syncthreads();
      }
      if (!GridSync(sh, count, arrivals += G, l.polls)) break;
    }

    // ---- Moves: every mover leaves its cluster and joins its target --------
    const uint32_t M = *movers;
    if (blockIdx.x == 0 && tid == 0) l.st->ctr[(round + 1) % 3] = LoopCounters{};
    if (M) {
      const uint64_t limit = (uint64_t(M) + 31) & ~uint64_t(31);
      for (uint64_t i = uint64_t(blockIdx.x) * kLT + tid; i < limit; i += uint64_t(G) * kLT) {
        const bool in = i < M;
        const uint32_t v = in ? a.movers[i] : 0u;
        const uint32_t c = in ? a.C[v] : kNone;
        const uint32_t t = in ? a.moves[v] : n;
        const double kv = in ? a.k[v] : 0.0;
        if (in) l.old_cluster[i] = c;
        {
          const unsigned peers = __match_any_sync(kFull, c);
          const double tot = GroupSum(peers, kv);
          if (in && int(lane) == __ffs(peers) - 1) {
            atomicSub(&a.s_mut[c], uint32_t(__popc(peers)));
            atomicAdd(&a.K_mut[c], -tot);
            l.mod_stamp[c] = rv.stamp;
          }
        }
        const bool isnew = in && t == n;
        if (isnew) l.new_stamp[v] = rv.stamp;
        const unsigned nb = __ballot_sync(kFull, isnew);
        if (nb && lane == 0) atomicAdd(&ctr->new_movers, uint32_t(__popc(nb)));
        const bool join = in && t != n;
        const unsigned peers = __match_any_sync(kFull, join ? t : kNone);
        const double tot = GroupSum(peers, join ? kv : 0.0);
        if (join && int(lane) == __ffs(peers) - 1) {
          atomicAdd(&a.s_mut[t], uint32_t(__popc(peers)));
          atomicAdd(&a.K_mut[t], tot);
          l.mod_stamp[t] = rv.stamp;
        }
        if (join) a.C_mut[v] = t;
      }
      if (!GridSync(sh, count, arrivals += G, l.polls)) break;

      // New clusters take the ascending list of empty ids, in ascending
      // vertex order: each CTA counts both in its slice of the ids, then
      // writes its part of the two lists.
      const uint32_t N = ctr->new_movers;
      if (N) {
        // Thread t holds `per` consecutive ids (a multiple of 4, at most
        // 4 * 32), one bit each.
        const uint32_t per = ((n + G * kLT - 1) / (G * kLT) + 3) & ~3u;
        const uint64_t lo = uint64_t(blockIdx.x * kLT + tid) * per;
        uint32_t zm[kMaskWords], wm[kMaskWords], z = 0, w = 0;
#pragma unroll
        for (int q = 0; q < kMaskWords; ++q) {
          zm[q] = wm[q] = 0;
          const uint64_t e = min(uint64_t(n), min(lo + per, lo + 32 * (q + 1)));
          for (uint64_t i = lo + 32 * q; i < e; i += 4) {
            const unsigned sh4 = unsigned(i - lo) & 31u;
            if (i + 4 <= e) {
              const uint4 s4 = *reinterpret_cast<const uint4*>(a.s_mut + i);
              const uint4 w4 = *reinterpret_cast<const uint4*>(l.new_stamp + i);
              zm[q] |= ((s4.x == 0u) | (s4.y == 0u) << 1 | (s4.z == 0u) << 2 | (s4.w == 0u) << 3) << sh4;
              wm[q] |= ((w4.x == rv.stamp) | (w4.y == rv.stamp) << 1 | (w4.z == rv.stamp) << 2 |
                        (w4.w == rv.stamp) << 3) << sh4;
            } else {
              for (uint64_t j = i; j < e; ++j) {
                zm[q] |= uint32_t(a.s_mut[j] == 0u) << (unsigned(j - lo) & 31u);
                wm[q] |= uint32_t(l.new_stamp[j] == rv.stamp) << (unsigned(j - lo) & 31u);
              }
            }
          }
          z += __popc(zm[q]);
          w += __popc(wm[q]);
        }
        // Ranks inside the CTA: zeros in the low, new movers in the high word.
        unsigned long long pair = (static_cast<unsigned long long>(w) << 32) | z;
        const unsigned long long inc = WarpInclusiveScan<unsigned long long>(pair);
        if (lane == 31) sh.red64[warp] = inc;
        __syncthreads();
        unsigned long long before = inc - pair, total = 0;
#pragma unroll
        for (int q = 0; q < kLW; ++q) {
          if (unsigned(q) < warp) before += sh.red64[q];
          total += sh.red64[q];
        }
        if (tid == 0) {
          l.st->zeros[blockIdx.x] = uint32_t(total);
          l.st->news[blockIdx.x] = uint32_t(total >> 32);
        }
        if (!GridSync(sh, count, arrivals += G, l.polls)) break;
        uint32_t zb = 0, wb = 0;
        for (uint32_t i = tid; i < blockIdx.x; i += kLT) {
          zb += l.st->zeros[i];
          wb += l.st->news[i];
        }
        zb = BlockSum32(zb, sh.red_a) + uint32_t(before);
        wb = BlockSum32(wb, sh.red_b) + uint32_t(before >> 32);
#pragma unroll
        for (int q = 0; q < kMaskWords; ++q) {
          for (uint32_t mk = zm[q]; mk && zb < N; mk &= mk - 1) l.zero_ids[zb++] = uint32_t(lo + 32 * q + __ffs(mk) - 1);
          for (uint32_t mk = wm[q]; mk; mk &= mk - 1) l.new_list[wb++] = uint32_t(lo + 32 * q + __ffs(mk) - 1);
        }
        if (!GridSync(sh, count, arrivals += G, l.polls)) break;
        for (uint32_t i = blockIdx.x * kLT + tid; i < N; i += G * kLT) {
          const uint32_t v = l.new_list[i];
          const uint32_t cid = l.zero_ids[i];
          a.C_mut[v] = cid;
          a.s_mut[cid] = 1u;
          a.K_mut[cid] = a.k[v];
          l.mod_stamp[cid] = rv.stamp;
        }
        if (!GridSync(sh, count, arrivals += G, l.polls)) break;
      }
      // FP32 images of the modified clusters' weights.
      for (uint32_t i = blockIdx.x * kLT + tid; i < M; i += G * kLT) {
        const uint32_t c0 = l.old_cluster[i], c1 = a.C[a.movers[i]];
        l.Kf_mut[c0] = FilterF32(a.K[c0]);
        l.Kf_mut[c1] = FilterF32(a.K[c1]);
      }
    }

    // ---- Next frontier: the neighbours of the marked rows -------------------
    if (!all_move) {
      Pusher p{l.next_stamp, a.off, rv.stamp};
      const bool by_cluster = l.move_method == PCC_NBHR_CLUSTER_MOVE;
      auto marked = [&](uint32_t v) {
        return by_cluster ? l.mod_stamp[a.C[v]] == rv.stamp : a.moved_stamp[v] == rv.stamp;
      };
      if (!by_cluster || M) {
        // Entries [b, e) by T threads (thread t), eight ids in flight each.
        auto push = [&](uint64_t b, uint64_t e, unsigned t, unsigned T) {
          for (uint64_t j0 = b + t; j0 < e; j0 += 8ull * T) {
            uint32_t u[8], cur[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) u[k] = j0 + uint64_t(T) * k < e ? a.nbr[j0 + uint64_t(T) * k] : kNone;
#pragma unroll
            for (int k = 0; k < 8; ++k) cur[k] = u[k] != kNone ? l.next_stamp[u[k]] : rv.stamp;
#pragma unroll
            for (int k = 0; k < 8; ++k)
              if (cur[k] != rv.stamp) p.Mark(u[k], cur[k]);
          }
        };
        // Each kind of row starts at the CTA where the kind before it ended.
        uint32_t turn = 0;
        auto shifted = [&]() { return blockIdx.x >= turn ? blockIdx.x - turn : blockIdx.x + G - turn; };
        for (uint32_t item = blockIdx.x; item < l.num_chunks; item += G) {
          const uint32_t v = l.big_v[l.chunk_hub[item]];
          if (!marked(v)) continue;
          const uint64_t b = a.off[v] + l.chunk_start[item];
          push(b, min(a.off[v + 1], b + kLoopChunk), tid, kLT);
        }
        turn = l.num_chunks % G;
        // Degree 257-4096: a team per row.
        const uint32_t r0 = sh.push_start[kBinW512], r1 = sh.push_start[kBinGlobal];
        for (uint32_t i = r0 + shifted() * kTeams + team; i < r1; i += G * kTeams) {
          const uint32_t v = l.push_list[i];
          if (marked(v)) push(a.off[v], a.off[v + 1], tid & (kCtaWarps * 32 - 1), kCtaWarps * 32);
        }
        turn = (turn + (r1 - r0 + kTeams - 1) / kTeams) % G;
        // Degree 33-256: a warp per row.
        const uint32_t r2 = sh.push_start[kBinW128];
        for (uint32_t i = r2 + shifted() * kLW + warp; i < r0; i += G * kLW) {
          const uint32_t v = l.push_list[i];
          if (marked(v)) push(a.off[v], a.off[v + 1], lane, 32);
        }
        turn = (turn + (r0 - r2 + kLW - 1) / kLW) % G;
        // Degree <= 32: a warp walks the entries of 32 rows.
        uint32_t* incl = reinterpret_cast<uint32_t*>(extra + size_t(warp) * wslots);
        uint32_t* rowb = incl + 32;  // row starts relative to nbr (entries < 2^32)
        for (uint32_t i0 = (shifted() * kLW + warp) * 32; i0 < r2; i0 += G * kLT) {
          uint32_t d = 0, b = 0;
          if (i0 + lane < r2) {
            const uint32_t v = l.push_list[i0 + lane];
            if (marked(v)) {
              b = uint32_t(a.off[v]);
              d = uint32_t(a.off[v + 1]) - b;
            }
          }
          const uint32_t inc = WarpInclusiveScan<uint32_t>(d);
          incl[lane] = inc;
          rowb[lane] = b - (inc - d);
          const uint32_t total = __shfl_sync(kFull, inc, 31);
          __syncwarp();
          for (uint32_t e0 = 0; e0 < total; e0 += 128) {
            uint32_t u[4], cur[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const uint32_t e = e0 + 32 * k + lane;
              u[k] = kNone;
              if (e < total) {
                uint32_t lo = 0;  // the first row with incl > e
#pragma unroll
                for (uint32_t h = 16; h; h >>= 1)
                  if (incl[lo + h - 1] <= e) lo += h;
                u[k] = a.nbr[uint32_t(rowb[lo] + e)];
              }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) cur[k] = u[k] != kNone ? l.next_stamp[u[k]] : rv.stamp;
#pragma unroll
            for (int k = 0; k < 4; ++k)
              if (cur[k] != rv.stamp) p.Mark(u[k], cur[k]);
          }
          __syncwarp();
        }
        const uint32_t c = __reduce_add_sync(kFull, p.cnt);
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) p.deg += __shfl_xor_sync(kFull, p.deg, o);
        if (lane == 0) {
          sh.red_a[warp] = c;
          sh.red64[warp] = p.deg;
        }
        __syncthreads();
        if (tid == 0) {
          uint32_t cs = 0;
          unsigned long long ds = 0;
          for (int q = 0; q < kLW; ++q) {
            cs += sh.red_a[q];
            ds += sh.red64[q];
          }
          if (cs) {
            atomicAdd(&ctr->frontier, cs);
            atomicAdd(&ctr->pend_edges, ds);
          }
        }
      }
    }
    if (!GridSync(sh, count, arrivals += G, l.polls)) break;

    // ---- End of the round ----------------------------------------------------
    const uint32_t F = all_move ? n : ctr->frontier;
    const unsigned long long E = all_move ? l.m : ctr->pend_edges;
    const bool next = F > 0;
    if (blockIdx.x == 0 && tid == 0) {
      LoopHead& h = l.st->head;
      h.rounds += 1;
      h.edge_visits += front_edges;
      h.vertex_visits += front_size;
      h.visited += visited;
      h.moves += M;
      if (next) h.level_moved = 1;
      h.rs.stamp = rv.stamp;
    }
    rv.front_val = rv.stamp;
    rv.all = all_move;
    rv.stamp += 1;
    front_edges = E;
    front_size = F;
    visited = all_move ? l.binned : F;
    if (!next) break;
  }
  __syncthreads();
  if (tid == 0 && !sh.ok) l.st->head.error = kErrBarrier;
  if (tid < kNumFamilies && sh.fam_v[tid]) {
    atomicAdd(&a.ctr->fam_entries[tid], sh.fam_e[tid]);
    atomicAdd(&a.ctr->fam_vertices[tid], sh.fam_v[tid]);
  }
}

static_assert(kLoopIdsPerCta == uint64_t(kLT) * kMaskWords * 32, "ids of a CTA");

template <typename V, bool kConv>
Status LaunchLoop(Context* ctx, RoundLoopArgs& l) {
  auto kernel = RoundLoopKernel<V, kConv>;
  constexpr size_t kSlotBytes = 4 + sizeof(V) + 1;
  int per_sm = 0;
  const size_t smem = size_t(l.table_slots) * kSlotBytes;
  PCC_RETURN_IF_ERROR(PrepareKernel(kernel, kLT, smem, size_t(2 * kHubSmallMax) * kSlotBytes, &per_sm));
  if (per_sm <= 0) return MakeError(PCC_INTERNAL, "round kernel cannot be configured");
  // One CTA per 1024 entries (two steps of each of its warps) or per 16,384
  // vertices (the empty-id scan), at most every resident CTA: a barrier's cost
  // grows with the CTAs that arrive at it.  The smallest levels need none.
  uint64_t want = std::max<uint64_t>((l.m + 1023) / 1024, (uint64_t(l.a.n) + 16383) / 16384);
  if (l.m <= 1024 && l.a.n <= kLoopIdsPerCta) want = 1;
  const unsigned cap = std::min<unsigned>(unsigned(ctx->num_sms) * unsigned(per_sm), kLoopMaxCtas);
  const unsigned grid = unsigned(std::max<uint64_t>(1, std::min<uint64_t>(want, cap)));
  if (uint64_t(grid) * kLoopIdsPerCta < l.a.n) return MakeError(PCC_INTERNAL, "too many vertices for the round kernel");
  void* args[] = {&l};
  PCC_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kernel), dim3(grid), dim3(kLT), args, smem,
                                       ctx->stream));
  PCC_COUNT(1);
  return LaunchCheck();
}

}  // namespace

void SetLoopHubs(RoundLoopArgs* l, const HubPlan& plan, const HubState& st) {
  l->small_v = plan.small_v;
  l->num_small = plan.num_small;
  l->num_big = plan.num_big;
  l->big_v = plan.big_v;
  l->big_base = plan.loop_base;
  l->big_cap = plan.loop_cap;
  l->big_nslices = plan.loop_nslices;
  l->big_sbase = plan.loop_sbase;
  l->chunk_hub = plan.chunk_hub;
  l->chunk_start = plan.chunk_start;
  l->num_chunks = plan.num_chunks;
  l->slice_hub = plan.loop_slice_hub;
  l->slice_start = plan.loop_slice_start;
  l->num_slices = plan.num_loop_slices;
  l->gkeys = st.gkeys.p;
  l->gvals = st.gvals.p;
  l->gt_int = st.gt_int.p;
  l->gpart_val = st.gpart_val.p;
  l->gpart_id = st.gpart_id.p;
  l->gdone = st.gdone.p;
}

Status RunRoundLoop(Context* ctx, RoundLoopArgs l, const SumMode& mode, const uint32_t* host_counts,
                    uint32_t max_deg, LoopHead* head) {
  // Table slots of a CTA: 16 warps x 256 or four teams x 2048 (which also
  // holds 16 warps x 512 and a hub of degree 4096).
  bool wide = max_deg > kHubMinDegree;
  for (int b = kBinW256; b <= kBinW1000; ++b) wide = wide || host_counts[b] > 0;
  l.table_slots = wide ? 2 * kHubSmallMax : 4096;
  constexpr size_t kSent = offsetof(LoopState, zeros);
  static_assert(Context::kPinLoop + kSent <= Context::kPinnedBytes, "staging");
  unsigned char* stage;
  PCC_RETURN_IF_ERROR(ctx->Pinned(Context::kPinLoop, &stage));
  std::memset(stage, 0, kSent);
  std::memcpy(stage, head, sizeof(LoopHead));
  std::memcpy(stage + offsetof(LoopState, barrier), &kBarrierStart, sizeof(kBarrierStart));
  PCC_CUDA(cudaMemcpyAsync(l.st, stage, kSent, cudaMemcpyHostToDevice, ctx->stream));
  if (!mode.narrow) {
    PCC_RETURN_IF_ERROR((LaunchLoop<long long, true>(ctx, l)));
  } else if (mode.conv) {
    PCC_RETURN_IF_ERROR((LaunchLoop<int, true>(ctx, l)));
  } else {
    PCC_RETURN_IF_ERROR((LaunchLoop<int, false>(ctx, l)));
  }
  PCC_CUDA(cudaMemcpyAsync(stage, l.st, sizeof(LoopHead), cudaMemcpyDeviceToHost, ctx->stream));
  PCC_RETURN_IF_ERROR(Sync(ctx));
  std::memcpy(head, stage, sizeof(LoopHead));
  if (head->error) return MakeError(PCC_INTERNAL, "device error flag " + std::to_string(head->error));
  return Status::Ok();
}

}  // namespace pcc
