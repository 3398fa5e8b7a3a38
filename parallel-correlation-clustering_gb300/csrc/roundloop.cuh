// roundloop.cuh -- all best-move rounds of a level in one kernel
// (roundloop.cu).
#pragma once

#include "hubs.cuh"

namespace pcc {

// Counters of one round.  Three sets take turns: a round's set is cleared
// while the round before it is in its apply phase.
struct LoopCounters {
  uint32_t queue[4];   // best-move stages: work taken beyond the first items
  uint32_t movers;
  uint32_t new_movers;
  uint32_t frontier;   // vertices of the next frontier
  uint32_t pad;
  unsigned long long pend_edges;  // their degree sum
};

// Device state of the kernel: the counter sets, the grid barrier and each
// CTA's counts of empty ids and new movers in its slice of the vertices.
constexpr uint32_t kLoopMaxCtas = 1024;
// Sent before and read after a run (with the counters, zero at its start, and
// the barrier's count).
struct LoopHead {
  RoundState rs;             // in: stamp and the round-0 frontier; out: the last stamp
  uint32_t level_moved;      // some round's next frontier was not empty
  uint32_t rounds;
  uint32_t error;            // kErrBarrier
  uint32_t pad;
  unsigned long long edge_visits, vertex_visits, visited, moves;
};
struct LoopState {
  LoopHead head;
  LoopCounters ctr[3];
  uint32_t barrier;
  uint32_t pad;
  uint32_t zeros[kLoopMaxCtas];
  uint32_t news[kLoopMaxCtas];
};

struct RoundLoopArgs {
  BMArgs a;                 // best-move arguments (rs null; front_stamp: next_stamp)
  const uint32_t* list;     // vertices evaluated, by degree bin
  const uint32_t* starts;   // their bins' starts (kNumBins + 1)
  const uint32_t* push_list;  // rows of degree > 0, by degree bin
  const uint32_t* push_starts;
  uint64_t m;
  uint64_t binned;          // vertices on `list`
  uint32_t num_inner;       // rounds at most
  int32_t move_method;      // PCC_*_MOVE
  uint32_t polls;           // of a barrier, then it gives up (Context::barrier_polls)
  uint32_t* mod_stamp;
  uint32_t* new_stamp;
  uint32_t* next_stamp;
  uint32_t* old_cluster;    // per mover: the cluster it left (n entries)
  uint32_t* zero_ids;
  uint32_t* new_list;
  float* Kf_mut;
  LoopState* st;
  uint32_t table_slots;     // shared-memory table slots of a CTA
  // Hubs (degree > 1000): HubPlan and HubState.
  const uint32_t* small_v;
  uint32_t num_small;
  uint32_t num_big;
  const uint32_t* big_v;
  const unsigned long long* big_base;
  const uint32_t* big_cap;
  const uint32_t* big_nslices;
  const uint32_t* big_sbase;
  const uint32_t* chunk_hub;
  const uint32_t* chunk_start;
  uint32_t num_chunks;
  const uint32_t* slice_hub;
  const uint32_t* slice_start;
  uint32_t num_slices;
  uint32_t* gkeys;
  unsigned long long* gvals;
  long long* gt_int;
  double* gpart_val;
  uint32_t* gpart_id;
  uint32_t* gdone;
};

// Vertices whose empty ids one CTA can rank (roundloop.cu).
constexpr uint64_t kLoopIdsPerCta = 65536;

// Whether a level can run in the kernel: exact sums, at most kLoopMaxEntries
// entries, and no more vertices than one CTA per SM can rank.
inline bool RoundLoopFits(const Context* ctx, const DevGraph& g, const SumMode& mode) {
  return mode.exact && g.n > 0 && g.m <= kLoopMaxEntries &&
         g.n <= kLoopIdsPerCta * uint64_t(ctx->num_sms);
}

// Fills the hub fields from the level's plan and state.
void SetLoopHubs(RoundLoopArgs* l, const HubPlan& plan, const HubState& st);

// Runs the rounds and waits for them.  bins: host counts of `list`; *head: in
// the round state, out the run's results.
Status RunRoundLoop(Context* ctx, RoundLoopArgs l, const SumMode& mode, const uint32_t* host_counts,
                    uint32_t max_deg, LoopHead* head);

}  // namespace pcc
