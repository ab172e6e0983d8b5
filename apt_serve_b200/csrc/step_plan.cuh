// The device-side plan of a layer-step whose hidden-cached requests are attended directly: the K/V kernel's chunk list
// and the groups of hidden-cached requests.  Written by step_plan_kernel (hidden_attention.cu).
#pragma once

#include "attention_common.cuh"

namespace aps {

constexpr int kMaxGrid = 192;             // most SMs the plan keeps bounds of pieces for
constexpr int kMaxLevels = 5;             // sizes of pieces the scores work is cut into
constexpr int kMaxPieces = kMaxGrid * kMaxLevels;

// ---- the plan of one group of hidden requests (device memory) --------------------------
struct GroupPlan {
  int n;                      // requests of the group
  int slice;                  // 128-column blocks per item of the sum kernel
  int turns;                  // which cache blocks' weights have their first term last (SumColumns::turn_mask)
  int levels, per_level;      // pieces of the scores work: levels x per_level
  int next_piece, next_item;  // work counters of the scores and the sum kernel
  int req[kGroup];            // batch row of each request, longest first
  int ord[kGroup];            // its place in the group in batch order (folded queries)
  int len[kGroup];            // its length in tokens
  int tile_off[kGroup + 1];   // first scores tile
  int blk_off[kGroup + 1];    // first 16-token block of p
  int bound_tile[kMaxPieces + 1];   // piece c: from (bound_tile[c], bound_step[c]) to the next bound
  int bound_step[kMaxPieces + 1];
};

// The pieces [x, y] that left partial sums of a scores tile, as the scores kernel noted them, kept within those there are.  When
// one of that kernel's waits has run out, the entries of the tiles it did not reach are what the scratch held before: the
// output is then NaN by the status word, but the softmax in between must not follow them out of the scratch.
__host__ __device__ inline int2 clamp_pieces(int2 c, int n_pieces) {
  const int last = n_pieces - 1;
  c.x = c.x < 0 ? 0 : c.x > last ? last : c.x;
  c.y = c.y < 0 ? 0 : c.y > last ? last : c.y;
  return c;
}

struct PlanArgs {
  int* plan; int* part_offset; int2* kv_chunks; int* hid_slot; int2* hid_list; GroupPlan* groups;
  const int32_t* seq_lens; const int32_t* cache_type;
  int batch, max_tokens, kv_present, n_groups, steps, grid_scores, max_slice, item_target;
  int turns;   // four bits for each slice
};
int launch_step_plan(const PlanArgs* plan, const NewTokenWrite& n, cudaStream_t stream);   // plan may be NULL: the new-token writes alone

}  // namespace aps
