// Arguments of the vocabulary-parallel local pass over the shards that a device holds.
#pragma once
#include "sampling_params.cuh"

namespace ftb200 {

constexpr int kVpMaxShards = 64;           // shards of one launch
constexpr int kVpMaxSmem   = 221 * 1024;  // dynamic; the rest is the kernel's own

struct VpArgs {
    const void* logits[kVpMaxShards];
    u64*        out;       // [n_shards][local_batch][2 + cap]
    int         n_shards;
    int         vocab;     // columns of all shards together, from `offset` on
    int         offset;    // token id of the first column
    int         row_bytes, cand_cap, spec_cap;
};

// Shared memory of a launch: the row (with up to 7 columns in front of it), candidates, listed special columns.
inline void vp_select_plan(VpArgs& V, int shard, int cap, int max_k, int specials, size_t* smem)
{
    V.row_bytes = ((shard + 7) / 8 + 1) * 16;
    V.cand_cap  = max_k <= 256 ? 1024 : 2048;
    V.cand_cap  = V.cand_cap < cap ? (cap + 1) & ~1 : V.cand_cap;
    V.spec_cap  = specials;
    *smem       = (size_t)V.row_bytes + (size_t)V.cand_cap * 8 + (size_t)V.spec_cap * 8;
}

}  // namespace ftb200
