// flat.cuh -- the flattened subgraph-counting kernel.
//
// Same counts as the DFS kernel (match.cuh), another execution: a warp holds
// a buffer of partial embeddings per level and extends 32 of them at once.
// Their source lists are laid end to end and lane t takes every 32nd position,
// so a step tests 32 candidates whatever the list lengths are (one DFS node at
// a time leaves half of the lanes idle on lists of 16, and pays its set-up
// per node).  Membership in the other backward neighbours' lists is one
// 16-byte load of the row's hash table.
#pragma once

#include <cstdint>

#include "common.h"
#include "graph.h"

namespace tdfs {

struct FlatCfg {
  int32_t entries;     // partial embeddings buffered per warp, over all levels of a plan
  int32_t warp_bytes;  // shared memory per warp
  int32_t idle_ms;     // bounded idle wait before a warp reports a timeout
  int32_t split_ns;    // work may be given away after this long on one base subtree
  int32_t segments;    // 1: labeled plans read the label segments of rows (DevGraph::colidx_l)
};

// Vertices up to this degree: 32 lists laid end to end stay within 32 bits.
constexpr int64_t kFlatMaxDegree = int64_t(1) << 26;

// Shared memory per warp with `entries` buffered partial embeddings, the
// entries that let 4 CTAs of 8 warps share an SM, and the most that one CTA of
// `warps` warps can have.
size_t flat_warp_bytes(int entries);
int flat_auto_entries();
int flat_max_entries(int warps);

int flat_blocks_per_sm(bool labeled, int warps_per_block, size_t smem);

// The most CTAs of a launch (every warp has a mailbox in the ring's memory).
int flat_max_blocks(int warps_per_block);

// Reset the control block and the mask of idle warps (stream-ordered).
void init_flat(RunCtl *ctl, SplitUnit *units, cudaStream_t stream);

// Launch over the slot table `tab` (filled by the host); `units` is the split
// ring's memory.
int launch_flat(bool labeled, const DevGraph &g, RunCtl *ctl, SlotTable *tab, SplitUnit *units, const FlatCfg &cfg,
                int blocks, int warps_per_block, cudaStream_t stream);

}  // namespace tdfs
