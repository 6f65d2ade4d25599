// flat.cuh -- the flattened subgraph-counting kernel.
//
// Same counts as the DFS kernel (match.cuh), another execution: a warp holds
// a buffer of partial embeddings per level and extends 32 of them at once.
// Their source lists are laid end to end and lane t takes every 32nd position,
// so a step tests 32 candidates whatever the list lengths are (one DFS node at
// a time leaves half of the lanes idle on lists of 16, and pays its set-up
// per node).  Membership in the other backward neighbours' lists is one
// 32-byte load of a bucket of the row's hash table.
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
  int32_t check;       // clocks between offers of work
  int32_t segments;    // 1: labeled plans read the label segments of rows (DevGraph::colidx_l)
  int32_t wide;        // 1: the 80-register build (3 CTAs of 256 threads per SM)
  int32_t share;       // 1: idle warps wait to be given work; 0: they leave
};

// Vertices up to this degree: 32 lists laid end to end stay within 32 bits.
constexpr int64_t kFlatMaxDegree = int64_t(1) << 26;

// Shared memory per warp with `entries` buffered partial embeddings, the least
// that a launch's plans can work with, the
// entries that let 4 CTAs of 8 warps share an SM, and the most that one CTA of
// `warps` warps can have.
size_t flat_warp_bytes(int entries);
int flat_min_entries(int levels, int tmax);  // `levels` levels in shared memory, tails of up to tmax vertices
int flat_auto_entries();
int flat_max_entries(int warps);

int flat_blocks_per_sm(bool labeled, bool wide, bool big, int warps_per_block, size_t smem);

// ---- launch records -----------------------------------------------------------
// What a launch over n slots reads and writes besides the graph, in one block
// that the host fills and uploads with one copy:
//   RunCtl | count[n] | FlatCtl | mask of idle warps | FlatInfo[n] | FlatPlan[n]
// The first two come back with one copy, or, with FlatTable::host set, are
// written to (pinned) host memory by one warp of the last CTA.  The copy costs
// a small launch 2 to 7 us more (a call over 1 slot 33.5 against 29.6 us, 128
// slots 46.8 against 39.9), the one warp costs a large one more: 512 slots 90 us
// either way, 1024 slots 141 against 127 with the copy, 16384 1.86 against 1.60 ms.
constexpr int kHostSlots = 512;
constexpr int kFlatBoxes = 8192;  // mailboxes, one per warp of the grid
constexpr int kIdleWords = kFlatBoxes / 32;

// A launch does not need its whole grid on the GPU at once: another kernel may
// hold part of the SMs for as long as it likes.  Where warps wait for work, it
// belongs to nobody before a running CTA takes it, and a CTA counts as busy
// from when it starts, so the CTAs that run finish the launch and one that
// starts later finds nothing.  One atomic does both: a CTA adds kCtaJoin + its
// warps to `ticket`, which takes a ticket per warp and counts the CTA.  Where
// warps leave when they run dry (FlatCfg::share 0), every CTA gets its turn:
// there the host deals the first tickets and counts all CTAs (the atomics of
// 592 CTAs on one word take 3.5 us, a tenth of a triangle count on the n=4096
// ER graph).
constexpr int kJoinShift = 50;  // tickets below, CTAs that have started above
constexpr unsigned long long kCtaJoin = 1ull << kJoinShift;
struct alignas(128) FlatCtl {
  unsigned long long ticket;  // the next ticket; above kJoinShift, the CTAs that have started
  char pad0_[120];
  int32_t pending;            // filled mailboxes - CTAs without a busy warp; the launch is complete when
                              // no tickets are left and this plus the started CTAs is 0
  char pad1_[124];
  int32_t gone;               // CTAs that have left
  char pad3_[124];
  int64_t tickets;            // tickets of all slots
  int32_t slots;
  char pad2_[116];
};

// A slot: tickets [ticket0, ..) of the launch are its level-0 chunks.
struct FlatInfo {
  int64_t ticket0;
  int64_t e_begin, e_end;  // as in SlotInfo
  int32_t stride, phase, chunk, perm;
};

// A mailbox: up to 32 partial embeddings (tuples of level + 1 vertices).
// With `range`, one embedding, of whose children only those in [lo, hi] are
// to be extended.
constexpr int kBoxInts = 153;
struct FlatBox {
  int32_t full;  // 0 empty, 1 filled by the warp that cleared the idle bit
  int32_t level, n, slot;
  int32_t range, lo, hi;
  int32_t v[kBoxInts];
};
constexpr size_t kFlatBoxBytes = sizeof(FlatBox) * kFlatBoxes;

// Level 2 of plans that reuse its candidate sets (FlatPlan::reuse2), on graphs
// whose sets may not fit shared memory: a buffer per warp in global memory.
// An entry whose siblings are all there is extended from them with one test
// per candidate; one whose siblings were cut off, from its shortest list with
// a test per other list (90% of a 5-clique's candidates on the power-law graph
// with 320 entries in shared memory).
constexpr int kBigEntries = 2048;
constexpr size_t kBigBytes = (size_t)kBigEntries * 6;

struct FlatTable {
  RunCtl *run;
  unsigned long long *count;  // raw counts (before the |Aut| multiplier)
  FlatCtl *ctl;
  unsigned *idle;
  FlatInfo *info;
  FlatPlan *plan;
  FlatBox *box;
  int32_t *big;  // kBigBytes per warp, or nullptr
  void *host;    // where RunCtl and count[] go at the end, or nullptr

  static constexpr size_t at_ctl(int n) { return sizeof(RunCtl) + (((size_t)n * 8 + 127) & ~size_t(127)); }
  static constexpr size_t readback(int n) { return sizeof(RunCtl) + (size_t)n * 8; }
  static constexpr size_t bytes(int n) {
    return at_ctl(n) + sizeof(FlatCtl) + 4 * kIdleWords + (size_t)n * (sizeof(FlatInfo) + sizeof(FlatPlan));
  }
  // The views of the block at `base` (device, or its host image).
  static FlatTable of(void *base, int n, FlatBox *box, int32_t *big, void *host) {
    char *b = static_cast<char *>(base);
    FlatTable t;
    t.run = reinterpret_cast<RunCtl *>(b);
    t.count = reinterpret_cast<unsigned long long *>(b + sizeof(RunCtl));
    b += at_ctl(n);
    t.ctl = reinterpret_cast<FlatCtl *>(b);
    t.idle = reinterpret_cast<unsigned *>(b + sizeof(FlatCtl));
    t.info = reinterpret_cast<FlatInfo *>(t.idle + kIdleWords);
    t.plan = reinterpret_cast<FlatPlan *>(t.info + n);
    t.box = box;
    t.big = big;
    t.host = host;
    return t;
  }
  // The control block of a launch with this many CTAs, in a zeroed host image.
  void start(int blocks, int warps_per_block, bool share, int n) const {
    ctl->slots = n;
    if (share) return;  // CTAs take their first tickets and count themselves
    ctl->ticket = (unsigned long long)blocks * warps_per_block + kCtaJoin * blocks;
  }
};

// The most CTAs of a launch (every warp has a mailbox).
inline int flat_max_blocks(int warps_per_block) { return kFlatBoxes / warps_per_block; }
static_assert((unsigned long long)kFlatBoxes < 1ull << (64 - kJoinShift), "a join count for every CTA");

// Hubs: vertices with more neighbours than this.
constexpr int32_t kHubDegree = 512;

// How old a warp's base work must be before it gives some away, and the clocks
// between its looks for idle warps.  Giving work away early costs more than it
// gains where every warp has much of it, or the work is even (64-query ER burst
// 1.08 times as long at 20 us and 4096 clocks).  A launch with fewer than
// kFewEdges level-0 edges per warp in its share of the range, on a graph with
// hubs, is over when its few heavy edges are: they are to be spread soon.  Early
// against late over 216 batches of labeled random queries, shares of them and
// unlabeled cliques on two power-law graphs, as geometric means: 0.94 of the time
// below 8 edges per warp (0.87 to 1.03 by kind and range), 0.97 from 8 to 16, 0.99
// from 16 to 24; beyond, labeled batches take 1.05 times as long, one of them 2.6.
constexpr int kSplitNs = 60000, kCheckCycles = 16384;
constexpr int kFewEdges = 16, kFewSplitNs = 20000, kFewCheckCycles = 4096;

// Level-0 edges per ticket of a slot whose plan is enumerated down to level s,
// in a launch of `edges` level-0 edges over all slots; skewed: on a graph with
// hubs; `edge_chunk` and `stride` as in tdfs_options.
int flat_chunk(int64_t edges, int s, bool skewed, int stride, int warps, int edge_chunk);

// Launch over the slots of `t` (on the device).
int launch_flat(bool labeled, const DevGraph &g, const FlatTable &t, const FlatCfg &cfg, int blocks,
                int warps_per_block, cudaStream_t stream);

}  // namespace tdfs
