// common.h -- types shared by the host plan compiler, the C ABI and the
// sm_100a kernels of the tdfs B200 engine.
#pragma once

#include <cstdint>
#include <string>

#include "../../include/tdfs.h"

namespace tdfs {

constexpr int kMaxK = TDFS_MAX_PATTERN;  // pattern vertices (src/config.h:11)
constexpr int kWarp = 32;

// Condition operators, numbered as the reference's CondOperator
// (src/pattern.h:21).
enum CondOp : int { kLess = 0, kLarger = 1, kNonEqual = 2 };

// Device plan table: everything the DFS kernel reads about one pattern.  It
// is passed by value as a __grid_constant__ kernel parameter (or sits in a
// device array for batched launches), so it lives in the constant bank.
struct DevPlan {
  int32_t k;          // pattern vertices, 3..7
  int32_t labeled;    // lb (1) or ulb (0) semantics
  int32_t orient;     // level-0 edges kept only when r < c (unlabeled)
  int32_t deg[3];     // pattern degrees of vertices 0, 1, 2 (job filter)
  int32_t label[kMaxK];       // pattern vertex labels (255 = matches nothing)
  int32_t nbn[kMaxK];         // backward neighbours of vertex i
  int8_t bn[kMaxK][kMaxK];
  int32_t dep[kMaxK];         // reuse: candidates of vertex dep[i] (or -1)
  int32_t nsh[kMaxK];         // extra backward neighbours under reuse
  int8_t bnsh[kMaxK][kMaxK];
  uint8_t larger[kMaxK];      // bit j: x > phi(j)
  uint8_t less[kMaxK];        // bit j: x < phi(j)
  uint8_t neq[kMaxK];         // bit j: x != phi(j)
  uint8_t pad_;
  uint64_t multiplicity;      // |Aut| multiplier (unlabeled)
};

// ---- flat plans (flat.cu) ---------------------------------------------------
// One candidate set as the flat kernel produces or counts it: the backward
// neighbours whose lists are intersected, the label, and bit masks over the
// earlier vertices j of the conditions x > phi(j), x < phi(j), x != phi(j).
// With dep != 0 the set is also the candidate set of the earlier vertex dep
// intersected with the lists of bnsh (the plan's reuse level).
struct FlatStep {
  uint8_t nbn;
  uint8_t bn[kMaxK - 1];
  uint8_t label;
  uint8_t larger, less, neq;
  uint8_t dep, nsh;
  uint8_t bnsh[3];
};

// How the flat kernel runs a plan: vertices 2..s are enumerated (step[i - 2]);
// the t = k - 1 - s vertices after s are counted below each level-s node from
// the sizes of the candidate sets term[]: term_of[m] is the set shared by the
// tail vertices in bit mask m (kNoTerm: empty).  form 0: tuples of distinct
// vertices by inclusion-exclusion; form 1: the tail vertices have one and the
// same set and a total order among them, so the tuples are its t-subsets.
constexpr uint8_t kNoTerm = 255;
struct FlatPlan {
  int32_t k, orient;
  int32_t deg[3];
  int32_t label[2];     // of pattern vertices 0 and 1
  uint8_t s, t, form, nterm;
  uint8_t reuse2;       // 1: some set is taken from the candidate sets of vertex 2
  uint8_t pad_[3];
  uint8_t term_of[8];
  FlatStep step[4];
  FlatStep term[7];
};

// The flat form of a plan; false when it has none (flat_plan.cpp).
bool flat_plan(const DevPlan &d, FlatPlan *out);

// Device view of a resident data graph.
struct DevGraph {
  const int64_t *rowptr;   // n + 1
  const int32_t *colidx;   // nedges (+ padding)
  const int32_t *src;      // edge -> source vertex, nedges
  const uint8_t *label;    // n, or nullptr
  const int32_t *maxnd;    // max degree over each vertex's neighbours
  const int32_t *lperm;    // level-0 label index (labeled graphs), or nullptr
  const int32_t *colidx_l; // labeled graphs with few labels: every row re-sorted by (label, id), or nullptr
  const int32_t *loff;     // its segment starts: loff[v * (nlab + 1) + l], relative to rowptr[v]
  const int32_t *hash;     // row membership tables (see row_table_buckets), or nullptr
  const int32_t *loops;    // with hash: not 0 when some row holds its own vertex
  int32_t nlab;            // labels 0..nlab-1 have segments
  int64_t nedges;
  int32_t n;
  int32_t max_degree;
};

// ---- row membership tables ---------------------------------------------------
// Every adjacency row again as a hash table of 8-entry buckets (32 bytes: one
// load, one sector): "is y in row v?" costs one load, whatever the row's
// length, where a binary search costs log2(degree) dependent ones.  Row v owns
// the buckets [first, first + count) with first = row_table_at(rowptr[v]) + v, so
// no offset array is needed and a bucket holds 3.2 entries on average.  Entries
// fill a bucket in order, -1 is empty; a full bucket (about two in a hundred)
// overflows into the next one, cyclically within the row.
constexpr int kBucket = 8;
constexpr int64_t row_table_at(int64_t r) { return (r >> 2) + (r >> 4); }
inline int64_t row_table_buckets(int64_t n, int64_t nedges) { return row_table_at(nedges) + n + 1; }
constexpr uint32_t kRowHash = 0x9E3779B1u;  // 2^32 / golden ratio: neighbouring ids spread over the buckets

// Per-launch control block in device memory.  Counters that many warps touch
// sit on their own 128-byte lines so ticket atomics, idle polling and the
// final count do not serialise on one L2 line.
struct alignas(128) RunCtl {
  int32_t hungry;                // warps idle and looking for work
  char pad0_[124];
  unsigned long long steals;     // diagnostics: intra-block steals
  unsigned long long splits;     // diagnostics: units through the global queue
  int32_t error;                 // TDFS_ERR_* raised by the kernel
  int32_t pad_;
  unsigned long long idle_ns;    // diagnostics: summed time warps spent without work
  unsigned long long warp_ns;    // diagnostics: summed time warps ran
  int32_t finished;              // flat kernel: 1 = no work was left anywhere
  char pad1_[84];
};

// Error reporting shared by the C ABI implementation files.
void set_error(const char *fmt, ...);
int fail(int code, const char *fmt, ...);

}  // namespace tdfs
