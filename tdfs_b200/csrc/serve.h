// serve.h -- continuous-batching query server (serve.cpp).
#pragma once

#include <cstddef>
#include <cstdint>

#include "common.h"
#include "flat.cuh"
#include "graph.h"
#include "match.cuh"

namespace tdfs {

// Launch shape of the persistent match kernel (capi.cpp).
struct LaunchShape {
  int warps_per_block;
  int blocks;
  KernelCfg cfg;
};
int launch_shape(const tdfs_graph *g, int kmax, bool labeled, const tdfs_options &o, LaunchShape *out);

// The level-0 range of a slot over edge ids [eb, ee), through the graph's
// label index for labeled plans when use_index is set (capi.cpp).
void level0_range(const tdfs_graph *g, const DevPlan &p, int64_t eb, int64_t ee, bool use_index, SlotInfo *in);

// The device plan table of a compiled pattern, and its form for the flat
// kernel (nullptr when it has none) (capi.cpp).
const DevPlan &plan_device_table(const tdfs_plan *p);
const FlatPlan *plan_flat_table(const tdfs_plan *p);

// Launch shape of the flat kernel for plans with tails of up to tmax vertices,
// holding `levels` levels in shared memory (big: and level 2 of some plan in
// global memory), on a skewed graph or not, idle warps waiting to be given work
// (share) or leaving, from the options launch_shape has accepted (capi.cpp).
struct FlatShape {
  int warps_per_block;
  int blocks;
  FlatCfg cfg;
};
int flat_shape(int device, int levels, int tmax, bool skewed, bool big, bool share, bool labeled, const tdfs_options &o,
               FlatShape *out);

// Do these options leave the choice of the kernel to the library?  A work
// budget, stealing switched off, or a value for one of the DFS kernel's own
// knobs asks for the DFS kernel.
bool flat_options(const tdfs_options &o);

struct Server;
size_t query_bytes(int k, int cap, int warps_per_block);
int server_create(tdfs_graph *g, const tdfs_server_options *o, Server **out);
int server_submit(Server *s, const DevPlan &plan, uint64_t *ticket);
int server_wait(Server *s, uint64_t ticket, uint64_t *count, double *latency_us);
int server_stats(Server *s, tdfs_serve_stats *st);
int server_destroy(Server *s);

}  // namespace tdfs
