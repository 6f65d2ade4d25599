// graph.cu -- device-resident data graph: upload and one-time preprocessing.
//
// Replaces GraphPreprocessor::to_gpu (src/graph.h:34-50) and build_src_vtx
// (src/graph.h:195-212).  HBM layout:
//   rowptr  int64[n+1]        as in the file
//   colidx  int32[E + pad]    as in the file; padded by kColPad ints so that
//                             16-byte vector loads at the end stay in bounds
//   src     int32[E]          edge -> source vertex (built on the device)
//   maxnd   int32[n]          max degree over the neighbours of each vertex,
//                             so the level-0 test "some neighbour of c has
//                             degree >= deg(pattern vertex 2)"
//                             (src/gpu_match.cu:541-548) is one load
//   label   uint8[n]          labeled graphs only (labels must be < 255)
//   hash    int32[8 per bucket]  row membership tables (flat.cu), beside the
//                             label index and label rows of labeled graphs
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "csr.h"
#include "flat.cuh"
#include "graph.h"

namespace tdfs {

namespace {

__global__ void narrow_labels_kernel(const int32_t *__restrict__ in, int32_t n, uint8_t *__restrict__ out,
                                     int32_t *__restrict__ bad) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t l = in[i];
    if (l < 0 || l > 254) atomicExch(bad, 1);
    out[i] = (uint8_t)(l < 0 || l > 254 ? 255 : l);
  }
}

__device__ __forceinline__ unsigned lanes_below() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// ---- label rows and label index on the device (at most kSegLabels labels) --
// Both are stable counting sorts.  Within a warp, the lanes holding the same
// key are found with __match_any_sync; each lane's rank among them (lanes
// below it) plus the counts of the earlier chunks gives its position, so the
// output keeps the input order within every key, as a sequential pass would.

// Edge ids per tile of the label-index sort: small tiles for parallelism
// (one warp walks a tile in order), at most kMaxTiles of them so the
// (key, tile) histogram stays a few MB.
constexpr int64_t kMinTileEdges = 512;
constexpr int64_t kMaxTiles = 8192;
inline int64_t tile_edges(int64_t nedges) {
  const int64_t t = (nedges + kMaxTiles - 1) / kMaxTiles;
  return std::max(kMinTileEdges, (t + 31) & ~int64_t(31));
}
constexpr int kBuildWarps = 8;    // warps per CTA of the build kernels

// ---- the CSR's rules ------------------------------------------------------------
struct CsrCheck {
  int32_t bad;
  int32_t max_degree;
};

// The rules of validate_csr (csr.cpp) on the device copy: a verdict only.  What
// is wrong, and where, the host's pass then says, so the message is the same
// wherever a CSR is checked.  Reads inside the arrays whatever they hold: a
// row's range is only compared, and a descending pair of neighbours is looked
// up among the row starts.  6M edges take 0.10 ms; the host's pass takes 2.8 ms
// with 16 threads (the first of them has the hubs).
__global__ void check_csr_kernel(const int64_t *__restrict__ rowptr, const int32_t *__restrict__ colidx, int64_t n,
                                 int64_t nedges, CsrCheck *out) {
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int32_t md = 0;
  for (int64_t v = first; v < n; v += step) {
    const int64_t lo = rowptr[v], hi = rowptr[v + 1];
    if (lo < 0 || hi > nedges || hi < lo || hi - lo > INT32_MAX) out->bad = 1;
    else md = max(md, (int32_t)(hi - lo));
  }
  md = (int32_t)__reduce_max_sync(0xffffffffu, (unsigned)md);
  if ((threadIdx.x & 31) == 0 && md > 0) atomicMax(&out->max_degree, md);
  for (int64_t j = first; j < nedges; j += step) {
    const int32_t c = colidx[j];
    if (c < 0 || c >= n) out->bad = 1;
    if (j + 1 >= nedges || c < colidx[j + 1]) continue;
    int64_t a = 0, z = n;  // the first row that starts after j
    while (a < z) {
      const int64_t m = (a + z) >> 1;
      if (rowptr[m] <= j) a = m + 1; else z = m;
    }
    if (rowptr[a] != j + 1) out->bad = 1;
  }
}

// ---- what every row gives -------------------------------------------------------
// One pass over the rows writes all that is derived from them: the source of
// every edge, the largest degree among a vertex's neighbours, the row's
// membership table (row_table_buckets, cleared before), and on labeled graphs
// with segments the row again, stably partitioned by neighbour label (col_l),
// with each label's segment start relative to the row start (loff, nl + 1 per
// vertex, the last one the row length).
//
// A warp takes a row; rows of more than kLongRow edges are left to the whole
// CTA, each warp a contiguous part.  Neighbouring vertices go to different
// CTAs: with ids in degree order the hubs come first and would otherwise meet
// in one.  Bound by the chain of dependent loads per row (row, neighbours,
// their degrees and labels): 6M edges over 1.1M vertices take 0.48 ms, where the
// four kernels it replaces took 1.17 ms, 0.76 of them with one warp on a
// 21 000-edge row.
constexpr int kRowWarps = 16;
constexpr int64_t kLongRow = 512;

struct Rows {
  const int64_t *rowptr;
  const int32_t *colidx;
  int32_t n;
  int32_t *src, *maxnd;
  int32_t *hash, *loops;   // nullptr: no tables
  const uint8_t *lab;      // nullptr: no segments
  int32_t nl;
  int32_t *col_l, *loff;
};

// Into row [r, e)'s table: a slot is tried only when the ones before it in its
// bucket are taken, so entries fill a bucket in order whatever the order of
// the threads.
__device__ __forceinline__ void table_insert(int32_t *hash, int32_t v, int64_t r, int64_t e, int32_t x) {
  const uint32_t nb = (uint32_t)(row_table_at(e) - row_table_at(r)) + 1;
  int32_t *t = hash + kBucket * (row_table_at(r) + v);
  uint32_t b = __umulhi((uint32_t)x * kRowHash, nb);
  for (uint32_t tries = 0; tries < nb; ++tries) {
    for (int i = 0; i < kBucket; ++i)
      if (atomicCAS(t + kBucket * (int64_t)b + i, -1, x) == -1) return;
    b = b + 1 == nb ? 0 : b + 1;
  }
}

// First pass over edges [j0, j1) of row v = [b, e), a warp: sources, table, the
// largest neighbour degree + 1 (0 for none), and the label counts into cnt.
template <bool LAB>
__device__ __forceinline__ unsigned row_first(const Rows &R, int32_t v, int64_t b, int64_t e, int64_t j0, int64_t j1,
                                              int32_t *cnt) {
  const int lane = threadIdx.x & 31;
  unsigned m = 0;
  const bool whole = e - b <= 32;  // this warp has the row at once: its table needs no atomics
  for (int64_t c0 = j0; c0 < j1; c0 += 32) {
    const int64_t j = c0 + lane;
    const bool valid = j < j1;
    int key = -1;
    int32_t w = 0;
    if (valid) {
      w = R.colidx[j];
      R.src[j] = v;
      m = max(m, (unsigned)(R.rowptr[w + 1] - R.rowptr[w]) + 1u);
      if (LAB) key = (int)R.lab[w];
    }
    if (R.hash) {
      if (valid && w == v) *R.loops = 1;
      bool left = valid;
      if (whole) {
        const uint32_t nb = (uint32_t)(row_table_at(e) - row_table_at(b)) + 1;
        const int bk = valid ? (int)__umulhi((uint32_t)w * kRowHash, nb) : -1;
        const int rank = __popc(__match_any_sync(0xffffffffu, bk) & lanes_below());
        left = valid && rank >= kBucket;
        if (valid && !left) R.hash[kBucket * (row_table_at(b) + v + bk) + rank] = w;
        if (__any_sync(0xffffffffu, left)) {  // a bucket overflows: its other entries are in place first
          __threadfence();
          __syncwarp();
        }
      }
      if (left) table_insert(R.hash, v, b, e, w);
    }
    if (LAB) {
      const unsigned same = __match_any_sync(0xffffffffu, key);
      if (valid && lane == __ffs(same) - 1) cnt[key] += __popc(same);
      __syncwarp();
    }
  }
  return m;
}

// Second pass: every neighbour to its label's next place (cursors in cnt).
__device__ __forceinline__ void row_scatter(const Rows &R, int64_t b, int64_t j0, int64_t j1, int32_t *cnt) {
  const int lane = threadIdx.x & 31;
  for (int64_t c0 = j0; c0 < j1; c0 += 32) {
    const int64_t j = c0 + lane;
    const bool valid = j < j1;
    const int32_t w = valid ? R.colidx[j] : 0;
    const int key = valid ? (int)R.lab[w] : -1;
    const unsigned same = __match_any_sync(0xffffffffu, key);
    if (valid) R.col_l[b + cnt[key] + __popc(same & lanes_below())] = w;
    __syncwarp();
    if (valid && lane == __ffs(same) - 1) cnt[key] += __popc(same);
    __syncwarp();
  }
}

template <bool LAB>
__global__ void __launch_bounds__(32 * kRowWarps) rows_kernel(const Rows R) {
  __shared__ int32_t cnt_s[kRowWarps][kSegLabels];
  __shared__ unsigned max_s[kRowWarps];
  __shared__ int32_t long_s[32 * kRowWarps];
  __shared__ int nlong;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  int32_t *cnt = cnt_s[wib];
  // this CTA's rows: blockIdx.x + k * gridDim.x
  for (int64_t v = blockIdx.x + (int64_t)wib * gridDim.x; v < R.n; v += (int64_t)kRowWarps * gridDim.x) {
    const int64_t b = R.rowptr[v], e = R.rowptr[v + 1];
    if (e - b > kLongRow) continue;
    if (LAB && lane < kSegLabels) cnt[lane] = 0;
    __syncwarp();
    const unsigned m = __reduce_max_sync(0xffffffffu, row_first<LAB>(R, (int32_t)v, b, e, b, e, cnt));
    if (lane == 0) R.maxnd[v] = (int32_t)m - 1;
    if (LAB) {
      const int32_t c = lane < R.nl ? cnt[lane] : 0;
      int32_t incl = c;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int32_t t = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += t;
      }
      if (lane <= R.nl) R.loff[v * (R.nl + 1) + lane] = incl - c;  // lane nl: the row length
      __syncwarp();
      if (lane < R.nl) cnt[lane] = incl - c;  // scatter cursors
      __syncwarp();
      row_scatter(R, b, b, e, cnt);
      __syncwarp();
    }
  }
  for (int64_t k0 = 0; blockIdx.x + k0 * gridDim.x < R.n; k0 += 32 * kRowWarps) {
    __syncthreads();
    if (threadIdx.x == 0) nlong = 0;
    __syncthreads();
    const int64_t v = blockIdx.x + (k0 + threadIdx.x) * gridDim.x;
    if (v < R.n && R.rowptr[v + 1] - R.rowptr[v] > kLongRow) long_s[atomicAdd(&nlong, 1)] = (int32_t)v;
    __syncthreads();
    for (int k = 0; k < nlong; ++k) {
      const int64_t u = long_s[k];
      const int64_t b = R.rowptr[u], e = R.rowptr[u + 1];
      const int64_t part = ((e - b + kRowWarps - 1) / kRowWarps + 31) & ~(int64_t)31;
      const int64_t j0 = min(e, b + wib * part), j1 = min(e, j0 + part);
      if (LAB && lane < kSegLabels) cnt[lane] = 0;
      __syncwarp();
      const unsigned m = __reduce_max_sync(0xffffffffu, row_first<LAB>(R, (int32_t)u, b, e, j0, j1, cnt));
      if (lane == 0) max_s[wib] = m;
      __syncthreads();
      if (threadIdx.x == 0) {
        unsigned all = 0;
        for (int w = 0; w < kRowWarps; ++w) all = max(all, max_s[w]);
        R.maxnd[u] = (int32_t)all - 1;
      }
      if (LAB) {
        if (threadIdx.x == 0) {  // every warp's first place per label, label by label
          int32_t run = 0;
          for (int l = 0; l < R.nl; ++l) {
            R.loff[u * (R.nl + 1) + l] = run;
            for (int w = 0; w < kRowWarps; ++w) {
              const int32_t c = cnt_s[w][l];
              cnt_s[w][l] = run;
              run += c;
            }
          }
          R.loff[u * (R.nl + 1) + R.nl] = run;
        }
        __syncthreads();
        row_scatter(R, b, j0, j1, cnt);
      }
      __syncthreads();
    }
  }
}

// One warp per tile of `tile` consecutive edge ids: the number of the
// tile's edges with each group key nl * label(src) + label(dst), written
// key-major (hist[key * ntiles + tile]) so that one exclusive scan gives every
// (key, tile) its first position in the label index.
__global__ void edge_hist_kernel(const int32_t *__restrict__ src, const int32_t *__restrict__ colidx,
                                 const uint8_t *__restrict__ lab, int64_t nedges, int64_t tile, int nl,
                                 int32_t ntiles, int32_t *__restrict__ hist) {
  __shared__ int32_t cnt_s[kBuildWarps][kSegLabels * kSegLabels];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  int32_t *cnt = cnt_s[wib];
  const int G = nl * nl;
  const int64_t warps = (int64_t)gridDim.x * kBuildWarps;
  for (int64_t t = (int64_t)blockIdx.x * kBuildWarps + wib; t < ntiles; t += warps) {
    for (int k = lane; k < G; k += 32) cnt[k] = 0;
    __syncwarp();
    const int64_t b = t * tile, e = b + tile < nedges ? b + tile : nedges;
    for (int64_t c0 = b; c0 < e; c0 += 32) {
      const int64_t j = c0 + lane;
      const bool valid = j < e;
      const int key = valid ? (int)lab[src[j]] * nl + (int)lab[colidx[j]] : -1;
      const unsigned m = __match_any_sync(0xffffffffu, key);
      if (valid && lane == __ffs(m) - 1) cnt[key] += __popc(m);
      __syncwarp();
    }
    for (int k = lane; k < G; k += 32) hist[(int64_t)k * ntiles + t] = cnt[k];
    __syncwarp();
  }
}

// One CTA of 1024 threads: exclusive scan of the histogram in place, 4096
// entries at a time (four per thread, coalesced, then a scan of the warps'
// sums), and the group offsets goff[key] (goff[G] = the edge count).  125 000
// entries take 0.06 ms; each thread on a run of its own, as before, 0.22 ms.
__global__ void __launch_bounds__(1024) index_scan_kernel(int32_t *__restrict__ a, int64_t N, int G,
                                                          int32_t ntiles, int64_t nedges,
                                                          int64_t *__restrict__ goff) {
  __shared__ int32_t sums[32];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  int32_t carry = 0;  // edge ids fit 31 bits on labeled graphs
  for (int64_t i0 = 0; i0 < N; i0 += 4096) {
    const int64_t i = i0 + 4 * t;
    int32_t x[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) x[k] = i + k < N ? a[i + k] : 0;
    const int32_t mine = x[0] + x[1] + x[2] + x[3];
    int32_t incl = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int32_t u = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += u;
    }
    if (lane == 31) sums[w] = incl;
    __syncthreads();
    const int32_t s = sums[lane];
    int32_t all = s;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int32_t u = __shfl_up_sync(0xffffffffu, all, d);
      if (lane >= d) all += u;
    }
    int32_t run = carry + __shfl_sync(0xffffffffu, all - s, w) + incl - mine;
    carry += __shfl_sync(0xffffffffu, all, 31);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (i + k < N) a[i + k] = run;
      run += x[k];
    }
    __syncthreads();
  }
  for (int k = t; k < G; k += 1024) goff[k] = a[(int64_t)k * ntiles];
  if (t == 0) goff[G] = nedges;
}

// One warp per tile: every edge id to its place in the label index, from the
// scanned (key, tile) starts, in edge-id order within each key.
__global__ void edge_scatter_kernel(const int32_t *__restrict__ src, const int32_t *__restrict__ colidx,
                                    const uint8_t *__restrict__ lab, int64_t nedges, int64_t tile, int nl,
                                    int32_t ntiles, const int32_t *__restrict__ start,
                                    int32_t *__restrict__ perm) {
  __shared__ int32_t cur_s[kBuildWarps][kSegLabels * kSegLabels];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  int32_t *cur = cur_s[wib];
  const int G = nl * nl;
  const int64_t warps = (int64_t)gridDim.x * kBuildWarps;
  for (int64_t t = (int64_t)blockIdx.x * kBuildWarps + wib; t < ntiles; t += warps) {
    for (int k = lane; k < G; k += 32) cur[k] = start[(int64_t)k * ntiles + t];
    __syncwarp();
    const int64_t b = t * tile, e = b + tile < nedges ? b + tile : nedges;
    for (int64_t c0 = b; c0 < e; c0 += 32) {
      const int64_t j = c0 + lane;
      const bool valid = j < e;
      const int key = valid ? (int)lab[src[j]] * nl + (int)lab[colidx[j]] : -1;
      const unsigned m = __match_any_sync(0xffffffffu, key);
      if (valid) perm[cur[key] + __popc(m & lanes_below())] = (int32_t)j;
      __syncwarp();
      if (valid && lane == __ffs(m) - 1) cur[key] += __popc(m);
      __syncwarp();
    }
  }
}

// Report a failed CUDA call and clear the runtime's last-error slot, so the
// error cannot resurface in a later launch check.
int cuda_fail(cudaError_t e, const char *what) {
  (void)cudaGetLastError();
  return fail(TDFS_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

}  // namespace

namespace {

int run_rows(const Rows &R, int64_t nedges, cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  if (R.hash) {
    e = cudaMemsetAsync(R.hash, 0xff, 4 * kBucket * (size_t)row_table_buckets(R.n, nedges), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(R.loops, 0, sizeof(int32_t), st);
  }
  if (e == cudaSuccess && R.n > 0) {
    (void)cudaGetLastError();  // the check below must see this launch's error only
    const int blocks = (int)std::min<int64_t>((R.n + kRowWarps - 1) / kRowWarps, 148 * 4);
    if (R.lab) rows_kernel<true><<<blocks, 32 * kRowWarps, 0, st>>>(R);
    else rows_kernel<false><<<blocks, 32 * kRowWarps, 0, st>>>(R);
    e = cudaGetLastError();
  }
  return e == cudaSuccess ? TDFS_OK : cuda_fail(e, "graph preparation kernels");
}

}  // namespace

// Derived per-graph arrays into caller-provided device memory, no allocation:
// edge -> source, neighbour-degree maxima and (when labels is not null) 8-bit
// labels.  *bad becomes nonzero when a label lies outside [0, 254].
int prepare_graph_arrays(const int64_t *rowptr, const int32_t *colidx, int32_t n, int64_t nedges,
                         const int32_t *labels, int32_t *src, int32_t *maxnd, uint8_t *label8, int32_t *bad,
                         int32_t *hash, int32_t *loops, cudaStream_t st) {
  const Rows R{rowptr, colidx, n, src, maxnd, hash, loops, nullptr, 0, nullptr, nullptr};
  const int rc = run_rows(R, nedges, st);
  if (rc || !labels || n <= 0) return rc;
  narrow_labels_kernel<<<148 * 4, 256, 0, st>>>(labels, n, label8, bad);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? TDFS_OK : cuda_fail(e, "graph preparation kernels");
}

namespace {

// ---- launch workspaces, pooled per device ---------------------------------
std::mutex g_pool_mu;
std::vector<Workspace *> g_pool;        // idle workspaces (any device)
constexpr int kIdlePerDevice = 4;       // idle workspaces kept per device; more are freed

void free_workspace(Workspace *w) {
  release_graphs(w);
  cudaFree(w->ctl);
  cudaFreeHost(w->htab);
  cudaFree(w->big);
  if (w->gstream) cudaStreamDestroy(static_cast<cudaStream_t>(w->gstream));
  for (void *e : w->ev)
    if (e) cudaEventDestroy(static_cast<cudaEvent_t>(e));
  delete w;
}

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

bool reclaim_memory(int device, tdfs_graph *self);

}  // namespace

int acquire_workspace(tdfs_graph *g) {
  if (g->ws) return TDFS_OK;
  Workspace *w = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_pool_mu);
    for (size_t i = 0; i < g_pool.size(); ++i)
      if (g_pool[i]->device == g->device) {
        w = g_pool[i];
        g_pool.erase(g_pool.begin() + (long)i);
        break;
      }
  }
  if (!w) {
    // one device allocation (control block, ring, slot table) and one pinned
    // host allocation (staging copies of the slot table and control block)
    const size_t o_queue = align256(sizeof(RunCtl));
    const size_t o_tab = o_queue + align256(sizeof(SplitUnit) * kQueueCap + sizeof(QueueHdr));
    const size_t dev_bytes = o_tab + align256(sizeof(SlotTable));
    const size_t o_hctl = align256(sizeof(SlotTable));
    w = new Workspace{};
    w->device = g->device;
    char *d = nullptr, *h = nullptr;
    cudaError_t e = cudaMalloc(&d, dev_bytes);
    if (e == cudaErrorMemoryAllocation) {
      (void)cudaGetLastError();
      if (reclaim_memory(g->device, g)) e = cudaMalloc(&d, dev_bytes);
    }
    if (e == cudaSuccess) {
      e = cudaMallocHost(&h, o_hctl + sizeof(RunCtl));
      if (e != cudaSuccess) cudaFree(d);
    }
    if (e != cudaSuccess) {
      delete w;
      return cuda_fail(e, "launch workspace");
    }
    w->ctl = reinterpret_cast<RunCtl *>(d);
    w->queue = reinterpret_cast<SplitUnit *>(d + o_queue);
    w->tab = reinterpret_cast<SlotTable *>(d + o_tab);
    w->htab = reinterpret_cast<SlotTable *>(h);
    w->hctl = reinterpret_cast<RunCtl *>(h + o_hctl);
  }
  g->ws = w;
  g->ctl = w->ctl;
  g->queue = w->queue;
  g->tab = w->tab;
  g->htab = w->htab;
  g->hctl = w->hctl;
  return TDFS_OK;
}

namespace {

void release_workspace(tdfs_graph *g) {
  Workspace *w = g->ws;
  if (!w) return;
  g->ws = nullptr;
  g->ctl = nullptr;
  g->queue = nullptr;
  g->tab = nullptr;
  g->htab = nullptr;
  g->hctl = nullptr;
  std::lock_guard<std::mutex> lk(g_pool_mu);
  int idle = 0;
  for (Workspace *x : g_pool) idle += x->device == w->device;
  if (idle < kIdlePerDevice) g_pool.insert(g_pool.end(), 1, w);
  else free_workspace(w);
}

}  // namespace

namespace {

// ---- cached allocations ----------------------------------------------------
// A freed graph's device block and pinned staging block are kept for the next
// upload, so a create/free cycle of a small graph pays no cudaMalloc,
// cudaMallocHost or cudaFree (each costs more than the rest of its upload).
class BlockCache {
 public:
  BlockCache(bool pinned, size_t cap) : pinned_(pinned), cap_(cap) {}

  // A block of at least `need` bytes for `device` (the current device):
  // the smallest idle one within twice that, else a new allocation (after
  // returning this device's idle blocks when memory is short).
  cudaError_t take(int device, size_t need, void **p, size_t *bytes) {
    need = (need + kGrain - 1) & ~(kGrain - 1);
    {
      std::lock_guard<std::mutex> lk(mu_);
      int best = -1;
      for (size_t i = 0; i < idle_.size(); ++i) {
        const Block &b = idle_[i];
        if (b.device == device && b.bytes >= need && b.bytes <= 2 * need &&
            (best < 0 || b.bytes < idle_[(size_t)best].bytes))
          best = (int)i;
      }
      if (best >= 0) {
        *p = idle_[(size_t)best].p;
        *bytes = idle_[(size_t)best].bytes;
        idle_bytes_ -= *bytes;
        idle_.erase(idle_.begin() + best);
        return cudaSuccess;
      }
    }
    cudaError_t e = alloc(p, need);
    if (e == cudaErrorMemoryAllocation) {
      (void)cudaGetLastError();
      drop(device);
      e = alloc(p, need);
    }
    if (e == cudaSuccess) *bytes = need;
    return e;
  }

  // Keep a block for reuse, in the place of the ones idle the longest where
  // the cache is full (blocks of sizes no longer asked for would otherwise
  // make every create and free of a graph go to the driver); a block beyond
  // the byte cap is freed.
  void give(int device, void *p, size_t bytes) {
    if (!p) return;
    std::vector<void *> out;
    if (bytes > cap_) {
      out.push_back(p);
    } else {
      std::lock_guard<std::mutex> lk(mu_);
      int mine = 0;
      for (const Block &b : idle_) mine += b.device == device;
      for (size_t i = 0; i < idle_.size() && (mine >= kPerDevice || idle_bytes_ + bytes > cap_);) {
        if (idle_bytes_ + bytes > cap_ || idle_[i].device == device) {
          mine -= idle_[i].device == device;
          idle_bytes_ -= idle_[i].bytes;
          out.push_back(idle_[i].p);
          idle_.erase(idle_.begin() + (long)i);
        } else {
          ++i;
        }
      }
      idle_.push_back(Block{device, bytes, p});
      idle_bytes_ += bytes;
    }
    for (void *x : out) release(x);
  }

  // Free this device's idle blocks; false when there were none.
  bool drop(int device) {
    std::vector<Block> mine;
    {
      std::lock_guard<std::mutex> lk(mu_);
      for (size_t i = 0; i < idle_.size();) {
        if (idle_[i].device == device) {
          idle_bytes_ -= idle_[i].bytes;
          mine.push_back(idle_[i]);
          idle_.erase(idle_.begin() + (long)i);
        } else {
          ++i;
        }
      }
    }
    for (const Block &b : mine) release(b.p);
    return !mine.empty();
  }

 private:
  struct Block {
    int device;
    size_t bytes;
    void *p;
  };
  static constexpr size_t kGrain = size_t(1) << 20;  // sizes rounded to 1 MiB, so re-uploads fit exactly
  static constexpr int kPerDevice = 8;     // a graph's arrays and tables are a block each

  cudaError_t alloc(void **p, size_t bytes) { return pinned_ ? cudaMallocHost(p, bytes) : cudaMalloc(p, bytes); }
  void release(void *p) {
    if (pinned_) cudaFreeHost(p); else cudaFree(p);
  }
  std::mutex mu_;
  std::vector<Block> idle_;
  size_t idle_bytes_ = 0;
  const bool pinned_;
  const size_t cap_;
};

// never destroyed: the blocks may outlive the CUDA runtime at process exit
BlockCache &device_blocks() {
  static BlockCache *c = new BlockCache(false, size_t(512) << 20);
  return *c;
}
BlockCache &pinned_blocks() {
  static BlockCache *c = new BlockCache(true, size_t(256) << 20);
  return *c;
}

// ---- memory that can be given up ---------------------------------------------
std::mutex g_tables_mu;
std::vector<tdfs_graph *> g_with_tables;  // every graph that holds row membership tables

size_t table_bytes(int64_t n, int64_t nedges) { return 4 * kBucket * (size_t)row_table_buckets(n, nedges); }

void forget_tables(tdfs_graph *g) {  // (with g_tables_mu)
  const auto it = std::find(g_with_tables.begin(), g_with_tables.end(), g);
  if (it != g_with_tables.end()) g_with_tables.erase(it);
}

// Device memory is short: free what only makes counts faster -- cached blocks,
// idle workspaces' level-2 buffers and the row membership tables of graphs
// that no launch is reading (and of `self`, whose tables_mu the caller holds).
// True when there was any.
bool reclaim_memory(int device, tdfs_graph *self) {
  bool any = device_blocks().drop(device);
  {
    std::lock_guard<std::mutex> lk(g_pool_mu);
    for (Workspace *w : g_pool)
      if (w->device == device && w->big) {
        cudaFree(w->big);
        w->big = nullptr;
        w->big_bytes = 0;
        any = true;
      }
  }
  std::lock_guard<std::mutex> lk(g_tables_mu);
  for (tdfs_graph *g : std::vector<tdfs_graph *>(g_with_tables)) {
    if (g->device != device || (g != self && !g->tables_mu->try_lock())) continue;
    cudaFree(g->hash);
    g->hash = nullptr;
    g->bytes -= table_bytes(g->n, g->nedges);
    forget_tables(g);
    if (g != self) g->tables_mu->unlock();
    any = true;
  }
  return any;
}

int host_threads() {
  const unsigned t = std::thread::hardware_concurrency();
  return t ? (int)std::min(t, 32u) : 4;
}

// The label index and the label rows, written by the host straight into the
// pinned staging block they are uploaded from:
//  * perm: a stable counting sort of the edge ids by the group key
//    nl * label(src) + label(dst), with its group offsets `off`;
//  * with nlab > 0 (at most kSegLabels labels, nlab == nl): col_l, every row
//    re-sorted by (label, id), and loff, each row's segment starts relative
//    to the row start (nlab + 1 per vertex).
// Two passes over the edges (count, then scatter).  Large graphs split the
// rows over host threads in contiguous runs of about equal edge counts; each
// run scatters from its own group offsets, so the order stays stable.
void build_label_arrays(int64_t n, int64_t nedges, const int64_t *rowptr, const int32_t *colidx, const uint8_t *lab,
                        int nl, int nlab, int32_t *perm, int32_t *col_l, int32_t *loff, std::vector<int64_t> &off) {
  const int G = nl * nl;
  const int T = nedges < (int64_t(1) << 20) ? 1 : (int)std::min<int64_t>(host_threads(), nedges >> 19);
  std::vector<int64_t> rb((size_t)T + 1, 0);
  rb[(size_t)T] = n;
  for (int t = 1; t < T; ++t) {
    const int64_t want = nedges * t / T;
    rb[(size_t)t] = std::max(rb[(size_t)t - 1], (int64_t)(std::upper_bound(rowptr, rowptr + n + 1, want) - rowptr) - 1);
  }
  std::vector<int64_t> cnt((size_t)T * G, 0);  // per run and group: edges, then the run's scatter cursor
  auto count_run = [&](int t) {
    int64_t *c = cnt.data() + (size_t)t * G;
    for (int64_t v = rb[(size_t)t]; v < rb[(size_t)t + 1]; ++v) {
      int64_t *cv = c + (size_t)lab[v] * nl;
      if (nlab) {
        int32_t k[kSegLabels] = {0};
        for (int64_t j = rowptr[v]; j < rowptr[v + 1]; ++j) ++k[lab[colidx[j]]];
        int32_t *o = loff + (size_t)v * (nlab + 1);
        o[0] = 0;
        for (int l = 0; l < nlab; ++l) {
          o[l + 1] = o[l] + k[l];
          cv[l] += k[l];
        }
      } else {
        for (int64_t j = rowptr[v]; j < rowptr[v + 1]; ++j) ++cv[lab[colidx[j]]];
      }
    }
  };
  auto scatter_run = [&](int t) {
    int64_t *at = cnt.data() + (size_t)t * G;
    for (int64_t v = rb[(size_t)t]; v < rb[(size_t)t + 1]; ++v) {
      int64_t *av = at + (size_t)lab[v] * nl;
      const int64_t b = rowptr[v], e = rowptr[v + 1];
      if (nlab) {
        int32_t k[kSegLabels];
        const int32_t *o = loff + (size_t)v * (nlab + 1);
        for (int l = 0; l < nlab; ++l) k[l] = o[l];
        for (int64_t j = b; j < e; ++j) {
          const int32_t x = colidx[j];
          const int l = lab[x];
          perm[av[l]++] = (int32_t)j;
          col_l[b + k[l]++] = x;
        }
      } else {
        for (int64_t j = b; j < e; ++j) perm[av[lab[colidx[j]]]++] = (int32_t)j;
      }
    }
  };
  auto run = [&](auto &&f) {
    if (T == 1) {
      f(0);
      return;
    }
    std::vector<std::thread> th;
    for (int t = 0; t < T; ++t) th.emplace_back(f, t);
    for (auto &x : th) x.join();
  };
  run(count_run);
  off.assign((size_t)G + 1, 0);
  for (int gk = 0; gk < G; ++gk) {
    int64_t s = off[(size_t)gk];
    for (int t = 0; t < T; ++t) {  // run t scatters group gk from here
      const int64_t c = cnt[(size_t)t * G + gk];
      cnt[(size_t)t * G + gk] = s;
      s += c;
    }
    off[(size_t)gk + 1] = s;
  }
  run(scatter_run);
}

}  // namespace

// The graph arrays live in one device allocation, each part starting on a
// 256-byte boundary:
//   rowptr int64[n+1] | colidx int32[E + kColPad] | src int32[E] | maxnd int32[n]
//   | label uint8[n] | lperm int32[E] | colidx_l int32[E + kColPad] | loff int32[n (nlab+1)]
//   | scratch of the label index sort | self-loop flag and check result
// and the row membership tables in another, which the graph can lose.
// The device derives everything but the narrowed labels; with more labels than
// kSegLabels the host sorts the label index into a pinned staging block, laid
// out the same way, while the copies and kernels queued before it run.  One
// synchronisation at the end.
int graph_upload(int64_t n, int64_t nedges, const int64_t *rowptr, const int32_t *colidx, const int32_t *labels,
                 int device, int32_t max_degree, bool check, tdfs_graph **out) {
  int ndev = 0;
  // where the device cannot check the CSR the host does, so that what is wrong
  // with it is still what the caller is told
  auto checked = [&](int rc) {
    const std::string msg = tdfs_last_error();
    if (check)
      if (const int bad = validate_csr(n, nedges, rowptr, colidx, nullptr)) return bad;
    return fail(rc, "%s", msg.c_str());
  };
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    (void)cudaGetLastError();
    return checked(fail(TDFS_ERR_CUDA, "no CUDA device visible (the tdfs engine has no CPU path)"));
  }
  if (device < 0 || device >= ndev) return checked(fail(TDFS_ERR_ARG, "device %d out of range", device));
  int nl = 0;
  if (labels) {
    int32_t least = 0, most = -1;
    for (int64_t i = 0; i < n; ++i) {  // (no early exit: the loop vectorises)
      least = std::min(least, labels[i]);
      most = std::max(most, labels[i]);
    }
    if (least < 0 || most > 254)
      return checked(fail(TDFS_ERR_FORMAT, "vertex labels must lie in [0, 254] for the device label array"));
    nl = most + 1;
    if (nedges > INT32_MAX)
      return checked(fail(TDFS_ERR_CAPACITY, "labeled graphs hold at most 2^31 - 1 directed edges"));
  }
  // label-partitioned rows for graphs with at most kSegLabels labels
  const int nlab = labels && nl <= kSegLabels ? nl : 0;
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
  static_assert(kColPad % 4 == 0, "padding keeps 16-byte loads aligned");
  const size_t o_col = align256(sizeof(int64_t) * (size_t)(n + 1));
  const size_t o_src = o_col + align256(sizeof(int32_t) * (size_t)(nedges + kColPad));
  const size_t o_maxnd = o_src + align256(sizeof(int32_t) * (size_t)(nedges ? nedges : 1));
  const size_t o_label = o_maxnd + align256(sizeof(int32_t) * (size_t)(n ? n : 1));
  const size_t o_perm = o_label + align256((size_t)(labels && n ? n : 1));
  const size_t o_coll = o_perm + align256(sizeof(int32_t) * (size_t)(labels && nedges ? nedges : 1));
  const size_t o_loff = o_coll + align256(sizeof(int32_t) * (size_t)(nlab ? nedges + kColPad : 1));
  const size_t nloff = nlab ? (size_t)n * (size_t)(nlab + 1) : 0;
  // with label rows the label arrays are built on the device, which needs
  // scratch for the index sort: the (key, tile) histogram and the group
  // offsets; otherwise the host builds them into the staging block
  const bool dev_build = nlab > 0;
  const int G = nl * nl;
  const int64_t tile = tile_edges(nedges);
  const int32_t ntiles = dev_build ? (int32_t)((nedges + tile - 1) / tile) : 0;
  const size_t o_hist = o_loff + align256(sizeof(int32_t) * (nloff ? nloff : 1));
  const size_t o_goff = o_hist + align256(sizeof(int32_t) * (size_t)(dev_build && ntiles ? (int64_t)G * ntiles : 1));
  const size_t total = dev_build ? o_goff + align256(sizeof(int64_t) * (size_t)(G + 1)) : o_hist;
  void *arrays = nullptr, *stage = nullptr, *hash = nullptr;
  size_t array_bytes = 0, stage_bytes = 0, hash_bytes = 0;
  e = device_blocks().take(device, total + 256, &arrays, &array_bytes);
  if (e == cudaErrorMemoryAllocation) {
    (void)cudaGetLastError();
    if (reclaim_memory(device, nullptr)) e = device_blocks().take(device, total + 256, &arrays, &array_bytes);
  }
  if (e != cudaSuccess) return checked(cuda_fail(e, "graph arrays"));
  // the row membership tables, where the flat kernel can use them and the
  // device has room; without them every plan runs on the DFS kernel
  if (row_table_buckets(n, nedges) <= (int64_t)UINT32_MAX &&
      device_blocks().take(device, table_bytes(n, nedges), &hash, &hash_bytes) != cudaSuccess) {
    (void)cudaGetLastError();
    hash = nullptr;
  }
  if (labels) {
    e = pinned_blocks().take(device, dev_build ? (size_t)std::max<int64_t>(n, 1) : total - o_label, &stage,
                             &stage_bytes);
    if (e != cudaSuccess) {
      device_blocks().give(device, arrays, array_bytes);
      device_blocks().give(device, hash, hash_bytes);
      return checked(cuda_fail(e, "pinned staging for the label arrays"));
    }
  }
  char *base = static_cast<char *>(arrays);
  auto *g = new tdfs_graph;
  std::memset(g, 0, sizeof *g);
  g->device = device;
  g->n = n;
  g->nedges = nedges;
  g->max_degree = max_degree;
  g->labeled = labels != nullptr;
  g->arrays = arrays;
  g->array_bytes = array_bytes;
  g->staging = stage;
  g->staging_bytes = stage_bytes;
  g->rowptr = reinterpret_cast<int64_t *>(base);
  g->colidx = reinterpret_cast<int32_t *>(base + o_col);
  g->src = reinterpret_cast<int32_t *>(base + o_src);
  g->maxnd = reinterpret_cast<int32_t *>(base + o_maxnd);
  g->label = labels ? reinterpret_cast<uint8_t *>(base + o_label) : nullptr;
  g->lperm = labels ? reinterpret_cast<int32_t *>(base + o_perm) : nullptr;
  g->colidx_l = nlab ? reinterpret_cast<int32_t *>(base + o_coll) : nullptr;
  g->loff = nlab ? reinterpret_cast<int32_t *>(base + o_loff) : nullptr;
  g->nlab = nlab;
  g->hash = static_cast<int32_t *>(hash);
  g->hash_bytes = hash_bytes;
  g->loops = reinterpret_cast<int32_t *>(base + total);
  g->bytes = (dev_build ? o_hist : total) + (hash ? table_bytes(n, nedges) : 0);  // the scratch is not part of the graph
  const cudaStream_t st = cudaStreamPerThread;
  e = cudaMemcpyAsync(g->rowptr, rowptr, sizeof(int64_t) * (n + 1), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess && nedges)
    e = cudaMemcpyAsync(g->colidx, colidx, sizeof(int32_t) * nedges, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(g->colidx + nedges, 0x7f, sizeof(int32_t) * kColPad, st);
  auto *lab8 = static_cast<uint8_t *>(stage);
  CsrCheck ck{0, max_degree};
  if (e == cudaSuccess && check) {
    // nothing below may read rows that break the rules: wait for the verdict
    // (and narrow the labels meanwhile)
    auto *dck = reinterpret_cast<CsrCheck *>(base + total + 128);
    e = cudaMemsetAsync(dck, 0, sizeof *dck, st);
    if (e == cudaSuccess) {
      (void)cudaGetLastError();  // the check below must see this launch's error only
      const int blocks = (int)std::min<int64_t>((std::max(n, nedges) + 255) / 256 + 1, 148 * 8);
      check_csr_kernel<<<blocks, 256, 0, st>>>(g->rowptr, g->colidx, n, nedges, dck);
      e = cudaGetLastError();
    }
    if (labels)
      for (int64_t i = 0; i < n; ++i) lab8[i] = (uint8_t)labels[i];
    if (e == cudaSuccess) e = cudaMemcpyAsync(&ck, dck, sizeof ck, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess && ck.bad) {
      pinned_blocks().give(device, stage, stage_bytes);
      device_blocks().give(device, arrays, array_bytes);
      device_blocks().give(device, hash, hash_bytes);
      delete g;
      if (const int bad = validate_csr(n, nedges, rowptr, colidx, nullptr)) return bad;
      return fail(TDFS_ERR_FORMAT, "the rows changed while they were read");
    }
    g->max_degree = ck.max_degree;
  } else if (labels) {
    for (int64_t i = 0; i < n; ++i) lab8[i] = (uint8_t)labels[i];
  }
  if (g->max_degree > kFlatMaxDegree && g->hash) {  // the flat kernel's positions would not fit 32 bits
    device_blocks().give(device, g->hash, g->hash_bytes);
    g->hash = nullptr;
    g->bytes -= table_bytes(n, nedges);
  }
  Rows R{g->rowptr, g->colidx, (int32_t)n, g->src, g->maxnd, g->hash, g->loops, nullptr, 0, nullptr, nullptr};
  if (e == cudaSuccess && !nlab && run_rows(R, nedges, st) != TDFS_OK) e = cudaErrorUnknown;
  std::unique_ptr<LabelIndex> lindex;
  if (e == cudaSuccess && labels) {
    char *h = static_cast<char *>(stage);
    lindex.reset(new LabelIndex);
    lindex->nl = nl;
    lindex->nedges = nedges;
    if (dev_build) {
      // label rows and label index by the kernels above; the host keeps the
      // group offsets
      lindex->dev_perm = g->lperm;
      lindex->off.assign((size_t)G + 1, 0);
      e = cudaMemcpyAsync(g->label, lab8, (size_t)n, cudaMemcpyHostToDevice, st);
      if (e == cudaSuccess) e = cudaMemsetAsync(g->colidx_l + nedges, 0x7f, sizeof(int32_t) * kColPad, st);
      R.lab = g->label;
      R.nl = nl;
      R.col_l = g->colidx_l;
      R.loff = g->loff;
      if (e == cudaSuccess && run_rows(R, nedges, st) != TDFS_OK) e = cudaErrorUnknown;
      if (e == cudaSuccess && ntiles > 0) {
        auto *hist = reinterpret_cast<int32_t *>(base + o_hist);
        auto *goff = reinterpret_cast<int64_t *>(base + o_goff);
        const int blocks = (int)std::min<int64_t>((ntiles + kBuildWarps - 1) / kBuildWarps, 148 * 16);
        edge_hist_kernel<<<blocks, 32 * kBuildWarps, 0, st>>>(g->src, g->colidx, g->label, nedges, tile, nl,
                                                             ntiles, hist);
        index_scan_kernel<<<1, 1024, 0, st>>>(hist, (int64_t)G * ntiles, G, ntiles, nedges, goff);
        edge_scatter_kernel<<<blocks, 32 * kBuildWarps, 0, st>>>(g->src, g->colidx, g->label, nedges, tile, nl,
                                                                ntiles, hist, g->lperm);
        e = cudaGetLastError();
        if (e == cudaSuccess)
          e = cudaMemcpyAsync(lindex->off.data(), goff, sizeof(int64_t) * (size_t)(G + 1), cudaMemcpyDeviceToHost,
                              st);
      }
    } else {
      // while the device copies and preprocesses the CSR
      auto *perm = reinterpret_cast<int32_t *>(h + (o_perm - o_label));
      auto *col_l = reinterpret_cast<int32_t *>(h + (o_coll - o_label));
      auto *loff = reinterpret_cast<int32_t *>(h + (o_loff - o_label));
      lindex->perm = perm;
      build_label_arrays(n, nedges, rowptr, colidx, lab8, nl, nlab, perm, col_l, loff, lindex->off);
      if (nlab) std::memset(col_l + nedges, 0x7f, sizeof(int32_t) * kColPad);
      e = cudaMemcpyAsync(base + o_label, h, total - o_label, cudaMemcpyHostToDevice, st);
    }
  }
  // the staging block and the caller's arrays must outlive the copies
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    const int rc = cuda_fail(e, "graph upload");
    cudaStreamSynchronize(st);
    pinned_blocks().give(device, stage, stage_bytes);
    device_blocks().give(device, arrays, array_bytes);
    device_blocks().give(device, g->hash, g->hash_bytes);
    delete g;
    return rc;
  }
  g->lindex = lindex.release();
  g->tables_mu = new std::mutex;
  if (g->hash) {
    std::lock_guard<std::mutex> lk(g_tables_mu);
    g_with_tables.push_back(g);
  }
  *out = g;
  return TDFS_OK;
}

bool label_range(LabelIndex &x, int l0, int l1, int64_t eb, int64_t ee, int64_t *b, int64_t *e) {
  *b = *e = 0;
  if (l0 < 0 || l0 >= x.nl || l1 < 0 || l1 >= x.nl) return true;  // a label no vertex has: nothing to do
  const size_t key = (size_t)l0 * (size_t)x.nl + (size_t)l1;
  if (eb <= 0 && ee >= x.nedges) {
    *b = x.off[key];
    *e = x.off[key + 1];
    return true;
  }
  std::call_once(x.fetch_once, [&x] {
    if (x.perm || !x.dev_perm) return;
    x.fetched.resize((size_t)x.nedges);
    if (cudaMemcpy(x.fetched.data(), x.dev_perm, sizeof(int32_t) * (size_t)x.nedges, cudaMemcpyDeviceToHost) ==
        cudaSuccess)
      x.perm = x.fetched.data();
    else
      (void)cudaGetLastError();
  });
  if (!x.perm) return false;
  const int32_t *g0 = x.perm + x.off[key], *g1 = x.perm + x.off[key + 1];
  // ids ascend within a group: the edge-id range is a position range
  *b = x.off[key] + (std::lower_bound(g0, g1, (int32_t)std::min<int64_t>(eb, INT32_MAX)) - g0);
  *e = x.off[key] + (std::lower_bound(g0, g1, (int32_t)std::min<int64_t>(ee, INT32_MAX)) - g0);
  if (ee > INT32_MAX) *e = x.off[key + 1];
  return true;
}

void graph_release(tdfs_graph *g) {
  if (!g) return;
  int cur = 0;
  cudaGetDevice(&cur);
  cudaSetDevice(g->device);
  release_workspace(g);
  // the blocks go back to the caches, not to the driver: wait for anything
  // still reading them, as cudaFree would
  cudaDeviceSynchronize();
  {
    std::lock_guard<std::mutex> lk(g_tables_mu);
    forget_tables(g);
  }
  device_blocks().give(g->device, g->arrays, g->array_bytes);
  device_blocks().give(g->device, g->hash, g->hash_bytes);
  pinned_blocks().give(g->device, g->staging, g->staging_bytes);
  delete g->lindex;
  delete g->tables_mu;
  cudaSetDevice(cur);
  delete g;
}

DevGraph graph_view(const tdfs_graph *g) {
  DevGraph v;
  std::memset(static_cast<void *>(&v), 0, sizeof v);  // (views are compared as bytes)
  v.rowptr = g->rowptr;
  v.colidx = g->colidx;
  v.src = g->src;
  v.label = g->label;
  v.maxnd = g->maxnd;
  v.lperm = g->lperm;
  v.colidx_l = g->colidx_l;
  v.loff = g->loff;
  v.hash = g->hash;
  v.loops = g->loops;
  v.nlab = g->nlab;
  v.nedges = g->nedges;
  v.n = (int32_t)g->n;
  v.max_degree = g->max_degree;
  return v;
}

}  // namespace tdfs
