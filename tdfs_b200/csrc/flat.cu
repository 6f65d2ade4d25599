// flat.cu -- the flattened subgraph-counting kernel (design notes in flat.cuh).
// Count semantics follow src/gpu_match.cu:260-1080 as in match.cu; plans come
// in the form flat_plan.cpp derives.
#include <cuda_runtime.h>

#include <climits>
#include <mutex>

#include "flat.cuh"

namespace tdfs {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kTupleMax = kMaxK - 1;   // phi(0..5): the deepest enumerated level is 5
constexpr int kProbeMax = kMaxK - 2;   // lists tested per candidate besides its source
// A tail's block of entries ends before their lists pass this many positions:
// unlike the other scans it is not resumed in the middle, and work is only
// given away between blocks (32 entries with hub lists kept one warp busy for
// 0.4 ms; a labeled power-law batch with such a tail 1.93 -> 1.07 ms; 1024 and
// 16384 positions did the same).
constexpr int kTailSpan = 4096;
constexpr int kLookSteps = 32;         // 64-position steps of a scan between two looks at the idle mask

constexpr int kCntBytes = 7 * 32 * 4;
constexpr int kRangeMin = 4;           // children of one parent given away as a range

// Work given away goes straight to an idle warp: each warp has a mailbox and
// a bit in a grid-wide mask of idle warps.  A busy warp reads 32 words of the
// mask with one load, each lane claims one idle warp by clearing its bit, and
// the entries are spread over all of them.  No two warps meet on a counter,
// as they would on a shared ring (which passed 1.2 units per microsecond
// whatever the demand and left 60-90% of the warps of a power-law launch
// idle), and an idle warp reads its own line only.

struct FlatLevel {
  int32_t next;      // first entry of the block being extended (blocks of 32 entries)
  int32_t end;       // entries [next, end) are left to extend
  int32_t n;         // entries in the buffer (>= end: some may have been given away)
  uint32_t pos;      // positions of the block already done
  int32_t started;   // first entry not yet touched
  int32_t cutp;      // entry whose list the position pos lies inside, or -1
  int32_t hcut, tcut;  // parents whose children here are incomplete at the front / at the end, or -1
  int32_t groups;    // 0: entries came from elsewhere; siblings are not together
};

// Shared by a CTA's warps.
struct FlatCta {
  int32_t poll;    // 1: some idle warp of the CTA is watching FlatCtl::pending
  int32_t done;    // 1: no work is left anywhere
  int32_t all;     // 1: the whole grid has started
  int32_t active;  // busy warps
  int32_t left;    // warps still in the kernel
  long long first; // the CTA's first tickets: [first, first + warps)
  int32_t slot;    // slot whose counts are summed here first, -1 none
  unsigned long long sum, idle_ns, warp_ns;
};

struct alignas(16) FlatSmem {
  FlatPlan plan;
  int32_t slot;                     // slot of `plan`, -1 none
  int32_t cap, levels;              // entries per level and levels held in shared memory
  int32_t low;                      // the first of them: 2, or 3 when level 2 is in global memory
  int32_t rlevel, rlo, rhi;         // entries of level rlevel are extended only in [rlo, rhi]; rlevel 0: no range
  FlatLevel lev[kMaxK];             // levels 1..s
  int4 src[32];                     // per list (lanes with one, in order): address minus its first position (in bytes; x, y)
                                    // and the first row table to test (z first bucket, w bucket count;
                                    // 0 = no test)
  int32_t phi[kTupleMax][32];       // per lane: the partial embedding being extended
  uint2 more[kProbeMax - 1][32];    // per lane: the other row tables to test
  int32_t er[32], ec[32];           // level-1 entries: edges (phi(0), phi(1))
  uint8_t map[32];                  // rank among the lanes with a list -> lane
  int32_t root;                     // level of the entries this warp was given
  unsigned long long t_work;        // globaltimer when the current base work was taken
  unsigned long long idle_total, t_start;  // diagnostics
};

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }
__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}
__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// 1 << d, 0 for d > 31.
__device__ __forceinline__ unsigned bit_at(uint32_t d) {
  unsigned r;
  asm("shl.b32 %0, 1, %1;" : "=r"(r) : "r"(d));  // PTX clamps the shift
  return r;
}

template <bool LAB, bool BIG>
struct Flat {
  const DevGraph &G;
  const FlatCfg &cfg;
  const FlatTable &T;
  const int gid;
  FlatSmem &W;
  FlatCta &C;
  int32_t *X;  // entries: the vertices of every level, then the parents' entries one level up
  unsigned long long count = 0;  // per lane; summed at release
  int lane;

  __device__ Flat(const DevGraph &g, const FlatCfg &c, const FlatTable &t, int warp, FlatSmem &w, FlatCta &cta,
                  unsigned char *bufs)
      : G(g), cfg(c), T(t), gid(warp), W(w), C(cta), X(reinterpret_cast<int32_t *>(bufs)),
        lane(lane_id()) {}

  // Per lane: sizes of the tail's sets (plans with t >= 2 give up the end of
  // their entries for them).
  __device__ __forceinline__ uint32_t *cnt(int u) const {
    return reinterpret_cast<uint32_t *>(reinterpret_cast<unsigned char *>(X) + cfg.entries * 6 - kCntBytes) + 32 * u;
  }
  __device__ __forceinline__ int32_t *big() const { return T.big + (size_t)gid * (kBigBytes / 4); }
  __device__ __forceinline__ int low() const { return BIG ? W.low : 2; }
  __device__ __forceinline__ int32_t *xs(int l) const { return BIG && l < W.low ? big() : X + (l - low()) * W.cap; }
  __device__ __forceinline__ uint16_t *ps(int l) const {
    return BIG && l < W.low ? reinterpret_cast<uint16_t *>(big() + kBigEntries)
                            : reinterpret_cast<uint16_t *>(X + W.cap * W.levels) + (l - low()) * W.cap;
  }
  __device__ __forceinline__ int room(int l) const { return (BIG && l < W.low ? kBigEntries : W.cap) - 64; }
  __device__ __forceinline__ bool segmented() const { return LAB && cfg.segments && G.colidx_l != nullptr; }
  __device__ __forceinline__ const int32_t *lists() const { return segmented() ? G.colidx_l : G.colidx; }

  // Adjacency row of v as candidates of label `lab` are drawn from it: its
  // label segment when the graph has them, else the whole row.
  __device__ __forceinline__ void row(int32_t v, int lab, int64_t &b, uint32_t &len) const {
    const int64_t r = G.rowptr[v];
    if (segmented()) {
      b = r;
      len = 0;
      if (lab < G.nlab) {
        const int32_t *o = G.loff + (int64_t)v * (G.nlab + 1) + lab;
        const int32_t o0 = o[0];
        b = r + o0;
        len = (uint32_t)(o[1] - o0);
      }
    } else {
      b = r;
      len = (uint32_t)(G.rowptr[v + 1] - r);
    }
  }

  // Row v's membership table: false when the row is empty.
  __device__ __forceinline__ bool table(int32_t v, uint32_t &hb, uint32_t &nb) const {
    const int64_t r = G.rowptr[v], e = G.rowptr[v + 1];
    hb = (uint32_t)(row_table_at(r) + v);
    nb = (uint32_t)(row_table_at(e) - row_table_at(r)) + 1;
    return e > r;
  }
  struct Bucket {
    int32_t e[kBucket];
  };
  __device__ __forceinline__ Bucket bucket(uint32_t i) const {
    Bucket q;
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(q.e[0]), "=r"(q.e[1]), "=r"(q.e[2]), "=r"(q.e[3]), "=r"(q.e[4]), "=r"(q.e[5]), "=r"(q.e[6]),
          "=r"(q.e[7])
        : "l"(G.hash + (size_t)i * kBucket));
    return q;
  }
  __device__ __forceinline__ static bool holds(const Bucket &q, int32_t x) {
    bool h = false;
#pragma unroll
    for (int i = 0; i < kBucket; ++i) h |= q.e[i] == x;
    return h;
  }
  // Is x in the table, given its bucket q (offset b)?
  __device__ __forceinline__ bool found(Bucket q, uint32_t hb, uint32_t nb, uint32_t b, int32_t x) const {
    bool h = holds(q, x);
    for (uint32_t t = 1; t < nb && !h && q.e[kBucket - 1] >= 0; ++t) {  // full: it may have overflowed
      b = b + 1 == nb ? 0 : b + 1;
      q = bucket(hb + b);
      h = holds(q, x);
    }
    return h;
  }
  __device__ __forceinline__ bool member(int32_t v, int32_t x) const {
    uint32_t hb, nb;
    if (!table(v, hb, nb)) return false;
    const uint32_t b = __umulhi((uint32_t)x * kRowHash, nb);
    return found(bucket(hb + b), hb, nb, b, x);
  }

  // This lane's partial embedding: entry p of level L and its ancestors, into
  // W.phi.  Returns its ancestor entry at level `dep` (-1 when dep is 0).
  __device__ __forceinline__ int load_tuple(int L, int p, int dep) {
    int e = -1, q = p;
    for (int l = L; l >= 2; --l) {
      if (l == dep) e = q;
      W.phi[l][lane] = xs(l)[q];
      q = ps(l)[q];
    }
    W.phi[0][lane] = W.er[q];
    W.phi[1][lane] = W.ec[q];
    return e;
  }

  // Bounds of the order conditions of st under this lane's embedding.
  __device__ __forceinline__ void bounds(const FlatStep &st, int32_t &lo, int32_t &hi) const {
    lo = -1;
    hi = INT_MAX;
    if (!LAB) {
      for (unsigned m = st.larger; m; m &= m - 1) lo = max(lo, W.phi[__ffs(m) - 1][lane]);
      for (unsigned m = st.less; m; m &= m - 1) hi = min(hi, W.phi[__ffs(m) - 1][lane]);
    }
  }

  // Narrow the ascending range a[b, b + len) to the values in (lo, hi).
  template <typename T>
  __device__ __forceinline__ void trim(const int32_t *a, T &b, int &len, int32_t lo, int32_t hi) const {
    if (len > 0 && a[b] <= lo) {
      int s = 1, e = len;  // a[b + s - 1] <= lo
      while (s < e) {
        const int m = (s + e) >> 1;
        if (a[b + m] <= lo) s = m + 1; else e = m;
      }
      b += s;
      len -= s;
    }
    if (hi < INT_MAX && len > 0 && a[b + len - 1] >= hi) {
      int s = 0, e = len - 1;  // a[b + e] >= hi
      while (s < e) {
        const int m = (s + e) >> 1;
        if (a[b + m] < hi) s = m + 1; else e = m;
      }
      len = s;
    }
  }

  // Set up this lane's candidate scan for st (its embedding: entry p of level
  // L): the source's address, the first row table to test, and the others
  // (W.more).  Returns the number of source positions.
  __device__ int setup_lane(const FlatStep &st, int L, int p, int64_t &base, uint2 &first) {
    const int e = load_tuple(L, p, st.dep);
    // the shortest list is scanned, the others are tested
    uint32_t best = UINT_MAX;
    int64_t gb = 0;
    int tb = 0;
    for (int t = 0; t < st.nbn; ++t) {
      int64_t b;
      uint32_t len;
      row(W.phi[st.bn[t]][lane], st.label, b, len);
      if (len < best) {
        best = len;
        gb = b;
        tb = t;
      }
    }
    int len = (int)best;
    if (len == 0) return 0;
    // or, under reuse, the siblings of the ancestor at level dep, when they
    // are all in its buffer
    bool sib = false;
    int sb = 0;
    const int dep = st.dep;
    if (dep && W.lev[dep].groups) {
      const uint16_t *pp = ps(dep);
      const int me = pp[e];
      const bool later = !LAB && (st.larger >> dep & 1);  // only siblings after e can pass
      if (me != W.lev[dep].tcut && (later || me != W.lev[dep].hcut)) {
        int s = e + 1, t = W.lev[dep].n;
        while (s < t) {
          const int m = (s + t) >> 1;
          if (pp[m] <= me) s = m + 1; else t = m;
        }
        sb = e + 1;
        if (!later) {
          int a = 0, z = e;
          while (a < z) {
            const int m = (a + z) >> 1;
            if (pp[m] < me) a = m + 1; else z = m;
          }
          sb = a;
        }
        if (s - sb <= len) {
          sib = true;
          len = s - sb;
        }
      }
    }
    if (!LAB) {
      int32_t lo, hi;
      bounds(st, lo, hi);
      if (sib) trim(xs(dep), sb, len, lo, hi);
      else trim(lists(), gb, len, lo, hi);
    }
    if (len <= 0) return 0;
    int u = 0;
    const int nt = sib ? st.nsh : st.nbn;
    uint32_t hb0 = 0, nb0 = 0;
    for (int t = 0; t < nt; ++t) {
      if (!sib && t == tb) continue;
      uint32_t hb, nb;
      if (!table(W.phi[sib ? st.bnsh[t] : st.bn[t]][lane], hb, nb)) return 0;
      if (u == 0) {
        hb0 = hb;
        nb0 = nb;
      } else {
        W.more[u - 1][lane] = make_uint2(hb, nb);
      }
      ++u;
    }
    for (u = max(u, 1); u < st.nbn - 1; ++u) W.more[u - 1][lane] = make_uint2(0u, 0u);
    base = reinterpret_cast<int64_t>(sib ? xs(dep) + sb : lists() + gb);
    first = make_uint2(hb0, nb0);
    return len;
  }

  // Entries of level l that no scan has touched.
  __device__ __forceinline__ int untouched(int l) const {
    const FlatLevel &H = W.lev[l];
    return H.end - (H.pos ? H.started : H.next);
  }
  // 32 words of the idle mask, another part of it each time; lanes beyond the
  // grid's words get 0.
  __device__ __forceinline__ unsigned idle_word(int &w) const {
    const unsigned words = (gridDim.x * (blockDim.x >> 5) + 31) >> 5;
    w = (int)(((unsigned)(clock64() >> 6) + (unsigned)(gid * 7 + lane)) % words);
    return lane < words ? *(volatile unsigned *)&T.idle[w] : 0u;
  }
  // May this warp give work away yet (its base work is old enough)?
  __device__ __forceinline__ bool may_give() const {
    return now_ns() - W.t_work >= (unsigned long long)cfg.split_ns;
  }
  __device__ __forceinline__ bool someone_idle() const {
    int w;
    return __any_sync(kFull, idle_word(w) != 0 && may_give());
  }

  // The candidates of st for the block of up to 32 entries at W.lev[L].next.
  // mode 0: stored as entries of level L + 1 (until that buffer is full);
  // mode 1: counted into `count`; mode 2: counted per entry into sizes[].
  // Modes 0 and 1 resume at, and leave, the block's position in W.lev[L]; they
  // stop early (false) when a warp is idle and there are entries to give it.
  // FIXED -1: the mode is an argument and one copy of this code serves all
  // three.  Labeled launches take it: the warps of an SM run many small plans
  // there, and with a copy per mode the kernel outgrew the instruction cache
  // (no_instruction 10.6 cycles per issue; power-law labeled batch 3.62 against
  // 2.92 ms, ER 0.187 against 0.150).  Unlabeled ones run long scans of few
  // plans and do better without the mode's tests in the step (5-clique share
  // 21.4 against 25.1 ms).
  template <int FIXED>
  __device__ __forceinline__ bool scan(const FlatStep &st, int L, int how, uint32_t *sizes, int &width) {
    const int mode = FIXED >= 0 ? FIXED : how;
    FlatLevel &H = W.lev[L];
    const int first = H.next;
    int len = 0;
    int64_t base = 0;
    uint2 table0 = make_uint2(0u, 0u);
    if (first + lane < H.end) len = setup_lane(st, L, first + lane, base, table0);
    uint32_t incl = (uint32_t)len;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const uint32_t t = __shfl_up_sync(kFull, incl, s);
      if (lane >= s) incl += t;
    }
    const uint32_t off = len > 0 ? incl - (uint32_t)len : ~0u;  // lanes without a list start nowhere
    if (mode == 2) {
      // a tail's block ends before its lists grow past kTailSpan positions
      const unsigned fit = __ballot_sync(kFull, lane < width && incl <= (uint32_t)kTailSpan);
      width = max(__popc(fit), 1);
    }
    const uint32_t total = __shfl_sync(kFull, incl, mode == 2 ? width - 1 : 31);
    const unsigned act = __ballot_sync(kFull, len > 0);
    if (len > 0) {
      const int rank = __popc(act & lanemask_lt());
      base -= 4 * (int64_t)off;
      W.map[rank] = (uint8_t)lane;
      W.src[rank] = make_int4((int)base, (int)(base >> 32), (int)table0.x, (int)table0.y);
    }
    __syncwarp();
    uint32_t pos = mode < 2 ? H.pos : 0u;
    int cur = __popc(__ballot_sync(kFull, off < pos));  // lists that start before pos
    const unsigned le = lanemask_lt() | (1u << lane);
    const int M = st.nbn - 1;
    const unsigned neq = st.neq;
    const bool lab = LAB && !segmented();
    int32_t *ox = nullptr;
    uint16_t *op = nullptr;
    int n = 0;
    if (mode == 0) {
      ox = xs(L + 1);
      op = ps(L + 1);
      n = W.lev[L + 1].n;
    }
    const int most = mode == 0 ? room(L + 1) : 0;
    bool early = false;
    for (int step = 0; pos < total; ++step, pos += 64) {
      if (mode == 0 && n > most) break;
      if (mode < 2 && (step & (kLookSteps - 1)) == kLookSteps - 1 && someone_idle()) {
        bool give = H.end > first + 32 || __any_sync(kFull, len > 0 && off >= pos);
        for (int l = W.root; l < L; ++l) give |= untouched(l) > 0;
        if (give) {
          early = true;
          break;
        }
      }
      int o[2];
      int32_t x[2];
      uint2 t0[2] = {make_uint2(0u, 0u), make_uint2(0u, 0u)};
      bool ok[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const uint32_t b = pos + 32 * u;
        // the lists that start inside these 32 positions, as a bit mask: a
        // lane's owner is the last one that starts at or before it
        const unsigned m = __reduce_or_sync(kFull, bit_at(off - b));
        const int r = cur + __popc(m & le) - 1;
        cur += __popc(m);
        ok[u] = b + (uint32_t)lane < total;
        o[u] = 0;
        x[u] = 0;
        if (ok[u]) {
          const int4 src = W.src[r];
          o[u] = W.map[r];
          // (a generic load: sources lie in global or in shared memory)
          const int64_t at = ((int64_t)src.y << 32 | (uint32_t)src.x) + 4 * (int64_t)(b + (uint32_t)lane);
          x[u] = *reinterpret_cast<const int32_t *>(at);
          t0[u] = make_uint2((unsigned)src.z, (unsigned)src.w);
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        if (lab && ok[u]) ok[u] = G.label[x[u]] == st.label;
        for (unsigned m = neq; m; m &= m - 1) ok[u] &= W.phi[__ffs(m) - 1][o[u]] != x[u];
      }
      for (int m = 0; m < M && __any_sync(kFull, ok[0] || ok[1]); ++m) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (m > 0) t0[u] = W.more[m - 1][o[u]];
          if (ok[u] && t0[u].y) {
            const uint32_t at = __umulhi((uint32_t)x[u] * kRowHash, t0[u].y);
            ok[u] = found(bucket(t0[u].x + at), t0[u].x, t0[u].y, at, x[u]);
          }
        }
      }
      if (mode == 0) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const unsigned m = __ballot_sync(kFull, ok[u]);
          if (ok[u]) {
            const int at = n + __popc(m & lanemask_lt());
            ox[at] = x[u];
            op[at] = (uint16_t)(first + o[u]);
          }
          n += __popc(m);
        }
      } else if (mode == 1) {
        count += (unsigned)ok[0] + (unsigned)ok[1];
      } else {
#pragma unroll
        for (int u = 0; u < 2; ++u)
          if (ok[u]) atomicAdd(&sizes[o[u]], 1u);
      }
    }
    __syncwarp();
    if (mode == 2) return true;
    const bool done = pos >= total;
    const unsigned in = __ballot_sync(kFull, off < pos && off + (uint32_t)len > pos);
    const unsigned before = __ballot_sync(kFull, off < pos);
    if (lane == 0) {
      if (mode == 0) W.lev[L + 1].n = n;
      if (done) {
        H.next = min(first + 32, H.end);
        H.pos = 0;
        H.started = H.next;
        H.cutp = -1;
      } else {
        H.pos = pos;
        H.started = before ? first + 32 - __clz(before) : first;
        H.cutp = in ? first + __ffs(in) - 1 : -1;
      }
    }
    __syncwarp();
    return !early;
  }

  // Start filling level L + 1 from the entries of level L.
  __device__ void fill_begin(int L) {
    FlatLevel &H = W.lev[L], &D = W.lev[L + 1];
    if (lane == 0) {
      D.next = D.end = D.n = 0;
      D.pos = 0;
      D.started = 0;
      D.cutp = -1;
      D.hcut = H.pos ? H.cutp : -1;
      D.groups = 1;
    }
    __syncwarp();
  }
  // Level L + 1 is full, or level L has no entries left.
  __device__ void fill_end(int L) {
    FlatLevel &H = W.lev[L], &D = W.lev[L + 1];
    if (lane == 0) {
      D.end = D.n;
      D.tcut = H.pos ? H.cutp : -1;
      if (BIG && W.rlevel == L + 1) {
        // given a range of one entry's children: the others serve as siblings only
        const int32_t *x = xs(L + 1);
        D.next = below(x, D.n, W.rlo);
        D.end = below(x, D.n, W.rhi + 1);
        if (D.end < D.n) {  // nothing in range beyond this fill
          H.next = H.end;
          H.pos = 0;
        }
      }
    }
    __syncwarp();
  }

  // Entries of the ascending x[0, n) below v.
  __device__ __forceinline__ static int below(const int32_t *x, int n, int32_t v) {
    int a = 0, z = n;
    while (a < z) {
      const int m = (a + z) >> 1;
      if (x[m] < v) a = m + 1; else z = m;
    }
    return a;
  }

  // Size of the set st of this lane's embedding (in W.phi), st having a single
  // list: the list's part inside the bounds, less the earlier vertices found
  // in it (on labeled plans those of the set's label).
  __device__ uint32_t closed_count(const FlatStep &st) {
    const int32_t v = W.phi[st.bn[0]][lane];
    int64_t b;
    uint32_t ulen;
    row(v, st.label, b, ulen);
    int len = (int)ulen;
    int32_t lo, hi;
    bounds(st, lo, hi);
    if (!LAB) trim(lists(), b, len, lo, hi);
    if (len <= 0) return 0;
    int c = len;
    for (unsigned m = st.neq; m; m &= m - 1) {
      const int j = __ffs(m) - 1;
      const int32_t y = W.phi[j][lane];
      if (j == 1 && (st.neq & 1) && y == W.phi[0][lane]) continue;  // a self-loop edge: one value
      if (y > lo && y < hi && member(v, y)) --c;
    }
    return (uint32_t)c;
  }

  // Single lists are counted in closed form, except on whole rows with labels.
  __device__ __forceinline__ bool closed(const FlatStep &st) const { return st.nbn == 1 && (!LAB || segmented()); }

  // The tuples of distinct vertices below this lane's entry, from the sizes of
  // the tail's sets in cnt().
  __device__ __forceinline__ unsigned long long tuples() const {
    const FlatPlan &F = W.plan;
    auto at = [&](int m) -> unsigned long long {
      const int u = F.term_of[m];
      return u == kNoTerm ? 0ull : (unsigned long long)cnt(u)[lane];
    };
    const unsigned long long a = at(1);
    if (F.form == 1) {
      // subsets of two or three; counts are modulo 2^64, so 3 is divided out of a
      // factor that holds it and not out of the product, which passes 2^64 from
      // 3.3M candidates on
      const unsigned long long pairs = a * (a - 1) / 2;
      if (F.t == 2) return pairs;
      return (uint32_t)a % 3 == 2 ? pairs * ((a - 2) / 3) : pairs / 3 * (a - 2);
    }
    const unsigned long long b = at(2);
    if (F.t == 2) return a * b - at(3);
    const unsigned long long c = at(4);
    return a * b * c - at(3) * c - at(5) * b - at(6) * a + 2 * at(7);
  }

  // One block of level L: extended into level L + 1, or, at level s, counted.
  // `filling`: level L + 1 is being filled.  Returns whether it still is.
  __device__ bool advance(int L, bool filling) {
    FlatLevel &H = W.lev[L];
    const FlatPlan &F = W.plan;
    const bool leaf = L == F.s, tail = leaf && F.t > 1;
    int width = 32;  // entries of this block
    if (!leaf && !filling) fill_begin(L);
    if (!LAB && !leaf) {
      while (H.next < H.end && W.lev[L + 1].n <= room(L + 1))
        if (!scan<0>(F.step[L - 1], L, 0, nullptr, width)) return true;
      fill_end(L);
      return false;
    }
    if (!LAB && F.t == 1 && !closed(F.term[0])) {
      scan<1>(F.term[0], L, 1, nullptr, width);
      return false;
    }
    const int p = H.next + lane;
    const bool mine = p < H.end;
    bool scanned = false;
    const int sets = tail ? F.nterm : 1;
    for (int u = 0; u < sets; ++u) {
      const FlatStep &st = leaf ? F.term[u] : F.step[L - 1];
      if (leaf && closed(st)) {
        uint32_t c = 0;
        if (mine) {
          load_tuple(L, p, 0);
          c = closed_count(st);
        }
        if (tail) cnt(u)[lane] = c;
        else count += c;
      } else {
        if (tail) cnt(u)[lane] = 0;
        __syncwarp();
        if (LAB) scan<-1>(st, L, tail ? 2 : leaf ? 1 : 0, tail ? cnt(u) : nullptr, width);
        else scan<2>(st, L, 2, cnt(u), width);
        scanned = true;
      }
      __syncwarp();
    }
    if (LAB && !leaf) {
      if (H.next < H.end && W.lev[L + 1].n <= room(L + 1)) return true;
      fill_end(L);
      return false;
    }
    if (tail && mine && lane < width) count += tuples();
    __syncwarp();
    if (tail || !scanned) {  // the whole block is done (a scan of mode 1 keeps its own place)
      if (lane == 0) {
        H.next = min(H.next + width, H.end);
        H.started = H.next;
      }
      __syncwarp();
    }
    return false;
  }

  // ---- query slots -------------------------------------------------------------

  __device__ void load_plan(int s) {
    if (W.slot == s) return;
    flush();
    const int32_t *srcw = reinterpret_cast<const int32_t *>(&T.plan[s]);
    int32_t *dstw = reinterpret_cast<int32_t *>(&W.plan);
    for (int t = lane; t < (int)(sizeof(FlatPlan) / 4); t += 32) dstw[t] = __ldcg(srcw + t);
    __syncwarp();
    if (lane < 11 && !*G.loops) {
      // no self-loops: a neighbour of phi(j) differs from phi(j)
      FlatStep &st = lane < 4 ? W.plan.step[lane] : W.plan.term[lane - 4];
      for (int t = 0; t < st.nbn; ++t) st.neq &= (uint8_t)~(1u << st.bn[t]);
    }
    if (lane == 0) {
      W.slot = s;
      W.low = BIG && W.plan.reuse2 ? 3 : 2;
      W.levels = max(1, (int)W.plan.s - W.low + 1);  // levels low..s
      W.cap = ((cfg.entries - (W.plan.t > 1 ? kCntBytes / 6 + 1 : 0)) / W.levels) & ~31;
    }
    __syncwarp();
  }

  // Add this warp's count to its slot's: through shared memory for the slot
  // most warps of the CTA started with, so a launch of one slot does one
  // atomic per CTA and not per warp on it.
  __device__ void flush() {
    unsigned long long c = count;
    count = 0;
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) c += __shfl_xor_sync(kFull, c, d);
    if (lane == 0 && c) {
      if (W.slot == C.slot) atomicAdd(&C.sum, c);
      else atomicAdd(&T.count[W.slot], c);
    }
    __syncwarp();
  }

  // Ticket t of slot s: its edges that pass get_job's filter
  // (src/gpu_match.cu:531-556) become level-1 entries.
  __device__ bool fetch_chunk(int s, long long t) {
    const FlatInfo &in = T.info[s];
    const FlatPlan &F = W.plan;
    const int chunk = __ldcg(&in.chunk);
    const int64_t e = __ldcg(&in.e_begin) + (t * __ldcg(&in.stride) + __ldcg(&in.phase)) * (int64_t)chunk + lane;
    bool ok = lane < chunk && e < __ldcg(&in.e_end);
    int32_t r = 0, c = 0;
    if (ok) {
      const int64_t ed = __ldcg(&in.perm) ? (int64_t)G.lperm[e] : e;
      r = G.src[ed];
      c = G.colidx[ed];
      if (!LAB && F.orient && !(r < c)) ok = false;
      if (LAB && ok && ((int32_t)G.label[r] != F.label[0] || (int32_t)G.label[c] != F.label[1])) ok = false;
      if (ok && (G.rowptr[r + 1] - G.rowptr[r] < F.deg[0] || G.rowptr[c + 1] - G.rowptr[c] < F.deg[1] ||
                 G.maxnd[c] < F.deg[2]))
        ok = false;
    }
    const unsigned mask = __ballot_sync(kFull, ok);
    if (!mask) return false;
    if (ok) {
      const int at = __popc(mask & lanemask_lt());
      W.er[at] = r;
      W.ec[at] = c;
    }
    install(1, __popc(mask));
    return true;
  }

  // Entries [0, n) of level l become this warp's base work.
  __device__ void install(int l, int n) {
    if (lane == 0) {
      for (int j = 1; j <= l; ++j) {
        FlatLevel &H = W.lev[j];
        H.next = H.end = H.started = 0;
        H.pos = 0;
        H.cutp = -1;
        H.groups = 0;
      }
      W.lev[l].end = W.lev[l].n = n;
      W.root = l;
      W.rlevel = 0;
      W.t_work = now_ns();
    }
    __syncwarp();
  }

  // Take over ticket t of the launch: find its slot and fetch its edges.
  // Tickets ascend, so the search starts at the slot of the last one.
  __device__ bool start_ticket(long long t, int &hint) {
    const int n = T.ctl->slots;
    int s = hint;
    for (;; s += 31) {
      // the last slot that starts at or before t; slots in [s, s + 32) at a time
      const bool le = s + lane < n && __ldg(&T.info[s + lane].ticket0) <= t;
      const int c = __popc(__ballot_sync(kFull, le));
      if (c < 32) {
        s += c - 1;
        break;
      }
    }
    hint = s;
    load_plan(s);
    return fetch_chunk(s, t - __ldg(&T.info[s].ticket0));
  }

  // The next ticket that yields edges; false when none is left.
  __device__ bool next_ticket(int &hint) {
    for (;;) {
      long long t = 0;
      if (lane == 0) t = (long long)(atomicAdd(&T.ctl->ticket, 1ull) & (kCtaJoin - 1));
      t = __shfl_sync(kFull, t, 0);
      if (t >= T.ctl->tickets) return false;
      if (start_ticket(t, hint)) return true;
    }
  }

  // ---- giving work away -------------------------------------------------------

  // Give up to half of the untouched entries of the shallowest level that has
  // some to idle warps, if there are any.  Entries whose extension reads their
  // siblings (reuse) go as a range of one parent's children: the receiver
  // makes the parent's children again, so that it has the siblings too.
  __device__ void donate(int base, int level) {
    int l = base, take = 0, parent = -1;
    for (; l <= level; ++l) {
      const FlatLevel &H = W.lev[l];
      int avail = untouched(l);
      bool other = l < level || H.pos;  // work stays here besides these entries
      if (BIG && avail >= 2 * kRangeMin && l >= 2 && H.groups &&
          (l < W.plan.s ? W.plan.step[l - 1] : W.plan.term[0]).dep == l) {
        const uint16_t *pp = ps(l);
        const int me = pp[H.end - 1];
        int a = H.end - avail, z = H.end - 1;  // the first untouched child of me
        while (a < z) {
          const int m = (a + z) >> 1;
          if (pp[m] < me) a = m + 1; else z = m;
        }
        if (H.end - a >= 2 * kRangeMin) {
          parent = me;
          other |= a > H.end - avail;
          avail = H.end - a;
        }
      }
      take = other ? (avail + 1) >> 1 : avail >> 1;
      if (take > 0) break;
    }
    if (l > level) return;
    int w;
    const unsigned idle = idle_word(w);
    unsigned have = __ballot_sync(kFull, idle != 0);
    if (!have) return;
    bool mine = idle != 0 && __popc(have & lanemask_lt()) < take;
    int target = 0;
    if (mine) {
      const int r = (gid + lane) & 31;  // start at another bit than other warps
      const unsigned rot = __funnelshift_r(idle, idle, r);
      const unsigned bit = 1u << ((__ffs(rot) - 1 + r) & 31);
      mine = (atomicAnd(&T.idle[w], ~bit) & bit) != 0;
      target = w * 32 + __ffs(bit) - 1;
    }
    have = __ballot_sync(kFull, mine);
    const int boxes = __popc(have);
    if (!boxes) return;
    // entries [from, end) of level l, `per` to a box
    const int per = parent >= 0 ? max(kRangeMin, (take + boxes - 1) / boxes)
                                : min(min(32, kBoxInts / (l + 1)), (take + boxes - 1) / boxes);
    take = min(take, per * boxes);
    const int used = (take + per - 1) / per;
    const int rank = __popc(have & lanemask_lt());
    if (mine) W.src[rank].x = target;
    if (lane == 0) atomicAdd(&T.ctl->pending, used);
    __syncwarp();
    const int from = W.lev[l].end - take;
    for (int t = lane; t < take && parent < 0; t += 32) {
      int32_t *v = T.box[W.src[t / per].x].v + (t % per) * (l + 1);
      int q = from + t;
      for (int j = l; j >= 2; --j) {
        v[j] = xs(j)[q];
        q = ps(j)[q];
      }
      v[0] = W.er[q];
      v[1] = W.ec[q];
    }
    const bool fill = mine && rank < used;
    if (fill) {
      FlatBox &b = T.box[target];
      b.slot = W.slot;
      const int mine_n = min(per, take - rank * per);
      if (BIG && parent >= 0) {
        int q = parent;
        for (int j = l - 1; j >= 2; --j) {
          b.v[j] = xs(j)[q];
          q = ps(j)[q];
        }
        b.v[0] = W.er[q];
        b.v[1] = W.ec[q];
        b.lo = xs(l)[from + rank * per];
        b.hi = xs(l)[from + rank * per + mine_n - 1];
      }
      b.level = parent >= 0 ? l - 1 : l;
      b.n = parent >= 0 ? 1 : mine_n;
      b.range = parent >= 0;
    }
    __threadfence();
    __syncwarp();
    if (fill) *(volatile int32_t *)&T.box[target].full = 1;
    else if (mine) atomicOr(&T.idle[target >> 5], 1u << (target & 31));  // claimed but not needed
    if (lane == 0) {
      W.lev[l].end = from;
      atomicAdd(&T.run->splits, (unsigned long long)used);
    }
    __syncwarp();
  }

  // Take over the entries in this warp's mailbox; returns their level.
  __device__ int open_box() {
    __threadfence();
    const FlatBox &box = T.box[gid];
    const int l = __ldcg(&box.level), n = __ldcg(&box.n);
    load_plan(__ldcg(&box.slot));
    if (lane < n) {
      const int32_t *v = box.v + lane * (l + 1);
      W.er[lane] = __ldcg(v);
      W.ec[lane] = __ldcg(v + 1);
      for (int j = 2; j <= l; ++j) {
        xs(j)[lane] = __ldcg(v + j);
        ps(j)[lane] = (uint16_t)lane;
      }
    }
    install(l, n);
    if (BIG && lane == 0 && __ldcg(&box.range)) {
      W.rlevel = l + 1;
      W.rlo = __ldcg(&box.lo);
      W.rhi = __ldcg(&box.hi);
    }
    __syncwarp();
    return l;
  }

  // p: FlatCtl::pending as just read.  Is no CTA busy and no mailbox full?  The
  // count of started CTAs is read after p, and it only grows: a sum of 0 means
  // that when p was read every CTA started until then was idle.  A warp asks
  // once it has seen the last ticket go, and the atomic that takes a CTA's
  // tickets also counts it, so whoever took one is among them.  Once the whole
  // grid has started, p alone tells.  (Out of line: the code of labeled launches
  // is at the limit of the instruction cache; inlined in its three places it
  // cost a batch of 4 power-law queries 7 %, 0.645 to 0.692 ms, here 1.7 %.)
  __device__ __noinline__ static bool complete(int p, const FlatCtl *ctl, FlatCta &C) {
    const int grid = (int)gridDim.x;
    if (p == -grid) return true;
    if (*(volatile int32_t *)&C.all) return false;
    __threadfence();
    const int started = (int)(*(const volatile unsigned long long *)&ctl->ticket >> kJoinShift);
    if (started == grid) *(volatile int32_t *)&C.all = 1;
    return p + started == 0;
  }
  // A warp has run dry (lane 0).  True when it was its CTA's last busy one and
  // nothing is left anywhere.
  __device__ __forceinline__ bool cta_idle() const {
    return atomicSub(&C.active, 1) == 1 && complete(atomicSub(&T.ctl->pending, 1) - 1, T.ctl, C);
  }

  // Wait until this warp is given work (returns its level, installed) or none
  // will come (0).  A waiting warp reads its own mailbox; one per CTA also
  // reads the count of what is pending.  Bounded: after cfg.idle_ms the
  // launch reports a timeout.
  __device__ int wait_for_work() {
    int st = 0;  // 1: the mailbox is full, 2: stop
    const unsigned long long t0 = now_ns();
    flush();
    if (!cfg.share) {
      // light, even work: nothing to wait for
      if (lane == 0 && cta_idle()) T.run->finished = 1;
      __syncwarp();
      return 0;
    }
    if (lane == 0) {
      *(volatile int32_t *)&T.box[gid].full = 0;
      __threadfence();  // (the CTA's start comes before its idleness, too)
      atomicOr(&T.idle[gid >> 5], 1u << (gid & 31));
      if (cta_idle()) {
        T.run->finished = 1;
        *(volatile int32_t *)&C.done = 1;
      }
    }
    bool poller = false;
    unsigned nap = 200;
    for (;;) {
      if (lane == 0) {
        if (*(volatile int32_t *)&T.box[gid].full) st = 1;
        else if (*(volatile int32_t *)&C.done) st = 2;
        else if (poller || (poller = atomicCAS(&C.poll, 0, 1) == 0)) {
          if (complete(*(volatile int32_t *)&T.ctl->pending, T.ctl, C)) {
            *(volatile int32_t *)&C.done = 1;
            st = 2;
          }
        }
        if (!st && now_ns() - t0 > (unsigned long long)cfg.idle_ms * 1000000ull) {
          atomicCAS(&T.run->error, 0, TDFS_ERR_TIMEOUT);
          st = 2;
        }
      }
      st = __shfl_sync(kFull, st, 0);
      if (st) break;
      __nanosleep(nap);
      nap = min(2 * nap, 1600u);
    }
    if (lane == 0) {
      if (poller) atomicExch(&C.poll, 0);
      // the mailbox's place in `pending` becomes the CTA's when it had no busy warp
      if (st == 1 && atomicAdd(&C.active, 1) > 0) atomicSub(&T.ctl->pending, 1);
      W.idle_total += now_ns() - t0;
    }
    __syncwarp();
    return st == 1 ? open_box() : 0;
  }

  // Level l extends its entries into level l + 1, the level s counts.  `base`
  // is the level whose entries this warp was given; below it the warp takes
  // the next ticket or waits to be given some.
  __device__ void run() {
    if (lane == 0) {
      W.t_start = now_ns();
      W.slot = -1;
      W.idle_total = 0;
    }
    __syncwarp();
    int level = 0, base = 1, hint = 0;
    bool more = false;
    const long long mine = C.first + (threadIdx.x >> 5);
    bool dry = C.first + (blockDim.x >> 5) >= T.ctl->tickets;  // none besides the CTA's first ones
    long long checked = clock64();
    if (mine < T.ctl->tickets && start_ticket(mine, hint)) level = 1;
    for (;;) {
      if (level < base) {
        level = 0;
        if (!dry) {
          if (next_ticket(hint)) level = base = 1;
          else dry = true;
        }
        if (!level) {
          level = base = wait_for_work();
          if (!level) break;
        }
        continue;
      }
      const FlatLevel &H = W.lev[level];
      if (H.next >= H.end && !more) {
        --level;
        continue;
      }
      const bool inner = level < W.plan.s;
      more = advance(level, more);
      if (inner && !more && W.lev[level + 1].n > 0) ++level;
      const long long c = clock64();
      int due = 0;
      if (c - checked > cfg.check) {
        checked = c;
        due = may_give();
      }
      if (__shfl_sync(kFull, due, 0)) donate(base, level);
    }
    // the CTA's sums, by its last warp; the results, by the grid's
    int last = 0;
    if (lane == 0) {
      atomicAdd(&C.idle_ns, W.idle_total);
      atomicAdd(&C.warp_ns, now_ns() - W.t_start);
      __threadfence_block();
      if (atomicSub(&C.left, 1) == 1) {
        __threadfence_block();
        if (C.sum) atomicAdd(&T.count[C.slot], C.sum);
        atomicAdd(&T.run->idle_ns, C.idle_ns);
        atomicAdd(&T.run->warp_ns, C.warp_ns);
        if (T.host) {
          __threadfence();
          last = atomicAdd(&T.ctl->gone, 1) == (int)gridDim.x - 1;
        }
      }
    }
    if (__shfl_sync(kFull, last, 0)) {
      __threadfence();
      const int words = (int)(FlatTable::readback(T.ctl->slots) / 4);
      for (int i = lane; i < words; i += 32)
        static_cast<volatile int32_t *>(T.host)[i] = __ldcg(reinterpret_cast<const int32_t *>(T.run) + i);
    }
  }
};

// Two register budgets of one kernel: 64 for 4 CTAs of 256 threads per SM, and
// 80 for 3, whose scan step has more loads in flight: on skewed graphs, where
// long scans dominate, it is the faster one (R-MAT 4-clique share 17.0 against
// 19.0 ms, house slice 38.5 against 40.4), on small uniform graphs the warps
// count (64-query burst 1.11 times as long with 80).
template <bool LAB, int MINB, bool BIG>
__global__ void __launch_bounds__(256, MINB) flat_kernel(const __grid_constant__ DevGraph G,
                                                      const __grid_constant__ FlatCfg cfg,
                                                      const __grid_constant__ FlatTable T) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ FlatCta cta;
  if (threadIdx.x == 0) {
    cta.poll = cta.done = 0;
    cta.all = !cfg.share;
    cta.active = cta.left = (int)(blockDim.x >> 5);
    const unsigned warps = blockDim.x >> 5;
    cta.first = cfg.share ? (long long)(atomicAdd(&T.ctl->ticket, kCtaJoin + warps) & (kCtaJoin - 1))
                          : (long long)blockIdx.x * warps;
    cta.slot = 0;
    cta.sum = cta.idle_ns = cta.warp_ns = 0;
  }
  __syncthreads();
  const int me = threadIdx.x >> 5;
  unsigned char *base = smem + (size_t)me * cfg.warp_bytes;
  FlatSmem &W = *reinterpret_cast<FlatSmem *>(base);
  Flat<LAB, BIG> f(G, cfg, T, (int)blockIdx.x * (int)(blockDim.x >> 5) + me, W, cta, base + sizeof(FlatSmem));
  f.run();
}

template <bool LAB, int MINB, bool BIG>
cudaError_t flat_smem(size_t smem) {
  static std::mutex mu;
  static size_t set_to[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64) return e != cudaSuccess ? e : cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lk(mu);
  if (smem <= set_to[dev]) return cudaSuccess;
  e = cudaFuncSetAttribute(flat_kernel<LAB, MINB, BIG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) set_to[dev] = smem;
  return e;
}

}  // namespace

int flat_min_entries(int levels, int tmax) { return 64 * levels + (tmax > 1 ? kCntBytes / 6 + 33 : 0); }

size_t flat_warp_bytes(int entries) {
  return (sizeof(FlatSmem) + (size_t)entries * 6 + 15) & ~(size_t)15;
}

int flat_auto_entries() {
  constexpr int kPerWarp = (228 * 1024 / 4 - 1024 - 128) / 8 & ~15;  // 4 CTAs of 8 warps on 228 KB, 1 KB per CTA reserved
  static_assert(kPerWarp > (int)sizeof(FlatSmem) + 5 * 64 * 6, "room for 64 entries of every level");
  return (kPerWarp - (int)sizeof(FlatSmem)) / 6 & ~31;
}

int flat_max_entries(int warps) { return (227 * 1024 / warps - 48 - (int)sizeof(FlatSmem)) / 6 & ~31; }

namespace {

template <bool LAB, int MINB, bool BIG>
int flat_fit(int threads, size_t smem) {
  int n = 0;
  cudaError_t e = flat_smem<LAB, MINB, BIG>(smem);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, flat_kernel<LAB, MINB, BIG>, threads, smem);
  return e == cudaSuccess ? n : -1;
}

template <bool LAB, int MINB, bool BIG>
cudaError_t flat_go(const DevGraph &g, const FlatTable &t, const FlatCfg &cfg, int blocks, int threads, size_t smem,
                    cudaStream_t stream) {
  const cudaError_t e = flat_smem<LAB, MINB, BIG>(smem);
  if (e != cudaSuccess) return e;
  (void)cudaGetLastError();  // the check below must see this launch's error only
  flat_kernel<LAB, MINB, BIG><<<blocks, threads, smem, stream>>>(g, cfg, t);
  return cudaGetLastError();
}

}  // namespace

int flat_blocks_per_sm(bool labeled, bool wide, bool big, int warps_per_block, size_t smem) {
  const int threads = warps_per_block * 32;
  if (big) return labeled ? flat_fit<true, 3, true>(threads, smem) : flat_fit<false, 3, true>(threads, smem);
  if (wide) return labeled ? flat_fit<true, 3, false>(threads, smem) : flat_fit<false, 3, false>(threads, smem);
  return labeled ? flat_fit<true, 4, false>(threads, smem) : flat_fit<false, 4, false>(threads, smem);
}

int flat_chunk(int64_t edges, int s, bool skewed, int stride, int warps, int edge_chunk) {
  if (edge_chunk > 0) return edge_chunk;
  if (stride > 1) return 32;  // the documented round-robin deal
  // Full lanes at the first levels against even shares.  A plan counted at its
  // edges has little work per edge and wants all 32 lanes (triangles of the
  // n=4096 ER graph: 87 us with 1 edge per ticket, 39 with 4, 25 with 32); each
  // level more multiplies an edge's work (64-query burst, s up to 4: 2.9 times as
  // long with 1 as with 4 or 8).  Where hubs make some edges thousands of
  // times heavier than others, consecutive ones (a hub's) go to different
  // warps: power-law labeled batch 2.6 ms with 1, 3.0 with 4; triangles 0.16
  // with 4, 0.22 with 32.
  int c = s <= 1 ? (skewed ? 8 : 32) : s == 2 ? 8 : skewed ? 1 : 4;
  // enough tickets to even the warps out; a quarter of the warps suffices for
  // the light edges of s = 1
  const int64_t least = s <= 1 ? warps / 4 : s == 2 ? 2ll * warps : 3ll * warps;
  while (c > 1 && edges / c < least) c >>= 1;
  return c;
}

int launch_flat(bool labeled, const DevGraph &g, const FlatTable &t, const FlatCfg &cfg, int blocks,
                int warps_per_block, cudaStream_t stream) {
  const size_t smem = (size_t)cfg.warp_bytes * warps_per_block;
  const int threads = warps_per_block * 32;
  auto go = [&](auto f) { return f(g, t, cfg, blocks, threads, smem, stream); };
  const cudaError_t e = t.big      ? labeled ? go(flat_go<true, 3, true>) : go(flat_go<false, 3, true>)
                        : cfg.wide ? labeled ? go(flat_go<true, 3, false>) : go(flat_go<false, 3, false>)
                        : labeled  ? go(flat_go<true, 4, false>)
                                   : go(flat_go<false, 4, false>);
  if (e != cudaSuccess) return fail(TDFS_ERR_CUDA, "flat kernel launch: %s", cudaGetErrorString(e));
  return TDFS_OK;
}

}  // namespace tdfs
