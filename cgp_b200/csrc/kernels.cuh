// Device code of the multi-query traversal engine (sm_100a).
//
// One traversal group holds up to 64*W queries; every vertex carries W 64-bit
// mask words.  Per level the host-free control block (LevelCtl) decides the
// direction on the device, so a whole chunk of levels can be captured in one
// CUDA graph and replayed without host synchronisation.
//
// Reference correspondence (paths relative to the reference project root):
//   push  : expand_shared_node_{,warp_}kernel, frontier_engine.hxx:678-943,
//           expand_shared_node_{,warp_}hybrid_kernel, hybrid_engine.hxx:132-330
//   pull  : fused_ge_bfs_pull_*, frontier_engine.hxx:1561-1740 (bottom-up BFS)
//   next-frontier marking : mark_next_shared_frontier[_with_signal],
//           frontier_engine.hxx:117-173 (here warp-aggregated)
//   min relaxation : apply_min_reduce, reduce_ops.hxx:40-56 (here a single
//           atomicMin on the ordered uint32 image of the value)
#pragma once

#include <cstdint>
#include <type_traits>

#include <cuda_runtime.h>

#include "device_types.cuh"

namespace cgp {
namespace dev {

// ------------------------------------------------------------------ utils
template <int W>
__device__ __forceinline__ void load_mask(const uint64_t* p, uint64_t (&m)[W]) {
  if constexpr (W % 2 == 0) {
#pragma unroll
    for (int i = 0; i < W; i += 2) {
      ulonglong2 x = *reinterpret_cast<const ulonglong2*>(p + i);
      m[i] = x.x;
      m[i + 1] = x.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < W; ++i) m[i] = p[i];
  }
}

// Asks L2 to fetch the line holding p (no register is written, nothing waits).
__device__ __forceinline__ void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

template <int W>
__device__ __forceinline__ void store_mask(uint64_t* p, const uint64_t (&m)[W]) {
  if constexpr (W % 2 == 0) {
#pragma unroll
    for (int i = 0; i < W; i += 2) {
      *reinterpret_cast<ulonglong2*>(p + i) = make_ulonglong2(m[i], m[i + 1]);
    }
  } else {
#pragma unroll
    for (int i = 0; i < W; ++i) p[i] = m[i];
  }
}

template <int W>
__device__ __forceinline__ bool mask_any(const uint64_t (&m)[W]) {
  uint64_t a = 0;
#pragma unroll
  for (int i = 0; i < W; ++i) a |= m[i];
  return a != 0;
}

template <int W>
__device__ __forceinline__ bool any_bits(const uint64_t* m) {
  uint64_t a = 0;
  for (int i = 0; i < W; ++i) a |= m[i];
  return a != 0;
}

__device__ __forceinline__ uint64_t atomic_or64(uint64_t* p, uint64_t v) {
  return static_cast<uint64_t>(atomicOr(reinterpret_cast<unsigned long long*>(p),
                                        static_cast<unsigned long long>(v)));
}

// All 32 lanes call.  Lanes with `pred` append `v` to `list` (one atomicAdd
// per warp) and add `deg` to the edge counter.
__device__ __forceinline__ void warp_append(bool pred, int32_t v, uint64_t deg,
                                            int32_t* list,
                                            unsigned long long* count,
                                            unsigned long long* edges, int lane) {
  unsigned m = __ballot_sync(kFull, pred);
  if (m == 0) return;
  unsigned long long d = pred ? deg : 0ULL;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(kFull, d, o);
  int leader = __ffs(m) - 1;
  unsigned long long base = 0;
  if (lane == leader) {
    base = atomicAdd(count, static_cast<unsigned long long>(__popc(m)));
    atomicAdd(edges, d);
  }
  base = __shfl_sync(kFull, base, leader);
  if (pred) list[base + __popc(m & ((1u << lane) - 1u))] = v;
}

// Warp-sums `x` and lane 0 adds it to *dst (all lanes call).
__device__ __forceinline__ void warp_add(unsigned long long x, unsigned long long* dst, int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(kFull, x, o);
  if (lane == 0 && x) atomicAdd(dst, x);
}

template <int W>
__device__ __forceinline__ void warp_or_reduce(uint64_t (&m)[W]) {
  // two redux.sync per word (32-bit halves) instead of a 5-step shuffle tree
#pragma unroll
  for (int i = 0; i < W; ++i) {
    const unsigned lo = __reduce_or_sync(kFull, static_cast<unsigned>(m[i]));
    const unsigned hi = __reduce_or_sync(kFull, static_cast<unsigned>(m[i] >> 32));
    m[i] = (static_cast<uint64_t>(hi) << 32) | lo;
  }
}

// ORs each warp's union into ctl->active[par] (lane 0, nonzero words only).
template <int W>
__device__ __forceinline__ void flush_union(uint64_t (&uni)[W], uint64_t* dst,
                                            int lane) {
  warp_or_reduce<W>(uni);
  if (lane == 0) {
#pragma unroll
    for (int i = 0; i < W; ++i)
      if (uni[i]) atomic_or64(dst + i, uni[i]);
  }
}

// Position of the j-th (0-based) set bit of a 64-bit word, by halving with
// population counts.
__device__ __forceinline__ int select_bit64(uint64_t x, int j) {
  int pos = 0;
  int c = __popc(static_cast<unsigned>(x));
  if (j >= c) {
    j -= c;
    x >>= 32;
    pos += 32;
  }
  unsigned w = static_cast<unsigned>(x);
  c = __popc(w & 0xffffu);
  if (j >= c) { j -= c; w >>= 16; pos += 16; }
  c = __popc(w & 0xffu);
  if (j >= c) { j -= c; w >>= 8; pos += 8; }
  c = __popc(w & 0xfu);
  if (j >= c) { j -= c; w >>= 4; pos += 4; }
  c = __popc(w & 0x3u);
  if (j >= c) { j -= c; w >>= 2; pos += 2; }
  if (j >= static_cast<int>(w & 1u)) pos += 1;
  return pos;
}

// Bit c: 32-slot chunk c of the mask has a bit set.
template <int W>
__device__ __forceinline__ uint32_t chunk_bits(const uint64_t (&m)[W]) {
  uint32_t c = 0;
#pragma unroll
  for (int i = 0; i < W; ++i) {
    c |= (static_cast<uint32_t>(m[i]) != 0u ? 1u : 0u) << (2 * i);
    c |= (static_cast<uint32_t>(m[i] >> 32) != 0u ? 1u : 0u) << (2 * i + 1);
  }
  return c;
}

// Frontier summary of vertex u at `level`: its 32-slot chunks with a frontier
// bit, when the summary was written for this level (a stale word reads as
// "no chunk").  Only ever used to skip mask and row loads: a vertex of the
// current frontier always has its word, so no frontier bit is missed.
__device__ __forceinline__ uint32_t summary_chunks(const uint64_t* fsum, int level, int32_t u) {
  const uint64_t x = fsum[u];
  return (x >> 32) == static_cast<uint64_t>(level + 1) ? static_cast<uint32_t>(x) : 0u;
}

// Pointers of the current level.
struct LevelView {
  int level;
  int par;
  const int32_t* list;
  int32_t* nlist;
  const uint64_t* fcur;
  uint64_t* fnext;
  unsigned long long* ncount;
  unsigned long long* nedges;
  uint64_t* nactive;
};

__device__ __forceinline__ LevelView level_view(const GroupDev& g) {
  LevelView lv;
  lv.level = g.ctl->level;
  lv.par = lv.level & 1;
  lv.list = lv.par ? g.list1 : g.list0;
  lv.nlist = lv.par ? g.list0 : g.list1;
  lv.fcur = lv.par ? g.fbuf1 : g.fbuf0;
  lv.fnext = lv.par ? g.fbuf0 : g.fbuf1;
  lv.ncount = &g.ctl->count[lv.par ^ 1];
  lv.nedges = &g.ctl->edges[lv.par ^ 1];
  lv.nactive = g.ctl->active[lv.par ^ 1];
  return lv;
}

// Frontier vertices that a push level's tile kernels expand themselves: out-
// degree at most the returned limit.  Larger lists go to the heavy queue as
// kHeavyChunk-edge CTA work items: lists above heavy_degree always, and every
// list above 32 edges when the frontier is small (<= kSmallFrontier vertices,
// e.g. the sources' level) or skewed (more than 64 out-edges per vertex on
// average, e.g. the hubs reached by the sources): there a tile of 32 such
// vertices would be one warp's serial work while most warps of the grid have
// nothing to do.  (The heavy queue holds every vertex of out-degree > 32.)
constexpr unsigned long long kSmallFrontier = 4096;

// ... and at most this many out-edges stay with a tile on any level: a frontier
// of 86K vertices is one tile per warp, and a list of 2,000 edges among them was
// the level's whole time (R-MAT 20, 256 slots, 7.4M pairs: 1.6 ms).
constexpr int64_t kTileDegree = 256;

__device__ __forceinline__ int64_t push_light_limit(const GroupDev& g, const DevGraph& G,
                                                    unsigned long long count,
                                                    unsigned long long edges) {
  const bool spread = count <= kSmallFrontier || edges > 64ULL * count;
  if (g.hq_vertex == nullptr || G.heavy_degree <= 32) return G.heavy_degree;
  return spread ? 32 : min(G.heavy_degree, kTileDegree);
}

// Frontier vertices per tile: 32, or fewer (a power of two) while that leaves
// warps without a tile.  The lanes share a tile's edges either way, so a small
// frontier is spread over more warps, each with a shorter chain of steps.
__device__ __forceinline__ int tile_width(unsigned long long n, unsigned long long nwarps) {
  int w = 1;
  while (w < 32 && static_cast<unsigned long long>(w) * nwarps < n) w <<= 1;
  return w;
}

// ------------------------------------------------------- depth recording
// Records depth `depth_abs` (level + 1) for the newly visited bits `nw` of
// vertex n, words w0 .. w0 + WL of its W: direct mode writes values[n][q] =
// depth_abs - base[q]; planes mode ORs the bits into the planes of depth_abs's
// set bits.
template <int W, int DEPTH, int WL>
__device__ __forceinline__ void record_depth(const GroupDev& g, int64_t V, int32_t n, int w0,
                                            const uint64_t (&nw)[WL], int depth_abs,
                                            bool exclusive) {
  if constexpr (DEPTH == kDepthPlanes) {
    const int K = g.ctl->num_planes;
    for (int b = 0; b < K; ++b) {
      if (((depth_abs >> b) & 1) == 0) continue;
      uint64_t* p = g.planes + static_cast<size_t>(b) * static_cast<size_t>(V) * W +
                    static_cast<size_t>(n) * W + w0;
#pragma unroll
      for (int i = 0; i < WL; ++i) {
        if (!nw[i]) continue;
        if (exclusive) p[i] |= nw[i];
        else atomic_or64(p + i, nw[i]);
      }
    }
  } else if constexpr (DEPTH == kDepthDirect) {
    uint32_t* row = g.values + static_cast<size_t>(n) * static_cast<size_t>(g.Qg);
#pragma unroll
    for (int i = 0; i < WL; ++i) {
      uint64_t b = nw[i];
      while (b) {
        const int q = (w0 + i) * 64 + __ffsll(static_cast<long long>(b)) - 1;
        b &= b - 1;
        row[q] = static_cast<uint32_t>(depth_abs - g.slots[q].base);
      }
    }
  }
}

// --------------------------------------------------------------- BFS push
// One edge u->n of a push level for the visited-mask bits f of u.
template <int W, int DEPTH>
__device__ __forceinline__ bool bfs_visit(const GroupDev& g, int64_t V,
                                          const LevelView& lv, int32_t n,
                                          const uint64_t (&f)[W],
                                          uint64_t (&uni)[W],
                                          unsigned long long& pairs) {
  uint64_t* vis = g.visited + static_cast<size_t>(n) * W;
  uint64_t cur[W];
  load_mask<W>(vis, cur);
  uint64_t d[W];
  uint64_t any = 0;
#pragma unroll
  for (int i = 0; i < W; ++i) {
    d[i] = f[i] & ~cur[i];
    any |= d[i];
  }
  if (!any) return false;
  uint64_t nw[W];
  uint64_t anyn = 0;
#pragma unroll
  for (int i = 0; i < W; ++i) {
    nw[i] = 0;
    if (d[i]) {
      uint64_t old = atomic_or64(vis + i, d[i]);
      nw[i] = d[i] & ~old;
      anyn |= nw[i];
    }
  }
  if (!anyn) return false;
  uint64_t* fn = lv.fnext + static_cast<size_t>(n) * W;
#pragma unroll
  for (int i = 0; i < W; ++i) {
    if (nw[i]) {
      atomic_or64(fn + i, nw[i]);
      uni[i] |= nw[i];
      pairs += __popcll(nw[i]);
    }
  }
  record_depth<W, DEPTH, W>(g, V, n, 0, nw, lv.level + 1, false);
  return atomicMax(g.stamp + n, lv.level + 1) < lv.level + 1;
}

template <typename OT>
__device__ __forceinline__ uint64_t degree_of(const void* row, int32_t v) {
  return static_cast<uint64_t>(row_at<OT>(row, v + 1) - row_at<OT>(row, v));
}

// Appends the n vertices buffered in lanes 0..n-1 to the next frontier list
// with one reservation, adding their out-degrees to the edge counter (all
// lanes call).
template <typename OT>
__device__ __forceinline__ void flush_appends(int32_t v, int n, const DevGraph& G,
                                              const LevelView& lv, int lane) {
  unsigned long long e = lane < n ? degree_of<OT>(G.row, v) : 0ULL;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(kFull, e, o);
  unsigned long long base = 0;
  if (lane == 0) {
    base = atomicAdd(lv.ncount, static_cast<unsigned long long>(n));
    atomicAdd(lv.nedges, e);
  }
  base = __shfl_sync(kFull, base, 0);
  if (lane < n) lv.nlist[base + lane] = v;
}

// Per-warp buffer of vertices to append to the next frontier: lane i holds
// the i-th, and a reservation on the list's shared counters is made once per
// 32 vertices instead of once per step (those two counters are the most
// contended words of a level).  All lanes call add() and flush().
struct WarpAppender {
  int32_t v = 0;  // lane i: pending vertex i
  int n = 0;      // pending count (uniform)

  template <typename OT>
  __device__ __forceinline__ void add(bool pred, int32_t x, const DevGraph& G,
                                      const LevelView& lv, int lane) {
    const unsigned m = __ballot_sync(kFull, pred);
    if (m == 0) return;
    const int c = __popc(m);
    if (n + c > 32) flush<OT>(G, lv, lane);
    const int k = lane - n;  // this lane receives the k-th appended vertex
    const bool take = k >= 0 && k < c;
    const int src = take ? select_bit64(m, k) : lane;
    const int32_t got = __shfl_sync(kFull, x, src);
    if (take) v = got;
    n += c;
  }

  template <typename OT>
  __device__ __forceinline__ void flush(const DevGraph& G, const LevelView& lv, int lane) {
    if (n > 0) flush_appends<OT>(v, n, G, lv, lane);
    n = 0;
  }
};

// Push level, non-heavy frontier vertices: one warp per tile of 32 list
// entries; vertices with degree > 32 are expanded by the whole warp one at a
// time, smaller ones edge-balanced across the warp through a warp scan.
template <int W>
struct PushSmem {
  int64_t beg[kWarpsPerBlock][32];
  int32_t inc[kWarpsPerBlock][32];
  uint64_t f[kWarpsPerBlock][32][W];
};

template <int W, typename OT, int DEPTH>
__device__ __forceinline__ void bfs_push_tiles(const GroupDev& g, const DevGraph& G, unsigned bid,
                                               unsigned nblk, PushSmem<W>& sm,
                                               bool sweep = false) {
  int64_t (&s_beg)[kWarpsPerBlock][32] = sm.beg;
  int32_t (&s_inc)[kWarpsPerBlock][32] = sm.inc;
  uint64_t (&s_f)[kWarpsPerBlock][32][W] = sm.f;
  const LevelCtl* ctl = g.ctl;
  if (ctl->done || ctl->dir != kDirPush) return;
  const LevelView lv = level_view(g);
  WarpAppender ap;
  const unsigned long long n = ctl->count[lv.par];
  const int64_t light = push_light_limit(g, G, n, ctl->edges[lv.par]);
  uint64_t sel[W];
#pragma unroll
  for (int i = 0; i < W; ++i) sel[i] = ctl->bfs_bits[i] & ctl->expand[i];
  if (!mask_any<W>(sel)) return;

  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const unsigned long long gw = (static_cast<unsigned long long>(bid) * blockDim.x + threadIdx.x) >> 5;
  const unsigned long long nw = (static_cast<unsigned long long>(nblk) * blockDim.x) >> 5;
  uint64_t uni[W];
#pragma unroll
  for (int i = 0; i < W; ++i) uni[i] = 0;
  unsigned long long pairs = 0;

  const int tw = tile_width(n, nw);
  for (unsigned long long tile = gw; tile * tw < n; tile += nw) {
    const unsigned long long idx = tile * tw + lane;
    const bool valid = lane < tw && idx < n;
    int32_t u = valid ? lv.list[idx] : 0;
    int64_t beg = 0, end = 0;
    uint64_t f[W];
#pragma unroll
    for (int i = 0; i < W; ++i) f[i] = 0;
    if (valid) {
      beg = row_at<OT>(G.row, u);
      end = row_at<OT>(G.row, static_cast<int64_t>(u) + 1);
      load_mask<W>(lv.fcur + static_cast<size_t>(u) * W, f);
#pragma unroll
      for (int i = 0; i < W; ++i) f[i] &= sel[i];
      if (sweep) {  // no one else reads the mask: the buffer is clean for level + 1
        uint64_t z[W];
#pragma unroll
        for (int i = 0; i < W; ++i) z[i] = 0;
        store_mask<W>(const_cast<uint64_t*>(lv.fcur) + static_cast<size_t>(u) * W, z);
      }
    }
    const int64_t deg = end - beg;
    const bool work = valid && mask_any<W>(f) && deg > 0 && deg <= light;

    unsigned big = __ballot_sync(kFull, work && deg > 32);
    while (big) {
      const int src = __ffs(big) - 1;
      big &= big - 1;
      const int64_t bb = __shfl_sync(kFull, beg, src);
      const int64_t be = __shfl_sync(kFull, end, src);
      uint64_t bf[W];
#pragma unroll
      for (int i = 0; i < W; ++i) bf[i] = __shfl_sync(kFull, f[i], src);
      for (int64_t e0 = bb; e0 < be; e0 += 32) {
        const int64_t e = e0 + lane;
        int32_t nb = 0;
        bool app = false;
        if (e < be) {
          nb = G.col[e];
          app = bfs_visit<W, DEPTH>(g, G.V, lv, nb, bf, uni, pairs);
        }
        ap.add<OT>(app, nb, G, lv, lane);
      }
    }

    int sdeg = (work && deg <= 32) ? static_cast<int>(deg) : 0;
    int inc = sdeg;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int t = __shfl_up_sync(kFull, inc, o);
      if (lane >= o) inc += t;
    }
    const int total = __shfl_sync(kFull, inc, 31);
    if (total == 0) continue;
    s_beg[wib][lane] = beg;
    s_inc[wib][lane] = inc;
#pragma unroll
    for (int i = 0; i < W; ++i) s_f[wib][lane][i] = f[i];
    __syncwarp();
    for (int b0 = 0; b0 < total; b0 += 32) {
      const int p = b0 + lane;
      int32_t nb = 0;
      bool app = false;
      if (p < total) {
        int lo = 0, hi = 31;
        while (lo < hi) {
          int mid = (lo + hi) >> 1;
          if (s_inc[wib][mid] > p) hi = mid;
          else lo = mid + 1;
        }
        const int start = lo ? s_inc[wib][lo - 1] : 0;
        const int64_t e = s_beg[wib][lo] + (p - start);
        uint64_t of[W];
#pragma unroll
        for (int i = 0; i < W; ++i) of[i] = s_f[wib][lo][i];
        nb = G.col[e];
        app = bfs_visit<W, DEPTH>(g, G.V, lv, nb, of, uni, pairs);
      }
      ap.add<OT>(app, nb, G, lv, lane);
    }
    __syncwarp();
  }
  ap.flush<OT>(G, lv, lane);
  flush_union<W>(uni, lv.nactive, lane);
  warp_add(pairs, &g.ctl->lc.new_pairs, lane);
}

template <int W, typename OT, int DEPTH>
__global__ void __launch_bounds__(kBlock) k_bfs_push(GroupDev g, DevGraph G) {
  __shared__ PushSmem<W> sm;
  bfs_push_tiles<W, OT, DEPTH>(g, G, blockIdx.x, gridDim.x, sm);
}

// Heavy frontier queue.  At the start of a push level the frontier list is
// scanned once and every vertex of degree > heavy_degree is queued with its
// range of kHeavyChunk-edge chunks; one 64-bit atomicAdd hands out both the
// queue slot (high bits) and the first chunk (low bits), so chunk starts grow
// with the slot and a chunk finds its vertex by binary search.  The heavy
// push kernels then visit only the heavy vertices of this frontier instead of
// every heavy vertex of the graph.
constexpr int kQueueShift = 40;

template <typename OT>
__device__ __forceinline__ void heavy_queue_scan(const GroupDev& g, const DevGraph& G,
                                                 unsigned bid, unsigned nblk) {
  LevelCtl* ctl = g.ctl;
  if (ctl->done || ((ctl->dir != kDirPush || !ctl->has_bfs) && !ctl->sscatter)) return;
  const LevelView lv = level_view(g);
  const unsigned long long n = ctl->count[lv.par];
  const int64_t light = push_light_limit(g, G, n, ctl->edges[lv.par]);
  for (unsigned long long i = static_cast<unsigned long long>(bid) * blockDim.x + threadIdx.x;
       i < n; i += static_cast<unsigned long long>(nblk) * blockDim.x) {
    const int32_t u = lv.list[i];
    const int64_t deg = row_at<OT>(G.row, static_cast<int64_t>(u) + 1) - row_at<OT>(G.row, u);
    if (deg <= light) continue;
    const unsigned long long chunks = static_cast<unsigned long long>((deg + kHeavyChunk - 1) / kHeavyChunk);
    const unsigned long long old = atomicAdd(&ctl->hq_packed, (1ULL << kQueueShift) | chunks);
    const unsigned long long slot = old >> kQueueShift;
    if (slot >= static_cast<unsigned long long>(g.hq_cap)) {  // cannot happen with unique lists
      atomicOr(&ctl->status, kStatusQueueOverflow);
      continue;
    }
    g.hq_vertex[slot] = u;
    g.hq_start[slot] = static_cast<int64_t>(old & ((1ULL << kQueueShift) - 1));
  }
}

template <typename OT>
__global__ void __launch_bounds__(kBlock) k_heavy_queue(GroupDev g, DevGraph G) {
  heavy_queue_scan<OT>(g, G, blockIdx.x, gridDim.x);
}

// Queue slot of chunk c (the last slot whose first chunk is <= c).
__device__ __forceinline__ int heavy_queue_slot(const GroupDev& g, int nq, int64_t c) {
  int lo = 0, hi = nq - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (g.hq_start[mid] <= c) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Push level, heavy frontier vertices: the static heavy list is cut into
// kHeavyChunk-edge work items spread over all CTAs.
struct HeavySlotSmem {
  int32_t h;
};

template <int W, typename OT, int DEPTH>
__device__ __forceinline__ void bfs_push_chunks(const GroupDev& g, const DevGraph& G, unsigned bid,
                                                unsigned nblk, HeavySlotSmem& sm) {
  int32_t& s_h = sm.h;
  const LevelCtl* ctl = g.ctl;
  if (ctl->done || ctl->dir != kDirPush) return;
  const unsigned long long hq = ctl->hq_packed;
  const int nq = static_cast<int>(min(static_cast<long long>(hq >> kQueueShift),
                                      static_cast<long long>(g.hq_cap)));
  const int64_t nchunks = static_cast<int64_t>(hq & ((1ULL << kQueueShift) - 1));
  if (nq == 0) return;
  const LevelView lv = level_view(g);
  WarpAppender ap;
  const int lane = threadIdx.x & 31;
  uint64_t uni[W];
#pragma unroll
  for (int i = 0; i < W; ++i) uni[i] = 0;
  unsigned long long pairs = 0;
  for (int64_t c = bid; c < nchunks; c += nblk) {
    if (threadIdx.x == 0) s_h = heavy_queue_slot(g, nq, c);
    __syncthreads();
    const int h = s_h;
    __syncthreads();
    const int32_t u = g.hq_vertex[h];
    uint64_t f[W];
    load_mask<W>(lv.fcur + static_cast<size_t>(u) * W, f);
#pragma unroll
    for (int i = 0; i < W; ++i) f[i] &= ctl->bfs_bits[i] & ctl->expand[i];
    if (!mask_any<W>(f)) continue;
    const int64_t beg = row_at<OT>(G.row, u);
    const int64_t end = row_at<OT>(G.row, static_cast<int64_t>(u) + 1);
    const int64_t cb = beg + (c - g.hq_start[h]) * kHeavyChunk;
    const int64_t ce = min(end, cb + kHeavyChunk);
    for (int64_t e0 = cb + (threadIdx.x & ~31); e0 < ce; e0 += blockDim.x) {
      const int64_t e = e0 + lane;
      int32_t nb = 0;
      bool app = false;
      if (e < ce) {
        nb = G.col[e];
        app = bfs_visit<W, DEPTH>(g, G.V, lv, nb, f, uni, pairs);
      }
      ap.add<OT>(app, nb, G, lv, lane);
    }
  }
  ap.flush<OT>(G, lv, lane);
  flush_union<W>(uni, lv.nactive, lane);
  warp_add(pairs, &g.ctl->lc.new_pairs, lane);
}

template <int W, typename OT, int DEPTH>
__global__ void __launch_bounds__(kBlock) k_bfs_push_heavy(GroupDev g, DevGraph G) {
  __shared__ HeavySlotSmem sm;
  bfs_push_chunks<W, OT, DEPTH>(g, G, blockIdx.x, gridDim.x, sm);
}

// Which light-vertex pull form a BFS pull level uses.  The chunked form
// (k_bfs_pull_chunked) keeps 32 in-edges in flight per warp but checks early
// exit once per 32-edge batch; the lane-per-vertex form (k_bfs_pull) stops a
// vertex after the first in-edges that cover its needed bits.  The chunked
// form runs where few vertices stop early: the first pull level after push
// levels (bits are still rare, almost every in-edge is read) and levels after
// a pull level that read at least half of the in-edges.
__device__ __forceinline__ bool bfs_pull_chunked_level(const LevelCtl* ctl, int64_t E) {
  if (ctl->bfs_chunked != 1) return false;
  return ctl->prev_dir != kDirPull || 2 * ctl->prev_pull_edges >= static_cast<unsigned long long>(E);
}

// Zeroes the next-frontier buffer where the previous frontier left bits
// (exactly the vertices of that frontier's list).  Push levels only: a pull
// level rewrites every vertex's next mask.
template <int W>
__device__ __forceinline__ void clear_next(const GroupDev& g, int64_t E, unsigned bid,
                                           unsigned nblk) {
  const LevelCtl* ctl = g.ctl;
  if (ctl->done) return;
  // a lane-per-vertex pull level in vertex order rewrites every vertex's next
  // mask; the chunked one and the in-degree-ordered one (which skips vertices
  // without in-edges) write only the vertices they pull
  if (ctl->dir != kDirPush && !bfs_pull_chunked_level(ctl, E) && ctl->bfs_chunked != 2) return;
  const LevelView lv = level_view(g);
  const unsigned long long n = ctl->prev_count;
  const int32_t* plist = lv.nlist;  // list of the previous frontier
  for (unsigned long long i = static_cast<unsigned long long>(bid) * blockDim.x + threadIdx.x;
       i < n; i += static_cast<unsigned long long>(nblk) * blockDim.x) {
    uint64_t z[W];
#pragma unroll
    for (int k = 0; k < W; ++k) z[k] = 0;
    store_mask<W>(lv.fnext + static_cast<size_t>(plist[i]) * W, z);
  }
}

template <int W>
__global__ void __launch_bounds__(kBlock) k_clear_next(GroupDev g, int64_t E) {
  clear_next<W>(g, E, blockIdx.x, gridDim.x);
}

// --------------------------------------------------------------- BFS pull
// Lanes that share one vertex mask in the pull kernels, 16 bytes each, for masks
// of 64 bytes and more: a lane that loads a whole mask holds it three times over
// (needed, found, loaded words) and asks for its line once per 16 bytes.
// Chung-Lu 300K, 501 BFS in 8 words: the batch 12.5 -> 11.6 ms.  At 32 bytes a
// lane per mask is the faster one (R-MAT 20, 256 slots, light vertices of the
// first pull level: 138 us against 215 with two lanes, which keep half as many
// lists in flight).
template <int W>
struct PullLanes {
  static constexpr int kLanes = W >= 8 ? W / 2 : 1;    // lanes per mask
  static constexpr int kWords = W / kLanes;            // words per lane
  static constexpr int kGroups = 32 / kLanes;          // masks per warp load
};

// Finishes one lane's part of a pulled vertex (words w0 .. of its mask): writes
// its next mask, visited and depth.
template <int W, int DEPTH, int WL>
__device__ __forceinline__ void pull_commit(const GroupDev& g, int64_t V, const LevelView& lv,
                                            int32_t v, int w0, const uint64_t (&vis)[WL],
                                            const uint64_t (&nw)[WL], uint64_t (&uni)[WL],
                                            unsigned long long& pairs) {
  store_mask<WL>(lv.fnext + static_cast<size_t>(v) * W + w0, nw);
  if (!mask_any<WL>(nw)) return;
  uint64_t nv[WL];
#pragma unroll
  for (int i = 0; i < WL; ++i) {
    nv[i] = vis[i] | nw[i];
    uni[i] |= nw[i];
    pairs += __popcll(nw[i]);
  }
  store_mask<WL>(g.visited + static_cast<size_t>(v) * W + w0, nv);
  record_depth<W, DEPTH, WL>(g, V, v, w0, nw, lv.level + 1, true);
  // a later SSSP push of the same level must not append v a second time
  g.stamp[v] = lv.level + 1;
}

// ORs the lanes' parts over the lanes with the same words (sub = lane %
// kLanes): every lane gets its words' union.  All lanes call.
template <int W>
__device__ __forceinline__ void part_or_reduce(uint64_t (&m)[PullLanes<W>::kWords]) {
  using PL = PullLanes<W>;
  if constexpr (PL::kLanes == 1) {
    warp_or_reduce<W>(m);
  } else {
#pragma unroll
    for (int o = 16; o >= PL::kLanes; o >>= 1) {
#pragma unroll
      for (int i = 0; i < PL::kWords; ++i) m[i] |= __shfl_xor_sync(kFull, m[i], o);
    }
  }
}

// ORs the lanes' unions into the level's active words (see flush_union).
template <int W>
__device__ __forceinline__ void flush_union_parts(uint64_t (&uni)[PullLanes<W>::kWords],
                                                  uint64_t* dst, int lane) {
  using PL = PullLanes<W>;
  part_or_reduce<W>(uni);
  if (lane < PL::kLanes) {
#pragma unroll
    for (int i = 0; i < PL::kWords; ++i)
      if (uni[i]) atomic_or64(dst + lane * PL::kWords + i, uni[i]);
  }
}

// The lane's words of the bits that may still be found at this level.
template <int W>
__device__ __forceinline__ void pull_active(const LevelCtl* ctl, int par, int w0,
                                            uint64_t (&act)[PullLanes<W>::kWords]) {
#pragma unroll
  for (int i = 0; i < PullLanes<W>::kWords; ++i)
    act[i] = ctl->active[par][w0 + i] & ctl->bfs_bits[w0 + i] & ctl->expand[w0 + i];
}

// A pull level whose frontier holds fewer than 1/16 of the vertices screens
// in-edges by the frontier summary: a source outside the frontier costs an
// 8-byte word that stays in L2 instead of its W-word mask.
__device__ __forceinline__ bool bfs_pull_uses_summary(const GroupDev& g, const LevelCtl* ctl,
                                                      const LevelView& lv, int64_t V) {
  return g.fsum != nullptr && ctl->dir == kDirPull &&
         16ULL * ctl->count[lv.par] < static_cast<unsigned long long>(V);
}

// Pull level (bottom-up): every non-heavy vertex with unvisited active bits
// ORs the current-frontier masks of its in-neighbours until every needed bit
// is found (early exit).  Reads only the current frontier, so depths are
// exactly level-synchronous.  Vertex order by default (a tile is kGroups
// consecutive vertices); with bfs_chunked == 2 the tiles run over the light
// table's vertices of in-degree 1..mid_degree (8 or 32) in decreasing in-degree
// order, so the lanes of a warp walk lists of about the same length (the next
// masks of the vertices left out are zeroed by k_clear_next).
template <int W, typename OT, int DEPTH>
__device__ __forceinline__ void bfs_pull_tiles(const GroupDev& g, const DevGraph& G, unsigned bid,
                                               unsigned nblk) {
  using PL = PullLanes<W>;
  constexpr int LP = PL::kLanes;
  constexpr int WL = PL::kWords;
  const LevelCtl* ctl = g.ctl;
  if (ctl->done || ctl->dir != kDirPull) return;
  if (G.n_plight_chunks > 0 && bfs_pull_chunked_level(ctl, G.E)) return;
  const LevelView lv = level_view(g);
  const int lane = threadIdx.x & 31;
  const int sub = lane % LP;   // this lane's words: w0 .. w0 + WL
  const int w0 = sub * WL;
  const unsigned group = ((LP < 32 ? (1u << LP) : 0u) - 1u) << (lane - sub);
  uint64_t act[WL];
  pull_active<W>(ctl, lv.par, w0, act);
  const unsigned long long gw = (static_cast<unsigned long long>(bid) * blockDim.x + threadIdx.x) >> 5;
  const unsigned long long nwarps = (static_cast<unsigned long long>(nblk) * blockDim.x) >> 5;
  const unsigned long long V = static_cast<unsigned long long>(G.V);
  const bool use_sum = bfs_pull_uses_summary(g, ctl, lv, G.V);
  uint64_t uni[WL];
#pragma unroll
  for (int i = 0; i < WL; ++i) uni[i] = 0;
  unsigned long long pairs = 0, pverts = 0, pedges = 0;
  const bool sorted = ctl->bfs_chunked == 2;
  // tiles over vertex ids, or over the light table's entries n_pmid .. end
  const unsigned long long n_items =
      sorted ? static_cast<unsigned long long>(G.plight_chunk_start[G.n_plight_chunks] - G.n_pmid) : V;

  for (unsigned long long tile = gw; tile * PL::kGroups < n_items; tile += nwarps) {
    const unsigned long long vv = tile * PL::kGroups + lane / LP;
    const bool valid = vv < n_items;
    const int32_t v = !valid ? 0 : sorted ? G.plight[G.n_pmid + vv] : static_cast<int32_t>(vv);
    uint64_t need[WL], acc[WL];
    int64_t beg = 0, end = 0;
#pragma unroll
    for (int i = 0; i < WL; ++i) {
      need[i] = 0;
      acc[i] = 0;
    }
    if (valid) {
      beg = row_at<OT>(G.prow, v);
      end = row_at<OT>(G.prow, static_cast<int64_t>(v) + 1);
      uint64_t vis[WL];
      load_mask<WL>(g.visited + static_cast<size_t>(v) * W + w0, vis);
#pragma unroll
      for (int i = 0; i < WL; ++i) need[i] = ~vis[i] & act[i];
    }
    const int64_t deg = end - beg;
    // heavy lists are the heavy kernels'; lists of mid_degree + 1 .. heavy_degree
    // in-edges are k_bfs_pull_mid's when the light table lists them
    const bool heavy = deg > G.heavy_degree || (G.n_pmid > 0 && deg > G.mid_degree);
    const bool wants = mask_any<WL>(need);
    const unsigned want_lanes = __ballot_sync(kFull, wants);
    const bool open = (want_lanes & group) != 0;  // some lane of the vertex
    const bool work = valid && !heavy && deg > 0 && open;
    pverts += work && sub == 0 ? 1 : 0;
    int walked = 0;  // in-edges this lane's words needed
    if (work && wants && deg <= 32) {
      const uint32_t nch = chunk_bits<WL>(need) << (2 * w0);
      // four in-edges per step: their column and mask loads are independent
      // and stay in flight together; each lane stops once its own words are
      // found (and the next step's columns are loaded a step ahead)
      int32_t un[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) un[j] = (beg + j < end) ? G.pcol[beg + j] : -1;
      for (int64_t e = beg; e < end; e += 4) {
        int32_t us[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          us[j] = un[j];
          un[j] = (e + 4 + j < end) ? G.pcol[e + 4 + j] : -1;
        }
        if (use_sum) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (us[j] >= 0 && !(summary_chunks(g.fsum, lv.level, us[j]) & nch)) us[j] = -1;
        }
        walked += end - e < 4 ? static_cast<int>(end - e) : 4;
        bool full = true;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (us[j] < 0) continue;
          uint64_t fu[WL];
          load_mask<WL>(lv.fcur + static_cast<size_t>(us[j]) * W + w0, fu);
#pragma unroll
          for (int i = 0; i < WL; ++i) acc[i] |= fu[i] & need[i];
        }
#pragma unroll
        for (int i = 0; i < WL; ++i) full &= acc[i] == need[i];
        if (full) break;
      }
    }
    // a vertex's in-edges count once: as far as the lane that needed most went
#pragma unroll
    for (int o = LP / 2; o > 0; o >>= 1) walked = max(walked, __shfl_xor_sync(kFull, walked, o));
    if (sub == 0) pedges += static_cast<unsigned long long>(walked);
    // longer lists, where no kernel of their own takes them: the warp per
    // vertex, kGroups in-edges per step
    unsigned big = __ballot_sync(kFull, work && deg > 32 && sub == 0);
    while (big) {
      const int src = __ffs(big) - 1;  // lane of the vertex's first words
      big &= big - 1;
      const int64_t bb = __shfl_sync(kFull, beg, src);
      const int64_t be = __shfl_sync(kFull, end, src);
      uint64_t bn[WL], a[WL];
#pragma unroll
      for (int i = 0; i < WL; ++i) {
        bn[i] = __shfl_sync(kFull, need[i], src + sub);
        a[i] = 0;
      }
      const uint32_t bch = chunk_bits<WL>(bn) << (2 * w0);
      for (int64_t e0 = bb; e0 < be; e0 += PL::kGroups) {
        const int64_t e = e0 + lane / LP;
        if (e < be) {
          if (sub == 0) ++pedges;
          const int32_t u = G.pcol[e];
          if (!use_sum || (summary_chunks(g.fsum, lv.level, u) & bch)) {
            uint64_t fu[WL];
            load_mask<WL>(lv.fcur + static_cast<size_t>(u) * W + w0, fu);
#pragma unroll
            for (int i = 0; i < WL; ++i) a[i] |= fu[i] & bn[i];
          }
        }
        part_or_reduce<W>(a);
        bool full = true;
#pragma unroll
        for (int i = 0; i < WL; ++i) full &= a[i] == bn[i];
        if (__all_sync(kFull, full)) break;
      }
      if (lane - sub == src) {
#pragma unroll
        for (int i = 0; i < WL; ++i) acc[i] = a[i];
      }
    }
    bool found = false;
    if (valid && !heavy) {
      uint64_t nwm[WL], vis[WL];
#pragma unroll
      for (int i = 0; i < WL; ++i) nwm[i] = acc[i] & need[i];
      // visited again (this warp's vertex: unchanged since the tile began);
      // not kept in registers across the in-edge loop
      load_mask<WL>(g.visited + static_cast<size_t>(v) * W + w0, vis);
      pull_commit<W, DEPTH, WL>(g, G.V, lv, v, w0, vis, nwm, uni, pairs);
      found = mask_any<WL>(nwm);
    }
    const unsigned new_lanes = __ballot_sync(kFull, found);
    const bool app = sub == 0 && (new_lanes & group) != 0;
    warp_append(app, v, static_cast<uint64_t>(deg), lv.nlist, lv.ncount, lv.nedges, lane);
  }
  flush_union_parts<W>(uni, lv.nactive, lane);
  warp_add(pairs, &g.ctl->lc.new_pairs, lane);
  warp_add(pverts, &g.ctl->lc.pull_vertices, lane);
  warp_add(pedges, &g.ctl->lc.pull_edges, lane);
}

template <int W, typename OT, int DEPTH>
__global__ void __launch_bounds__(kBlock, 3) k_bfs_pull(GroupDev g, DevGraph G) {
  bfs_pull_tiles<W, OT, DEPTH>(g, G, blockIdx.x, gridDim.x);
}

// Pull level (bottom-up), light vertices in CTA chunks of the pull CSR's light
// chunk table (<= kLightChunkVerts vertices, <= kLightChunkEdges in-edges):
// the CTA's warps split the chunk's in-edges evenly across vertex boundaries,
// each lane loads one in-edge's source frontier mask and ORs its needed bits
// into the vertex's accumulator in shared memory; before a batch a lane skips
// its in-edge once the vertex's accumulator covers its need (early exit per
// 32-edge batch).  After a barrier each vertex is committed once: next-frontier
// words (cleared beforehand by k_clear_next), visited, depth, stamp, append.
// Reads only the current frontier, so depths stay exactly level-synchronous.
template <int W, typename OT, int DEPTH>
__global__ void __launch_bounds__(kBlock) k_bfs_pull_chunked(GroupDev g, DevGraph G) {
  const LevelCtl* ctl = g.ctl;
  if (ctl->done || ctl->dir != kDirPull || G.n_plight_chunks == 0 ||
      !bfs_pull_chunked_level(ctl, G.E))
    return;
  const LevelView lv = level_view(g);
  __shared__ int32_t s_v[kLightChunkVerts];
  __shared__ int64_t s_beg[kLightChunkVerts];
  __shared__ int32_t s_pre[kLightChunkVerts + 1];
  __shared__ unsigned long long s_need[kLightChunkVerts][W];
  __shared__ unsigned long long s_acc[kLightChunkVerts][W];
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  uint64_t act[W];
#pragma unroll
  for (int i = 0; i < W; ++i)
    act[i] = ctl->active[lv.par][i] & ctl->bfs_bits[i] & ctl->expand[i];
  const bool use_sum = bfs_pull_uses_summary(g, ctl, lv, G.V);
  WarpAppender ap;
  uint64_t uni[W];
#pragma unroll
  for (int i = 0; i < W; ++i) uni[i] = 0;
  unsigned long long pairs = 0, pverts = 0, pedges = 0;
  for (int c = blockIdx.x; c < G.n_plight_chunks; c += gridDim.x) {
    const int cs = G.plight_chunk_start[c];
    const int nv = G.plight_chunk_start[c + 1] - cs;
    if (wib == 0) {
      int32_t v = 0;
      int64_t b = 0;
      int d = 0;
      if (lane < nv) {
        v = G.plight[cs + lane];
        b = row_at<OT>(G.prow, v);
        uint64_t vis[W];
        load_mask<W>(g.visited + static_cast<size_t>(v) * W, vis);
        bool any = false;
#pragma unroll
        for (int i = 0; i < W; ++i) {
          const uint64_t nd = ~vis[i] & act[i];
          s_need[lane][i] = nd;
          s_acc[lane][i] = 0;
          any |= nd != 0;
        }
        // a vertex that needs nothing contributes no in-edges to the walk
        d = any ? static_cast<int>(row_at<OT>(G.prow, static_cast<int64_t>(v) + 1) - b) : 0;
        pverts += any ? 1 : 0;
      }
      int inc = d;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(kFull, inc, o);
        if (lane >= o) inc += t;
      }
      if (lane < nv) {
        s_v[lane] = v;
        s_beg[lane] = b;
        s_pre[lane + 1] = inc;
      }
      if (lane == 0) s_pre[0] = 0;
    }
    __syncthreads();
    const int total = s_pre[nv];
    const int seg = (total + kWarpsPerBlock - 1) / kWarpsPerBlock;
    const int fa = min(total, wib * seg);
    const int fb = min(total, fa + seg);
    for (int f0 = fa; f0 < fb; f0 += 32) {
      const int f = f0 + lane;
      if (f < fb) {
        int lo = 0, hi = nv - 1;  // owner: last k with s_pre[k] <= f
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (s_pre[mid] <= f) lo = mid;
          else hi = mid - 1;
        }
        const int k = lo;
        uint64_t nd[W];
        bool open = false;
#pragma unroll
        for (int i = 0; i < W; ++i) {
          nd[i] = s_need[k][i];
          open |= (s_acc[k][i] & nd[i]) != nd[i];
        }
        if (open) {
          ++pedges;
          const int32_t u = G.pcol[s_beg[k] + (f - s_pre[k])];
          if (!use_sum || (summary_chunks(g.fsum, lv.level, u) & chunk_bits<W>(nd))) {
            uint64_t fu[W];
            load_mask<W>(lv.fcur + static_cast<size_t>(u) * W, fu);
#pragma unroll
            for (int i = 0; i < W; ++i) {
              const uint64_t x = fu[i] & nd[i];
              if (x) atomicOr(&s_acc[k][i], static_cast<unsigned long long>(x));
            }
          }
        }
      }
    }
    __syncthreads();
    // commit: warp wib takes vertices wib, wib + 8, ... (lane 0 of the warp)
    for (int k = wib; k < nv; k += kWarpsPerBlock) {
      bool app = false;
      const int32_t v = s_v[k];
      if (lane == 0) {
        uint64_t nw[W], vis[W];
        bool any = false;
#pragma unroll
        for (int i = 0; i < W; ++i) {
          nw[i] = s_acc[k][i] & s_need[k][i];
          any |= nw[i] != 0;
        }
        if (any) {
          load_mask<W>(g.visited + static_cast<size_t>(v) * W, vis);
          uint64_t nv2[W];
#pragma unroll
          for (int i = 0; i < W; ++i) {
            nv2[i] = vis[i] | nw[i];
            uni[i] |= nw[i];
            pairs += __popcll(nw[i]);
          }
          store_mask<W>(g.visited + static_cast<size_t>(v) * W, nv2);
          store_mask<W>(lv.fnext + static_cast<size_t>(v) * W, nw);
          record_depth<W, DEPTH, W>(g, G.V, v, 0, nw, lv.level + 1, true);
          app = g.stamp[v] < lv.level + 1;
          g.stamp[v] = lv.level + 1;
        }
      }
      ap.add<OT>(app, v, G, lv, lane);
    }
    __syncthreads();
  }
  ap.flush<OT>(G, lv, lane);
  flush_union<W>(uni, lv.nactive, lane);
  warp_add(pairs, &g.ctl->lc.new_pairs, lane);
  warp_add(pverts, &g.ctl->lc.pull_vertices, lane);
  warp_add(pedges, &g.ctl->lc.pull_edges, lane);
}

// Pull level, vertices with mid_degree + 1 .. heavy_degree in-edges (the first n_pmid
// entries of the pull CSR's light table, largest first): a warp per vertex,
// 64 in-edges per step (two column -> mask loads in flight per lane, then a
// warp OR-reduce and the early-exit test), one commit per vertex.  In the
// lane-per-vertex tile kernel these lists were a warp's serial work with one
// 32-edge step in flight; here they have a kernel and a register budget of
// their own.  Every listed vertex's next mask is written (zero when nothing
// is new), as the tile kernel does for its vertices.
template <int W, typename OT, int DEPTH>
__device__ __forceinline__ void bfs_pull_mid(const GroupDev& g, const DevGraph& G, unsigned bid,
                                             unsigned nblk) {
  using PL = PullLanes<W>;
  constexpr int LP = PL::kLanes;
  constexpr int WL = PL::kWords;
  constexpr int kLoads = LP > 2 ? 2 : LP;  // loads in flight per 32 columns
  const LevelCtl* ctl = g.ctl;
  if (ctl->done || ctl->dir != kDirPull || G.n_pmid == 0) return;
  if (G.n_plight_chunks > 0 && bfs_pull_chunked_level(ctl, G.E)) return;
  const LevelView lv = level_view(g);
  const int lane = threadIdx.x & 31;
  const int sub = lane % LP;
  const int w0 = sub * WL;
  uint64_t act[WL];
  pull_active<W>(ctl, lv.par, w0, act);
  const bool use_sum = bfs_pull_uses_summary(g, ctl, lv, G.V);
  const long long gw = (static_cast<long long>(bid) * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = (static_cast<long long>(nblk) * blockDim.x) >> 5;
  WarpAppender ap;
  uint64_t uni[WL];
#pragma unroll
  for (int i = 0; i < WL; ++i) uni[i] = 0;
  unsigned long long pairs = 0, pverts = 0, pedges = 0;
  for (long long i = gw; i < G.n_pmid; i += nwarps) {
    const int32_t v = G.plight[i];
    uint64_t vis[WL], need[WL], a[WL];
    load_mask<WL>(g.visited + static_cast<size_t>(v) * W + w0, vis);
#pragma unroll
    for (int k = 0; k < WL; ++k) {
      need[k] = ~vis[k] & act[k];
      a[k] = 0;
    }
    if (__any_sync(kFull, mask_any<WL>(need))) {
      if (lane == 0) ++pverts;
      const int64_t beg = row_at<OT>(G.prow, v);
      const int64_t end = row_at<OT>(G.prow, static_cast<int64_t>(v) + 1);
      const uint32_t nch = chunk_bits<WL>(need) << (2 * w0);
      // lane l holds columns l and 32 + l of a step of 64; the next step's are
      // in flight while this one's masks load
      int32_t n0 = -1, n1 = -1;
      if (beg + lane < end) n0 = G.pcol[beg + lane];
      if (beg + 32 + lane < end) n1 = G.pcol[beg + 32 + lane];
      for (int64_t e0 = beg; e0 < end; e0 += 64) {
        const int32_t c0 = n0, c1 = n1;
        n0 = n1 = -1;
        if (e0 + 64 + lane < end) n0 = G.pcol[e0 + 64 + lane];
        if (e0 + 96 + lane < end) n1 = G.pcol[e0 + 96 + lane];
        pedges += (c0 >= 0 ? 1 : 0) + (c1 >= 0 ? 1 : 0);
        // the columns, kGroups of them at a time, each by its kLanes lanes
#pragma unroll
        for (int j0 = 0; j0 < LP; j0 += kLoads) {
          int32_t u[2 * kLoads];
#pragma unroll
          for (int j = 0; j < kLoads; ++j) {
            const int at = (j0 + j) * PL::kGroups + lane / LP;
            u[2 * j] = __shfl_sync(kFull, c0, at);
            u[2 * j + 1] = __shfl_sync(kFull, c1, at);
          }
          if (use_sum) {
#pragma unroll
            for (int j = 0; j < 2 * kLoads; ++j)
              if (u[j] >= 0 && !(summary_chunks(g.fsum, lv.level, u[j]) & nch)) u[j] = -1;
          }
          uint64_t f[2 * kLoads][WL];
#pragma unroll
          for (int j = 0; j < 2 * kLoads; ++j) {
#pragma unroll
            for (int k = 0; k < WL; ++k) f[j][k] = 0;
            if (u[j] >= 0) load_mask<WL>(lv.fcur + static_cast<size_t>(u[j]) * W + w0, f[j]);
          }
#pragma unroll
          for (int j = 0; j < 2 * kLoads; ++j) {
#pragma unroll
            for (int k = 0; k < WL; ++k) a[k] |= f[j][k] & need[k];
          }
        }
        part_or_reduce<W>(a);
        bool full = true;
#pragma unroll
        for (int k = 0; k < WL; ++k) full &= a[k] == need[k];
        if (__all_sync(kFull, full)) break;
      }
    }
    bool found = false;
    if (lane < LP) {  // the first lane of every part
      uint64_t nw[WL];
#pragma unroll
      for (int k = 0; k < WL; ++k) nw[k] = a[k] & need[k];
      pull_commit<W, DEPTH, WL>(g, G.V, lv, v, w0, vis, nw, uni, pairs);
      found = mask_any<WL>(nw);
    }
    const bool any = __any_sync(kFull, found);
    ap.add<OT>(any && lane == 0, v, G, lv, lane);
  }
  ap.flush<OT>(G, lv, lane);
  flush_union_parts<W>(uni, lv.nactive, lane);
  warp_add(pairs, &g.ctl->lc.new_pairs, lane);
  warp_add(pverts, &g.ctl->lc.pull_vertices, lane);
  warp_add(pedges, &g.ctl->lc.pull_edges, lane);
}

template <int W, typename OT, int DEPTH>
__global__ void __launch_bounds__(kBlock, 3) k_bfs_pull_mid(GroupDev g, DevGraph G) {
  bfs_pull_mid<W, OT, DEPTH>(g, G, blockIdx.x, gridDim.x);
}

// Pull level, heavy vertices: chunks of their in-edges spread over CTAs; each
// CTA ORs its chunk into hacc[h] (skipping chunks once hacc covers the need).
template <int W>
struct PullHeavySmem {
  int skip;
  uint64_t red[kWarpsPerBlock][W];
};

template <int W, typename OT>
__device__ __forceinline__ void bfs_pull_chunks(const GroupDev& g, const DevGraph& G, unsigned bid,
                                                unsigned nblk, PullHeavySmem<W>& sm) {
  int& s_skip = sm.skip;
  uint64_t (&s_red)[kWarpsPerBlock][W] = sm.red;
  const LevelCtl* ctl = g.ctl;
  if (ctl->done || ctl->dir != kDirPull || G.n_pheavy == 0) return;
  const LevelView lv = level_view(g);
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  using PL = PullLanes<W>;
  constexpr int LP = PL::kLanes;
  constexpr int WL = PL::kWords;
  const int sub = lane % LP;
  const int w0 = sub * WL;
  for (int64_t c = bid; c < G.pheavy_chunks; c += nblk) {
    __syncthreads();  // the previous chunk's s_skip is read
    const int h = G.pheavy_ch[c];
    const int32_t v = G.pheavy[h];
    uint64_t vis[W], need[W];
    load_mask<W>(g.visited + static_cast<size_t>(v) * W, vis);
    bool anyneed = false;
#pragma unroll
    for (int i = 0; i < W; ++i) {
      need[i] = ~vis[i] & ctl->active[lv.par][i] & ctl->bfs_bits[i] & ctl->expand[i];
      anyneed |= need[i] != 0;
    }
    if (threadIdx.x == 0) {
      bool covered = true;
      const volatile uint64_t* ha = g.hacc + static_cast<size_t>(h) * W;
#pragma unroll
      for (int i = 0; i < W; ++i) covered &= (ha[i] & need[i]) == need[i];
      s_skip = (!anyneed || covered) ? 1 : 0;
    }
    __syncthreads();
    if (s_skip) continue;
    const int64_t cb = G.pheavy_cb[c];
    const int64_t ce = G.pheavy_ce[c];
    uint64_t a[WL], mine[WL];  // this lane's words
#pragma unroll
    for (int i = 0; i < WL; ++i) {
      a[i] = 0;
      mine[i] = 0;
#pragma unroll
      for (int k = 0; k < LP; ++k)
        if (sub == k) mine[i] = need[k * WL + i];
    }
    if (threadIdx.x == 0) atomicAdd(&g.ctl->lc.pull_edges, static_cast<unsigned long long>(ce - cb));
    const bool use_sum = bfs_pull_uses_summary(g, ctl, lv, G.V);
    const uint32_t nch = chunk_bits<WL>(mine) << (2 * w0);
    constexpr int kPer = kBlock / LP;  // in-edges per step of the block
    // two steps' loads in flight
    for (int64_t e = cb + threadIdx.x / LP; e < ce; e += 2 * kPer) {
      int32_t u[2] = {G.pcol[e], e + kPer < ce ? G.pcol[e + kPer] : -1};
      if (use_sum) {
#pragma unroll
        for (int j = 0; j < 2; ++j)
          if (u[j] >= 0 && !(summary_chunks(g.fsum, lv.level, u[j]) & nch)) u[j] = -1;
      }
      uint64_t f[2][WL];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
#pragma unroll
        for (int i = 0; i < WL; ++i) f[j][i] = 0;
        if (u[j] >= 0) load_mask<WL>(lv.fcur + static_cast<size_t>(u[j]) * W + w0, f[j]);
      }
#pragma unroll
      for (int i = 0; i < WL; ++i) a[i] |= (f[0][i] | f[1][i]) & mine[i];
    }
    part_or_reduce<W>(a);
    if (lane < LP) {
#pragma unroll
      for (int i = 0; i < WL; ++i) s_red[wib][w0 + i] = a[i];
    }
    __syncthreads();
    if (threadIdx.x < W) {
      uint64_t r = 0;
      for (int k = 0; k < kWarpsPerBlock; ++k) r |= s_red[k][threadIdx.x];
      if (r) atomic_or64(g.hacc + static_cast<size_t>(h) * W + threadIdx.x, r);
    }
    __syncthreads();
  }
}

template <int W, typename OT>
__global__ void __launch_bounds__(kBlock) k_bfs_pull_heavy(GroupDev g, DevGraph G) {
  __shared__ PullHeavySmem<W> sm;
  bfs_pull_chunks<W, OT>(g, G, blockIdx.x, gridDim.x, sm);
}

// Commits the heavy vertices of a pull level and resets their accumulators.
template <int W, typename OT, int DEPTH>
__device__ __forceinline__ void bfs_pull_heavy_commit(const GroupDev& g, const DevGraph& G,
                                                      unsigned bid, unsigned nblk) {
  const LevelCtl* ctl = g.ctl;
  if (ctl->done || ctl->dir != kDirPull || G.n_pheavy == 0) return;
  const LevelView lv = level_view(g);
  const int lane = threadIdx.x & 31;
  uint64_t uni[W];
#pragma unroll
  for (int i = 0; i < W; ++i) uni[i] = 0;
  unsigned long long pairs = 0, pverts = 0;
  const int64_t stride = static_cast<int64_t>(nblk) * blockDim.x;
  for (int64_t base = static_cast<int64_t>(bid) * blockDim.x + (threadIdx.x & ~31);
       base < G.n_pheavy; base += stride) {
    const int64_t h = base + lane;
    bool app = false;
    int32_t v = 0;
    uint64_t deg = 0;
    if (h < G.n_pheavy) {
      v = G.pheavy[h];
      uint64_t vis[W], nwm[W], acc[W];
      load_mask<W>(g.visited + static_cast<size_t>(v) * W, vis);
      load_mask<W>(g.hacc + static_cast<size_t>(h) * W, acc);
#pragma unroll
      for (int i = 0; i < W; ++i) {
        nwm[i] = acc[i] & ~vis[i] & ctl->active[lv.par][i] & ctl->bfs_bits[i] & ctl->expand[i];
        acc[i] = 0;
      }
      store_mask<W>(g.hacc + static_cast<size_t>(h) * W, acc);
      bool anyneed = false;
#pragma unroll
      for (int i = 0; i < W; ++i)
        anyneed |= (~vis[i] & ctl->active[lv.par][i] & ctl->bfs_bits[i] & ctl->expand[i]) != 0;
      pverts += anyneed ? 1 : 0;
      pull_commit<W, DEPTH, W>(g, G.V, lv, v, 0, vis, nwm, uni, pairs);
      app = mask_any<W>(nwm);
      deg = degree_of<OT>(G.prow, v);
    }
    warp_append(app, v, deg, lv.nlist, lv.ncount, lv.nedges, lane);
  }
  flush_union<W>(uni, lv.nactive, lane);
  warp_add(pairs, &g.ctl->lc.new_pairs, lane);
  warp_add(pverts, &g.ctl->lc.pull_vertices, lane);
}

template <int W, typename OT, int DEPTH>
__global__ void __launch_bounds__(kBlock) k_bfs_pull_heavy_commit(GroupDev g, DevGraph G) {
  bfs_pull_heavy_commit<W, OT, DEPTH>(g, G, blockIdx.x, gridDim.x);
}

// -------------------------------------------------------------- SSSP push
template <int WK>
__device__ __forceinline__ uint32_t relax(uint32_t du, const void* w, int64_t e) {
  if constexpr (WK == kWeightF32) {
    float r = __fadd_rn(__uint_as_float(du), static_cast<const float*>(w)[e]);
    return __float_as_uint(r);
  } else {
    uint32_t wt = (WK == kWeightU32) ? static_cast<const uint32_t*>(w)[e] : 1u;
    return du > 0xffffffffu - wt ? 0xffffffffu : du + wt;
  }
}

// Pairs handled per lane per step by the flattened scatter loops: their column,
// source and destination loads are independent and issued together.
constexpr int kPairSteps = 4;

// Relaxation with the weight already loaded (raw 32-bit pattern).
template <int WK>
__device__ __forceinline__ uint32_t relax_w(uint32_t du, uint32_t wbits) {
  if constexpr (WK == kWeightF32) {
    return __float_as_uint(__fadd_rn(__uint_as_float(du), __uint_as_float(wbits)));
  } else {
    const uint32_t wt = (WK == kWeightU32) ? wbits : 1u;
    return du > 0xffffffffu - wt ? 0xffffffffu : du + wt;
  }
}

template <int WK>
__device__ __forceinline__ uint32_t weight_bits(const void* w, int64_t e) {
  if constexpr (WK == kWeightNone) {
    return 1u;
  } else {
    return static_cast<const uint32_t*>(w)[e];
  }
}

// Vertices with at most this many active SSSP bits are scattered as flattened
// (edge, slot) pairs, those with more as slot lists.  A pair costs a search for
// its vertex and a division (some 80 instructions for 32 pairs); a list step
// (some 14) relaxes up to 32 slots over one edge, so it pays from about 6 on.
constexpr int kListBits = 6;

// Union of the slots improved by a block, one 32-bit word per 32 slots.
template <int W>
struct SlotUnion {
  uint32_t word[2 * W];
};

template <int W>
__device__ __forceinline__ void slot_union_clear(SlotUnion<W>& un) {
  if (threadIdx.x < 2 * W) un.word[threadIdx.x] = 0;
  __syncthreads();
}

// All threads call, after their last improvement.
template <int W>
__device__ __forceinline__ void slot_union_flush(const SlotUnion<W>& un, uint64_t* dst) {
  __syncthreads();
  if (threadIdx.x < 2 * W && un.word[threadIdx.x])
    atomicOr(reinterpret_cast<uint32_t*>(dst) + threadIdx.x, un.word[threadIdx.x]);
}

// Lists the set bits of a vertex's active mask (32-bit half c in lane c, c <
// 2W; 0 in the other lanes) into slots[], ascending; returns how many there
// are.  All lanes call.
__device__ __forceinline__ int list_slots(uint32_t half, int lane, uint16_t* slots) {
  const int mine = __popc(half);
  int inc = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(kFull, inc, o);
    if (lane >= o) inc += t;
  }
  int at = inc - mine;
  while (half) {
    slots[at++] = static_cast<uint16_t>(32 * lane + __ffs(half) - 1);
    half &= half - 1;
  }
  __syncwarp();
  return __shfl_sync(kFull, inc, 31);
}

// Scatters edges [eb, ee) of vertex u for the k slots in slots[] (one warp, all
// lanes call): lane j takes the j-th slot of each run of 32, keeps u's distance
// to it in a register and relaxes U edges per step.  Listed slots ascend, so a
// run of neighbouring slots reads neighbouring words, and a vertex with every
// slot active reads whole rows.
template <int W, typename OT, int WK, int U>
__device__ __forceinline__ void scatter_list(const GroupDev& g, const DevGraph& G,
                                             const LevelView& lv, int32_t u,
                                             const uint16_t* slots, int k, int64_t eb, int64_t ee,
                                             int lane, SlotUnion<W>& un,
                                             unsigned long long& improved, WarpAppender& ap) {
  const size_t Qg = static_cast<size_t>(g.Qg);
  for (int j0 = 0; j0 < k; j0 += 32) {
    const bool on = j0 + lane < k;
    const int q = on ? slots[j0 + lane] : 0;
    const uint32_t du = on ? g.values[static_cast<size_t>(u) * Qg + q] : 0xffffffffu;
    // 32 slots of one aligned chunk: the ballot of the improved lanes is its word
    const int q0 = __shfl_sync(kFull, q, 0);
    const bool chunk = __all_sync(kFull, on && (q0 & 31) == 0 && q == q0 + lane);
    for (int64_t e0 = eb; e0 < ee; e0 += 32) {
      int32_t nl = 0;
      uint32_t wl = 0;
      if (e0 + lane < ee) {
        nl = G.col[e0 + lane];
        wl = weight_bits<WK>(G.w, e0 + lane);
      }
      const int cnt = static_cast<int>(ee - e0 < 32 ? ee - e0 : 32);
      for (int i = 0; i < cnt; i += U) {
        int32_t nb[U];
        uint32_t cand[U], cur[U];
        bool any = false;
#pragma unroll
        for (int t = 0; t < U; ++t) {
          nb[t] = __shfl_sync(kFull, nl, i + t < cnt ? i + t : i);
          const uint32_t w = __shfl_sync(kFull, wl, i + t < cnt ? i + t : i);
          const bool go = on && i + t < cnt;
          cand[t] = go ? relax_w<WK>(du, w) : 0xffffffffu;
          cur[t] = go ? g.values[static_cast<size_t>(nb[t]) * Qg + q] : 0u;
        }
#pragma unroll
        for (int t = 0; t < U; ++t) any |= cand[t] < cur[t];
        if (!__any_sync(kFull, any)) continue;
#pragma unroll
        for (int t = 0; t < U; ++t) {
          bool imp = false;
          if (cand[t] < cur[t])
            imp = cand[t] < atomicMin(g.values + static_cast<size_t>(nb[t]) * Qg + q, cand[t]);
          const unsigned m = __ballot_sync(kFull, imp);
          if (m == 0) continue;
          uint32_t* fw = reinterpret_cast<uint32_t*>(lv.fnext + static_cast<size_t>(nb[t]) * W) + (q >> 5);
          if (chunk) {
            if (lane == 0) {
              atomicOr(fw, m);
              atomicOr(&un.word[q >> 5], m);
            }
          } else if (imp) {
            atomicOr(fw, 1u << (q & 31));
            atomicOr(&un.word[q >> 5], 1u << (q & 31));
          }
          improved += imp ? 1 : 0;
          bool app = false;
          if (lane == 0 && g.stamp[nb[t]] < lv.level + 1)
            app = atomicMax(g.stamp + nb[t], lv.level + 1) < lv.level + 1;
          ap.add<OT>(app, nb[t], G, lv, lane);
        }
      }
    }
  }
}

// One flattened pair's improvement (cand < the value read): atomicMin, frontier
// bit, union and stamp.  True when n must be appended.  Hub destinations
// receive many improvements per level: a plain read of the frontier word and
// of the stamp skips atomics that would change nothing (bits and stamps only
// grow within a level).
template <int W>
__device__ __forceinline__ bool scatter_commit(const GroupDev& g, const LevelView& lv, int32_t n,
                                               int q, uint32_t cand, SlotUnion<W>& un,
                                               unsigned long long& improved) {
  uint32_t* dst = g.values + static_cast<size_t>(n) * static_cast<size_t>(g.Qg) + q;
  if (cand >= atomicMin(dst, cand)) return false;
  const uint32_t bit = 1u << (q & 31);
  uint32_t* fw = reinterpret_cast<uint32_t*>(lv.fnext + static_cast<size_t>(n) * W) + (q >> 5);
  const bool seen = *fw & bit;
  const bool listed = g.stamp[n] >= lv.level + 1;
  if (!seen) atomicOr(fw, bit);
  atomicOr(&un.word[q >> 5], bit);
  ++improved;
  return !listed && atomicMax(g.stamp + n, lv.level + 1) < lv.level + 1;
}

template <int W>
struct SsspPushSmem {
  int64_t beg[kWarpsPerBlock][32];
  int32_t inc[kWarpsPerBlock][32];
  int32_t u[kWarpsPerBlock][32];
  uint8_t k[kWarpsPerBlock][32];
  uint16_t q[kWarpsPerBlock][32][kListBits];
  uint16_t slots[kWarpsPerBlock][64 * W];
  SlotUnion<W> un;
};

// Frontiers of at most this many vertices have their listed vertices scattered
// by the tile's own warp; larger ones queue them for sssp_list_vertices, which
// spreads them over all warps.  16,384 is what fills every warp's tile a few
// vertices wide (tile_width): up to there a queue would only add a barrier or a
// launch, beyond it one tile's lists are the level's tail.
constexpr unsigned long long kInlineLists = 16384;

// SSSP push over the frontier list, a warp per tile of 32 vertices.  Vertices
// with few active bits: the tile's (edge, slot) pairs are flattened and spread
// evenly over the lanes.  The others go by slot lists, here or queued.  sweep:
// zero each vertex's mask once it is read (lists of the frontier must all be
// scattered by the tiles themselves).
template <int W, typename OT, int WK>
__device__ __forceinline__ void sssp_push_tiles(const GroupDev& g, const DevGraph& G, unsigned bid,
                                                unsigned nblk, SsspPushSmem<W>& sm,
                                                bool sweep = false) {
  const LevelCtl* ctl = g.ctl;
  if (ctl->done || !ctl->sscatter) return;
  const LevelView lv = level_view(g);
  WarpAppender ap;
  const unsigned long long n = ctl->count[lv.par];
  const int64_t light = push_light_limit(g, G, n, ctl->edges[lv.par]);
  const bool here = n <= kInlineLists;
  slot_union_clear<W>(sm.un);
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const unsigned long long gw = (static_cast<unsigned long long>(bid) * blockDim.x + threadIdx.x) >> 5;
  const unsigned long long nwarps = (static_cast<unsigned long long>(nblk) * blockDim.x) >> 5;
  const size_t Qg = static_cast<size_t>(g.Qg);
  unsigned long long improved = 0, spairs = 0, sactive = 0;
  const int tw = tile_width(n, nwarps);
  for (unsigned long long tile = gw; tile * tw < n; tile += nwarps) {
    const unsigned long long idx = tile * tw + lane;
    const bool valid = lane < tw && idx < n;
    const int32_t u = valid ? lv.list[idx] : 0;
    int64_t beg = 0, end = 0;
    int k = 0;
    {
      uint64_t b[W];
#pragma unroll
      for (int i = 0; i < W; ++i) b[i] = 0;
      if (valid) {
        beg = row_at<OT>(G.row, u);
        end = row_at<OT>(G.row, static_cast<int64_t>(u) + 1);
        load_mask<W>(lv.fcur + static_cast<size_t>(u) * W, b);
      }
#pragma unroll
      for (int i = 0; i < W; ++i) {
        b[i] &= ctl->ssel[i];
        k += __popcll(b[i]);
      }
      if (k > 0 && k <= kListBits) {
        int at = 0;
#pragma unroll
        for (int i = 0; i < W; ++i) {
          while (b[i]) {
            sm.q[wib][lane][at++] = static_cast<uint16_t>(64 * i + __ffsll(static_cast<long long>(b[i])) - 1);
            b[i] &= b[i] - 1;
          }
        }
      }
    }
    const int64_t deg = end - beg;
    const bool work = valid && k > 0 && deg > 0 && deg <= light;
    spairs += work ? static_cast<unsigned long long>(k) * static_cast<unsigned long long>(deg) : 0ULL;
    sactive += static_cast<unsigned long long>(k);
    unsigned lists = __ballot_sync(kFull, work && k > kListBits);
    if (lists && !here) {
      unsigned long long base = 0;
      if (lane == 0)
        base = atomicAdd(&g.ctl->dense_count, static_cast<unsigned long long>(__popc(lists)));
      base = __shfl_sync(kFull, base, 0);
      if ((lists >> lane) & 1u) g.dense_list[base + __popc(lists & ((1u << lane) - 1u))] = u;
      lists = 0;
    }
    while (lists) {
      const int src = __ffs(lists) - 1;
      lists &= lists - 1;
      const int32_t lu = __shfl_sync(kFull, u, src);
      const int64_t lb = __shfl_sync(kFull, beg, src), le = __shfl_sync(kFull, end, src);
      const uint32_t half = lane < 2 * W
          ? reinterpret_cast<const uint32_t*>(lv.fcur + static_cast<size_t>(lu) * W)[lane] &
                reinterpret_cast<const uint32_t*>(ctl->ssel)[lane]
          : 0u;
      const int lk = list_slots(half, lane, sm.slots[wib]);
      scatter_list<W, OT, WK, 4>(g, G, lv, lu, sm.slots[wib], lk, lb, le, lane, sm.un, improved, ap);
      __syncwarp();
    }
    if (sweep && valid) {  // no one reads the mask any more: clean for level + 1
      uint64_t z[W];
#pragma unroll
      for (int i = 0; i < W; ++i) z[i] = 0;
      store_mask<W>(const_cast<uint64_t*>(lv.fcur) + static_cast<size_t>(u) * W, z);
    }
    // the rest: (edge, slot) pairs flattened over the lanes
    const int wk = (work && k <= kListBits) ? k * static_cast<int>(deg) : 0;
    int inc = wk;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(kFull, inc, o);
      if (lane >= o) inc += t;
    }
    const int total = __shfl_sync(kFull, inc, 31);
    if (total == 0) continue;
    sm.beg[wib][lane] = beg;
    sm.inc[wib][lane] = inc;
    sm.k[wib][lane] = static_cast<uint8_t>(k <= kListBits ? k : 0);
    sm.u[wib][lane] = u;
    __syncwarp();
    for (int b0 = 0; b0 < total; b0 += 32 * kPairSteps) {
      int32_t nb[kPairSteps];
      int qq[kPairSteps];
      uint32_t cand[kPairSteps], cur[kPairSteps];
#pragma unroll
      for (int t = 0; t < kPairSteps; ++t) {
        const int p = b0 + 32 * t + lane;
        nb[t] = 0;
        qq[t] = 0;
        cand[t] = 0xffffffffu;
        if (p < total) {
          int lo = 0, hi = 31;
          while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (sm.inc[wib][mid] > p) hi = mid;
            else lo = mid + 1;
          }
          const int local = p - (lo ? sm.inc[wib][lo - 1] : 0);
          const int ko = sm.k[wib][lo];
          const int eoff = local / ko;
          qq[t] = sm.q[wib][lo][local - eoff * ko];
          const int64_t e = sm.beg[wib][lo] + eoff;
          nb[t] = G.col[e];
          cand[t] = relax<WK>(g.values[static_cast<size_t>(sm.u[wib][lo]) * Qg + qq[t]], G.w, e);
        }
      }
#pragma unroll
      for (int t = 0; t < kPairSteps; ++t)
        cur[t] = cand[t] != 0xffffffffu ? g.values[static_cast<size_t>(nb[t]) * Qg + qq[t]] : 0u;
#pragma unroll
      for (int t = 0; t < kPairSteps; ++t) {
        const bool app = cand[t] < cur[t] &&
                         scatter_commit<W>(g, lv, nb[t], qq[t], cand[t], sm.un, improved);
        ap.add<OT>(app, nb[t], G, lv, lane);
      }
    }
    __syncwarp();
  }
  ap.flush<OT>(G, lv, lane);
  slot_union_flush<W>(sm.un, lv.nactive);
  warp_add(improved, &g.ctl->lc.improved, lane);
  warp_add(spairs, &g.ctl->lc.sssp_pairs, lane);
  warp_add(sactive, &g.ctl->lc.sssp_active, lane);
}

template <int W, typename OT, int WK>
__global__ void __launch_bounds__(kBlock) k_sssp_push(GroupDev g, DevGraph G) {
  __shared__ SsspPushSmem<W> sm;
  sssp_push_tiles<W, OT, WK>(g, G, blockIdx.x, gridDim.x, sm);
}

template <int W>
struct SsspListSmem {
  uint16_t slots[kWarpsPerBlock][64 * W];
  SlotUnion<W> un;
};

// The queued vertices of a level (more than kListBits active bits), one warp
// per vertex; U edges per step.  Before, such vertices held 2W row chunks in
// registers and walked all of them per edge whether active or not: on a grid
// with 1024 slots and some 27 active bits per vertex, 34 ms of a 209 ms batch.
template <int W, typename OT, int WK, int U>
__device__ __forceinline__ void sssp_list_vertices(const GroupDev& g, const DevGraph& G,
                                                   unsigned bid, unsigned nblk,
                                                   SsspListSmem<W>& sm) {
  const LevelCtl* ctl = g.ctl;
  if (ctl->done || !ctl->sscatter) return;
  const unsigned long long n = ctl->dense_count;
  if (n == 0) return;
  const LevelView lv = level_view(g);
  WarpAppender ap;
  slot_union_clear<W>(sm.un);
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const unsigned long long gw = (static_cast<unsigned long long>(bid) * blockDim.x + threadIdx.x) >> 5;
  const unsigned long long nwarps = (static_cast<unsigned long long>(nblk) * blockDim.x) >> 5;
  const uint32_t sel = lane < 2 * W ? reinterpret_cast<const uint32_t*>(ctl->ssel)[lane] : 0u;
  unsigned long long improved = 0;
  for (unsigned long long i = gw; i < n; i += nwarps) {
    const int32_t u = g.dense_list[i];
    const int64_t beg = row_at<OT>(G.row, u);
    const int64_t end = row_at<OT>(G.row, static_cast<int64_t>(u) + 1);
    const uint32_t half = lane < 2 * W
        ? reinterpret_cast<const uint32_t*>(lv.fcur + static_cast<size_t>(u) * W)[lane] & sel
        : 0u;
    const int k = list_slots(half, lane, sm.slots[wib]);
    scatter_list<W, OT, WK, U>(g, G, lv, u, sm.slots[wib], k, beg, end, lane, sm.un, improved, ap);
    __syncwarp();
  }
  ap.flush<OT>(G, lv, lane);
  slot_union_flush<W>(sm.un, lv.nactive);
  warp_add(improved, &g.ctl->lc.improved, lane);
}

template <int W, typename OT, int WK, int U>
__global__ void __launch_bounds__(kBlock, 4) k_sssp_list(GroupDev g, DevGraph G) {
  __shared__ SsspListSmem<W> sm;
  sssp_list_vertices<W, OT, WK, U>(g, G, blockIdx.x, gridDim.x, sm);
}

template <int W>
struct SsspHeavySmem {
  int32_t h;
  int32_t k;
  uint16_t q[64 * W];
  SlotUnion<W> un;
};

// SSSP push for the queued heavy frontier vertices: per chunk of kHeavyChunk
// edges the CTA lists the active slots once; with more than kListBits of them
// each warp scatters a slice of the edges by the list, else the CTA walks the
// (edge, slot) pairs.
template <int W, typename OT, int WK>
__device__ __forceinline__ void sssp_push_chunks(const GroupDev& g, const DevGraph& G,
                                                 unsigned bid, unsigned nblk,
                                                 SsspHeavySmem<W>& sm) {
  const LevelCtl* ctl = g.ctl;
  if (ctl->done || !ctl->sscatter) return;
  const unsigned long long hq = ctl->hq_packed;
  const int nq = static_cast<int>(min(static_cast<long long>(hq >> kQueueShift),
                                      static_cast<long long>(g.hq_cap)));
  const int64_t nchunks = static_cast<int64_t>(hq & ((1ULL << kQueueShift) - 1));
  if (nq == 0) return;
  const LevelView lv = level_view(g);
  WarpAppender ap;
  slot_union_clear<W>(sm.un);
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const size_t Qg = static_cast<size_t>(g.Qg);
  unsigned long long improved = 0;
  for (int64_t c = bid; c < nchunks; c += nblk) {
    if (threadIdx.x == 0) sm.h = heavy_queue_slot(g, nq, c);
    __syncthreads();
    const int h = sm.h;
    const int32_t u = g.hq_vertex[h];
    if (wib == 0) {
      const uint32_t half = lane < 2 * W
          ? reinterpret_cast<const uint32_t*>(lv.fcur + static_cast<size_t>(u) * W)[lane] &
                reinterpret_cast<const uint32_t*>(ctl->ssel)[lane]
          : 0u;
      const int k = list_slots(half, lane, sm.q);
      if (lane == 0) sm.k = k;
    }
    __syncthreads();
    const int k = sm.k;
    if (k == 0) {
      __syncthreads();
      continue;
    }
    const int64_t beg = row_at<OT>(G.row, u);
    const int64_t end = row_at<OT>(G.row, static_cast<int64_t>(u) + 1);
    const int64_t cb = beg + (c - g.hq_start[h]) * kHeavyChunk;
    const int64_t ce = min(end, cb + kHeavyChunk);
    if (threadIdx.x == 0) {
      atomicAdd(&g.ctl->lc.sssp_pairs, static_cast<unsigned long long>(ce - cb) * k);
      if (c == g.hq_start[h]) atomicAdd(&g.ctl->lc.sssp_active, static_cast<unsigned long long>(k));
    }
    if (k > kListBits) {
      const int64_t seg = (ce - cb + kWarpsPerBlock - 1) / kWarpsPerBlock;
      const int64_t wb = min(ce, cb + wib * seg);
      const int64_t we = min(ce, wb + seg);
      scatter_list<W, OT, WK, 4>(g, G, lv, u, sm.q, k, wb, we, lane, sm.un, improved, ap);
      __syncthreads();
      continue;
    }
    const int pairs = static_cast<int>(ce - cb) * k;
    for (int p0 = threadIdx.x & ~31; p0 < pairs; p0 += kPairSteps * blockDim.x) {
      int32_t nb[kPairSteps];
      int qq[kPairSteps];
      uint32_t cand[kPairSteps], cur[kPairSteps];
#pragma unroll
      for (int t = 0; t < kPairSteps; ++t) {
        const int p = p0 + t * static_cast<int>(blockDim.x) + lane;
        nb[t] = 0;
        qq[t] = 0;
        cand[t] = 0xffffffffu;
        if (p < pairs) {
          const int eoff = p / k;
          qq[t] = sm.q[p - eoff * k];
          const int64_t e = cb + eoff;
          nb[t] = G.col[e];
          cand[t] = relax<WK>(g.values[static_cast<size_t>(u) * Qg + qq[t]], G.w, e);
        }
      }
#pragma unroll
      for (int t = 0; t < kPairSteps; ++t)
        cur[t] = cand[t] != 0xffffffffu ? g.values[static_cast<size_t>(nb[t]) * Qg + qq[t]] : 0u;
#pragma unroll
      for (int t = 0; t < kPairSteps; ++t) {
        const bool app = cand[t] < cur[t] &&
                         scatter_commit<W>(g, lv, nb[t], qq[t], cand[t], sm.un, improved);
        ap.add<OT>(app, nb[t], G, lv, lane);
      }
    }
    __syncthreads();
  }
  ap.flush<OT>(G, lv, lane);
  slot_union_flush<W>(sm.un, lv.nactive);
  warp_add(improved, &g.ctl->lc.improved, lane);
}

template <int W, typename OT, int WK>
__global__ void __launch_bounds__(kBlock) k_sssp_push_heavy(GroupDev g, DevGraph G) {
  __shared__ SsspHeavySmem<W> sm;
  sssp_push_chunks<W, OT, WK>(g, G, blockIdx.x, gridDim.x, sm);
}


// ------------------------------------------------------------ SSSP gather
// Dense SSSP levels (most vertices in the frontier for many queries) run as a
// gather instead of a scatter: the warp that owns vertex v takes the minimum
// of dist[u][q] + w(u, v) over v's in-edges for all its SSSP slots at once,
// then writes the improved entries of v's row with plain stores.  No
// distance atomics, no per-(edge, query) frontier atomics: the improved bits
// of a 32-slot chunk come from one ballot.  Lane j owns slot 32c + j of
// chunk c; the sources' rows are read for every SSSP slot of the chunk (an
// entry that is not in the frontier relaxes to a value that cannot improve
// v, or to one that another relaxation would produce anyway), so per edge the
// warp issues 2W coalesced 128-byte loads and no data-dependent branches.
// Several in-edges are in flight per warp (GatherSteps) to cover latency.

// Relaxation of a stored value `du` over an edge with raw weight bits.  The
// unreached markers (0xffffffff; +inf for f32, whose sums stay +inf or become a
// NaN, larger than every value as a uint32) never improve anything.
template <int WK>
__device__ __forceinline__ uint32_t gather_relax(uint32_t du, uint32_t wbits) {
  if constexpr (WK == kWeightF32) {
    return __float_as_uint(__fadd_rn(__uint_as_float(du), __uint_as_float(wbits)));
  } else {
    const uint32_t wt = (WK == kWeightU32) ? wbits : 1u;
    return min(du, ~wt) + wt;  // saturates at 0xffffffff
  }
}

// In-edges gathered together per warp step: 2W x steps row loads per lane.
template <int W>
struct GatherSteps {
  static constexpr int value = W >= 16 ? 1 : (W >= 8 ? 2 : (W >= 4 ? 4 : 8));
};

// Bit c of the result: this lane's slot of chunk c is an SSSP slot that
// gathers at this level.
template <int W>
__device__ __forceinline__ uint32_t lane_sssp_chunks(const LevelCtl* ctl, int lane) {
  uint32_t sel = 0;
#pragma unroll
  for (int c = 0; c < 2 * W; ++c)
    sel |= static_cast<uint32_t>((ctl->gsel[c >> 1] >> (32 * (c & 1) + lane)) & 1ULL) << c;
  return sel;
}

// min-accumulates relaxations over in-edges [eb, ee) of the pull CSR into
// best[c] (lane's slot of chunk c).  Edges whose source has no SSSP frontier
// bit are skipped by a ballot.  All lanes call.
template <int W, int WK>
__device__ __forceinline__ void gather_edges(const GroupDev& g, const DevGraph& G,
                                             const LevelView& lv, const uint64_t* sb,
                                             uint32_t lsel, int64_t eb, int64_t ee, int lane,
                                             uint32_t (&best)[2 * W],
                                             unsigned long long& pairs,
                                             unsigned& scanned) {
  constexpr int C = 2 * W;
  constexpr int S = GatherSteps<W>::value;
  const size_t Qg = static_cast<size_t>(g.Qg);
  for (int64_t e0 = eb; e0 < ee; e0 += 32) {
    const int64_t e = e0 + lane;
    int32_t u = 0;
    uint32_t wb = 0;
    int k = 0;
    if (e < ee) {
      u = G.pcol[e];
      wb = weight_bits<WK>(G.pw, e);
      uint64_t m[W];
      load_mask<W>(lv.fcur + static_cast<size_t>(u) * W, m);
#pragma unroll
      for (int i = 0; i < W; ++i) k += __popcll(m[i] & sb[i]);
      ++scanned;
    }
    pairs += static_cast<unsigned long long>(k);
    unsigned live = __ballot_sync(kFull, k > 0);
    while (live) {
      int32_t us[S];
      uint32_t ws[S];
      bool ok[S];
#pragma unroll
      for (int t = 0; t < S; ++t) {
        ok[t] = live != 0;
        const int j = (__ffs(live) - 1) & 31;
        live &= live - 1;
        us[t] = __shfl_sync(kFull, u, j);
        ws[t] = __shfl_sync(kFull, wb, j);
      }
      uint32_t cur[S][C];
#pragma unroll
      for (int t = 0; t < S; ++t) {
        const uint32_t* row = g.values + static_cast<size_t>(us[t]) * Qg + lane;
#pragma unroll
        for (int c = 0; c < C; ++c)
          cur[t][c] = (ok[t] && ((lsel >> c) & 1u)) ? __ldcg(row + 32 * c) : 0xffffffffu;
      }
#pragma unroll
      for (int t = 0; t < S; ++t) {
#pragma unroll
        for (int c = 0; c < C; ++c) best[c] = min(best[c], gather_relax<WK>(cur[t][c], ws[t]));
      }
    }
  }
}

// Gather level, vertices of in-degree <= heavy_degree: one warp per vertex.
template <int W, typename OT, int WK>
__global__ void __launch_bounds__(kBlock, (W <= 4 ? 3 : 2)) k_sssp_pull(GroupDev g, DevGraph G) {
  const LevelCtl* ctl = g.ctl;
  if (ctl->done || ctl->sdir != kDirPull) return;
  const LevelView lv = level_view(g);
  constexpr int C = 2 * W;
  const int lane = threadIdx.x & 31;
  const uint64_t* sb = ctl->gsel;
  const uint32_t lsel = lane_sssp_chunks<W>(ctl, lane);
  const unsigned long long gw = (static_cast<unsigned long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const unsigned long long nwarps = (static_cast<unsigned long long>(gridDim.x) * blockDim.x) >> 5;
  const size_t Qg = static_cast<size_t>(g.Qg);
  uint64_t uni[W];
#pragma unroll
  for (int i = 0; i < W; ++i) uni[i] = 0;
  unsigned long long improved = 0, pairs = 0;
  unsigned scanned = 0, verts = 0;
  for (unsigned long long vv = gw; vv < static_cast<unsigned long long>(G.V); vv += nwarps) {
    const int32_t v = static_cast<int32_t>(vv);
    const int64_t beg = row_at<OT>(G.prow, v);
    const int64_t end = row_at<OT>(G.prow, static_cast<int64_t>(v) + 1);
    if (end == beg || end - beg > G.heavy_degree) continue;
    if (lane == 0) ++verts;  // one count per vertex, not per lane
    uint32_t* row = g.values + static_cast<size_t>(v) * Qg + lane;
    uint32_t best[C];
#pragma unroll
    for (int c = 0; c < C; ++c) best[c] = ((lsel >> c) & 1u) ? row[32 * c] : 0u;
    gather_edges<W, WK>(g, G, lv, sb, lsel, beg, end, lane, best, pairs, scanned);
    uint64_t nw[W];
#pragma unroll
    for (int i = 0; i < W; ++i) nw[i] = 0;
    // the warp owns v's row this level: the entries read above are unchanged
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const bool imp = ((lsel >> c) & 1u) && best[c] < row[32 * c];
      if (imp) row[32 * c] = best[c];
      nw[c >> 1] |= static_cast<uint64_t>(__ballot_sync(kFull, imp)) << (32 * (c & 1));
    }
    bool app = false;
    if (lane == 0 && mask_any<W>(nw)) {
#pragma unroll
      for (int i = 0; i < W; ++i) {
        if (!nw[i]) continue;
        atomic_or64(lv.fnext + static_cast<size_t>(v) * W + i, nw[i]);
        uni[i] |= nw[i];
        improved += __popcll(nw[i]);
      }
      app = atomicMax(g.stamp + v, lv.level + 1) < lv.level + 1;
    }
    warp_append(app, v, app ? degree_of<OT>(G.row, v) : 0, lv.nlist, lv.ncount, lv.nedges, lane);
  }
  flush_union<W>(uni, lv.nactive, lane);
  warp_add(improved, &g.ctl->lc.improved, lane);
  warp_add(pairs, &g.ctl->lc.sssp_pairs, lane);
  warp_add(scanned, &g.ctl->lc.spull_edges, lane);
  warp_add(verts, &g.ctl->lc.spull_vertices, lane);
}

// Gather level, heavy vertices (in-degree > heavy_degree): a CTA takes a
// chunk of kHeavyChunk in-edges, its warps min-reduce slices into shared
// memory, and the chunk's result is committed with one atomicMin per slot.
template <int W, typename OT, int WK>
__global__ void __launch_bounds__(kBlock) k_sssp_pull_heavy(GroupDev g, DevGraph G) {
  const LevelCtl* ctl = g.ctl;
  if (ctl->done || ctl->sdir != kDirPull || G.n_pheavy == 0) return;
  const LevelView lv = level_view(g);
  constexpr int C = 2 * W;
  __shared__ uint32_t s_best[C * 32];
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const uint64_t* sb = ctl->gsel;
  const uint32_t lsel = lane_sssp_chunks<W>(ctl, lane);
  const size_t Qg = static_cast<size_t>(g.Qg);
  uint64_t uni[W];
#pragma unroll
  for (int i = 0; i < W; ++i) uni[i] = 0;
  unsigned long long improved = 0, pairs = 0;
  unsigned scanned = 0;
  // every heavy vertex is gathered once per launch (all its chunks)
  if (blockIdx.x == 0 && threadIdx.x == 0)
    atomicAdd(&g.ctl->lc.spull_vertices, static_cast<unsigned long long>(G.n_pheavy));
  for (int64_t ch = blockIdx.x; ch < G.pheavy_chunks; ch += gridDim.x) {
    // the chunk's vertex and edge range: independent loads, no search
    const int32_t v = G.pheavy[G.pheavy_ch[ch]];
    const int64_t cb = G.pheavy_cb[ch];
    const int64_t ce = G.pheavy_ce[ch];
    for (int i = threadIdx.x; i < C * 32; i += blockDim.x) s_best[i] = 0xffffffffu;
    __syncthreads();
    const int64_t seg = (ce - cb + kWarpsPerBlock - 1) / kWarpsPerBlock;
    const int64_t wb = cb + wib * seg;
    const int64_t we = min(ce, wb + seg);
    uint32_t best[C];
#pragma unroll
    for (int c = 0; c < C; ++c) best[c] = 0xffffffffu;
    gather_edges<W, WK>(g, G, lv, sb, lsel, wb, we, lane, best, pairs, scanned);
#pragma unroll
    for (int c = 0; c < C; ++c)
      if (best[c] != 0xffffffffu) atomicMin(&s_best[32 * c + lane], best[c]);
    __syncthreads();
    // commit: warp wib takes chunks wib, wib + 8, ...
    bool any = false;
    for (int c = wib; c < C; c += kWarpsPerBlock) {
      const int q = 32 * c + lane;
      bool imp = false;
      if ((lsel >> c) & 1u) {
        const uint32_t b = s_best[q];
        uint32_t* p = g.values + static_cast<size_t>(v) * Qg + q;
        if (b < *p) imp = b < atomicMin(p, b);
      }
      const unsigned m = __ballot_sync(kFull, imp);
      if (m) {
        any = true;
        if (lane == 0) {
          const uint64_t bits = static_cast<uint64_t>(m) << (32 * (c & 1));
          atomic_or64(lv.fnext + static_cast<size_t>(v) * W + (c >> 1), bits);
          uni[c >> 1] |= bits;
          improved += __popc(m);
        }
      }
    }
    bool app = false;
    if (any && lane == 0) app = atomicMax(g.stamp + v, lv.level + 1) < lv.level + 1;
    warp_append(app, v, app ? degree_of<OT>(G.row, v) : 0, lv.nlist, lv.ncount, lv.nedges, lane);
    __syncthreads();
  }
  flush_union<W>(uni, lv.nactive, lane);
  warp_add(improved, &g.ctl->lc.improved, lane);
  warp_add(pairs, &g.ctl->lc.sssp_pairs, lane);
  warp_add(scanned, &g.ctl->lc.spull_edges, lane);
}


// ------------------------------------------------- SSSP gather, vectorised
// The same gather with vector loads, for groups whose rows are 16-byte
// aligned and hold a multiple of the vector width (the usual case): lane l
// owns the kElem consecutive slots (32r + l)*kElem .. +kElem of each part r,
// so a row costs kParts vector loads per lane instead of 2W scalar ones.
// The live in-edges of a 32-edge batch are compacted into shared memory by
// a ballot prefix, and full groups of kSteps edges are gathered without any
// per-load predicate.
template <int W>
struct GatherVec {
  static constexpr int kElem = W == 1 ? 2 : 4;      // slots per vector load
  static constexpr int kParts = 2 * W / kElem;      // vector loads per lane per row
  static constexpr int kSlots = kParts * kElem;     // slots per lane
  static constexpr int kSteps = W <= 2 ? 8 : (W == 4 ? 4 : (W == 8 ? 2 : 1));
  static constexpr int kLanesPerHalf = 32 / kElem;  // lanes covering one 32-bit mask half
};

template <int E>
__device__ __forceinline__ void load_vec_cg(const uint32_t* p, uint32_t* x) {
  if constexpr (E == 4) {
    const uint4 v = __ldcg(reinterpret_cast<const uint4*>(p));
    x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
  } else {
    const uint2 v = __ldcg(reinterpret_cast<const uint2*>(p));
    x[0] = v.x; x[1] = v.y;
  }
}

// load_vec_cg under a predicate; x keeps its values where on is 0.  (As an if
// the compiler branches around each load, and the rows of a step are no longer
// in flight together: R-MAT 20 gather levels 0.73 -> 1.1 ms.)
template <int E>
__device__ __forceinline__ void load_vec_cg_if(uint32_t on, const uint32_t* p, uint32_t* x) {
  if constexpr (E == 4) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %4, 0;\n\t"
        "@q ld.global.cg.v4.u32 {%0, %1, %2, %3}, [%5];\n\t}"
        : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]), "+r"(x[3])
        : "r"(on), "l"(p));
  } else {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t"
        "@q ld.global.cg.v2.u32 {%0, %1}, [%3];\n\t}"
        : "+r"(x[0]), "+r"(x[1])
        : "r"(on), "l"(p));
  }
}

template <int E>
__device__ __forceinline__ void load_vec(const uint32_t* p, uint32_t* x) {
  if constexpr (E == 4) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
  } else {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    x[0] = v.x; x[1] = v.y;
  }
}

template <int E>
__device__ __forceinline__ void store_vec(uint32_t* p, const uint32_t* x) {
  if constexpr (E == 4) *reinterpret_cast<uint4*>(p) = make_uint4(x[0], x[1], x[2], x[3]);
  else *reinterpret_cast<uint2*>(p) = make_uint2(x[0], x[1]);
}

// Weight of a row chunk that was not read: relaxing with it changes nothing,
// whatever the registers hold.
template <int WK>
__device__ __forceinline__ uint32_t dead_weight() {
  return WK == kWeightF32 ? 0x7f800000u : 0xffffffffu;
}

// best[j] = min(best[j], du[j] + w) for the E slots of one part; w is a raw
// weight (1 on unweighted graphs) or dead_weight().
template <int WK, int E>
__device__ __forceinline__ void relax_part(uint32_t* best, const uint32_t* du, uint32_t w) {
  if constexpr (WK == kWeightF32) {
#pragma unroll
    for (int k = 0; k < E; ++k)
      best[k] = min(best[k], __float_as_uint(__fadd_rn(__uint_as_float(du[k]), __uint_as_float(w))));
  } else {
    const uint32_t lim = ~w;
#pragma unroll
    for (int k = 0; k < E; ++k) best[k] = min(best[k], min(du[k], lim) + w);
  }
}

// Reads rows stage[i .. i + S) of a staging list of n (all of them when kWhole)
// into cur, for the lane's slots.  pbit[r] is the row chunk of the lane's part
// r, 0 when the lane has no gathering slot there.  Without kChunks every chunk
// is read.  Parts that are not read keep what the registers held.  (The
// entries are read again when they are relaxed: held across the loads they
// cost 4 registers a row, and the row gather spilled.)
template <int W, bool kChunks, bool kWhole, int S>
__device__ __forceinline__ void load_rows(const uint32_t* lanebase, unsigned Qg, const int4* stage,
                                          int i, int n,
                                          const uint32_t (&pbit)[GatherVec<W>::kParts],
                                          uint32_t (&cur)[S][GatherVec<W>::kSlots]) {
  using GV = GatherVec<W>;
  constexpr int E = GV::kElem;
#pragma unroll
  for (int t = 0; t < S; ++t) {
    if (!kWhole && i + t >= n) break;  // uniform
    const uint32_t u = static_cast<uint32_t>(stage[i + t].x);
    const uint32_t cm = kChunks ? static_cast<uint32_t>(stage[i + t].w) : 0xffffffffu;
    const uint32_t* row = lanebase + static_cast<uint64_t>(u) * Qg;
#pragma unroll
    for (int r = 0; r < GV::kParts; ++r)
      load_vec_cg_if<E>(cm & pbit[r], row + 32 * E * r, &cur[t][r * E]);
  }
}

// Relaxes one loaded row (weight w, row chunks cm).
template <int W, int WK, bool kChunks>
__device__ __forceinline__ void relax_row(uint32_t (&best)[GatherVec<W>::kSlots],
                                          const uint32_t (&cur)[GatherVec<W>::kSlots], uint32_t w,
                                          uint32_t cm,
                                          const uint32_t (&pbit)[GatherVec<W>::kParts]) {
  using GV = GatherVec<W>;
  if (WK == kWeightNone) w = 1u;
#pragma unroll
  for (int r = 0; r < GV::kParts; ++r)
    relax_part<WK, GV::kElem>(&best[r * GV::kElem], &cur[r * GV::kElem],
                              !kChunks || (cm & pbit[r]) ? w : dead_weight<WK>());
}

// The lane's row chunks, part by part (see load_rows).
template <int W>
__device__ __forceinline__ void part_chunks(uint32_t pmask, int lane,
                                            uint32_t (&pbit)[GatherVec<W>::kParts]) {
  using GV = GatherVec<W>;
#pragma unroll
  for (int r = 0; r < GV::kParts; ++r)
    pbit[r] = (pmask >> r) & 1u ? 1u << (((32 * r + lane) * GV::kElem) >> 5) : 0u;
}

// Lane masks for the vectorised gather: bit r of *parts: the lane's vector of
// part r lies inside the row (slot < Qg) and holds a slot that gathers at this
// level (otherwise the lane neither loads nor commits it: a 32-slot chunk
// without gathering slots is never read); bit j of *slots: slot j of the lane
// gathers.
template <int W>
__device__ __forceinline__ void gather_vec_masks(const uint64_t* gsel, int Qg, int lane,
                                                 uint32_t* parts, uint32_t* slots) {
  using GV = GatherVec<W>;
  uint32_t pm = 0, sm = 0;
#pragma unroll
  for (int r = 0; r < GV::kParts; ++r) {
    const int base = (32 * r + lane) * GV::kElem;
#pragma unroll
    for (int k = 0; k < GV::kElem; ++k) {
      const int q = base + k;
      if (q < Qg && ((gsel[q >> 6] >> (q & 63)) & 1ULL)) sm |= 1u << (r * GV::kElem + k);
    }
    if (base < Qg && ((sm >> (r * GV::kElem)) & ((1u << GV::kElem) - 1u))) pm |= 1u << r;
  }
  *parts = pm;
  *slots = sm;
}

// ORs the lanes' per-slot bits into 64-bit frontier words: `bits` holds the
// lane's kSlots bits (slot r*kElem + k at bit r*kElem + k).  For each part,
// the lane whose slots start a word receives it in words[r] (0 elsewhere).
template <int W>
__device__ __forceinline__ void gather_vec_words(uint32_t bits, int lane,
                                                 uint64_t (&words)[GatherVec<W>::kParts]) {
  using GV = GatherVec<W>;
  constexpr int E = GV::kElem;
  constexpr int L = GV::kLanesPerHalf;
#pragma unroll
  for (int r = 0; r < GV::kParts; ++r) {
    uint32_t h = ((bits >> (r * E)) & ((1u << E) - 1u)) << (E * (lane % L));
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) h |= __shfl_xor_sync(kFull, h, o);
    const uint32_t hi = __shfl_down_sync(kFull, h, L);
    words[r] = (lane % (2 * L) == 0) ? (static_cast<uint64_t>(hi) << 32) | h : 0ULL;
  }
}

// 32-slot chunks that hold a gathering SSSP slot at this level.
template <int W>
__device__ __forceinline__ uint32_t gather_chunks(const uint64_t* gsel) {
  uint64_t gs[W];
#pragma unroll
  for (int i = 0; i < W; ++i) gs[i] = gsel[i];
  return chunk_bits<W>(gs);
}

template <int W>
__device__ __forceinline__ uint32_t gather_chunks(const LevelCtl* ctl) {
  return gather_chunks<W>(ctl->gsel);
}

// Whether the gather screens in-edges by their source's frontier chunks (-1)
// or reads every in-edge's source row whole (the number of gathering slots).
// With the frontier summary: a whole-row gather reads E x (gathering chunks)
// row chunks, a screened one only the live ones, which the summary kernel
// counted (live_chunks); screening pays when fewer than 4/5 of them are live,
// and costs an 8-byte L2 word per in-edge.  Without it (no summary buffer):
// screen when the frontier's out-edges are less than half of all edges or its
// entries are sparse (the previous level improved fewer than 1/32 of the
// frontier's vertices x SSSP slots), reading the sources' W-word masks.
template <int W>
__device__ __forceinline__ int gather_screen_qs(const GroupDev& g, const LevelCtl* ctl,
                                                const LevelView& lv, int64_t E) {
  int qs = 0;
#pragma unroll
  for (int i = 0; i < W; ++i) qs += __popcll(ctl->gsel[i]);
  if (g.fsum != nullptr) {
    const unsigned long long whole =
        static_cast<unsigned long long>(E) * static_cast<unsigned long long>(__popc(gather_chunks<W>(ctl)));
    return 5 * ctl->lc.live_chunks < 4 * whole ? -1 : qs;
  }
  if (2 * ctl->edges[lv.par] < static_cast<unsigned long long>(E)) return -1;
  if (32 * ctl->prev_improved < ctl->count[lv.par] * static_cast<unsigned long long>(qs)) return -1;
  return qs;
}

// Writes the frontier summary of the current frontier's vertices on SSSP
// gather levels and sparse BFS pull levels (other levels return at once), and
// on gather levels counts the live row chunks a screened gather would read
// (out-degree x gathering chunks with a frontier bit).  Words of vertices
// outside the frontier keep an older level's stamp and read as empty.
template <int W, typename OT>
__device__ __forceinline__ void frontier_summary(const GroupDev& g, const DevGraph& G,
                                                 unsigned bid, unsigned nblk) {
  LevelCtl* ctl = g.ctl;
  if (ctl->done) return;
  const LevelView lv = level_view(g);
  const bool sssp = ctl->sdir == kDirPull && !ctl->bnd_on;  // else gather_bounds counts
  if (!sssp && !bfs_pull_uses_summary(g, ctl, lv, G.V)) return;
  const unsigned long long n = ctl->count[lv.par];
  const uint64_t stamp = static_cast<uint64_t>(lv.level + 1) << 32;
  const uint32_t gch = gather_chunks<W>(ctl);
  const int lane = threadIdx.x & 31;
  unsigned long long live = 0;
  const unsigned long long stride = static_cast<unsigned long long>(nblk) * blockDim.x;
  for (unsigned long long i0 = static_cast<unsigned long long>(bid) * blockDim.x + (threadIdx.x & ~31);
       i0 < n; i0 += stride) {
    const unsigned long long i = i0 + lane;
    if (i < n) {
      const int32_t v = lv.list[i];
      uint64_t m[W];
      load_mask<W>(lv.fcur + static_cast<size_t>(v) * W, m);
      const uint32_t cm = chunk_bits<W>(m);
      g.fsum[v] = stamp | cm;
      if (sssp) live += __popc(cm & gch) * degree_of<OT>(G.row, v);
    }
  }
  if (sssp) warp_add(live, &ctl->lc.live_chunks, lane);
}

template <int W, typename OT>
__global__ void __launch_bounds__(kBlock) k_frontier_summary(GroupDev g, DevGraph G) {
  frontier_summary<W, OT>(g, G, blockIdx.x, gridDim.x);
}

// ------------------------------------------------- bounds on row chunks
// An in-edge (u, v) of weight w can lower v's slot q only if d[u][q] + w <
// d[v][q].  With any reference value b[q] per slot, subtracted on both sides,
//   min_q (d[u][q] - b[q]) + w >= max_q (d[v][q] - b[q])
// proves that no slot of a 32-slot chunk improves, and the chunk of u's row
// need not be read.  On small-world graphs a distance is close to (a part of
// the vertex) + (a part of the source): with b = the row of the best connected
// vertex the differences of one vertex lie close together, and once most
// vertices are reached the test skips most chunks (R-MAT 17, 256 sources, the
// second to sixth gather level: 37, 81, 92, 96 and 99% of the live chunks).
// The minimum is taken over u's frontier slots (the others have offered their
// values before), the maximum over the slots with any frontier bit left.
// Rounding and clamping go the safe way on both sides, and values only fall
// during a level, so a skipped chunk never hides an improvement: a vertex
// lowered during the level is in the next frontier.
//
// uint32 distances: int32 offsets within +-2^30, larger values clamped the safe
// way (kBoundNone: no frontier slot, or no upper bound); f32: the offsets as
// floats (+inf for both).
constexpr uint32_t kBoundNone = 0x7fffffffu;
constexpr uint32_t kBoundNoneF32 = 0x7f800000u;
constexpr uint32_t kBoundMax = (1u << 30) - 1u;

template <int WK>
__device__ __forceinline__ uint32_t bound_none() {
  return WK == kWeightF32 ? kBoundNoneF32 : kBoundNone;
}

// Reference value of a slot: the hub's distance, 0 where there is none.
template <int WK>
__device__ __forceinline__ uint32_t bound_ref(uint32_t d) {
  if constexpr (WK == kWeightF32) return d >= 0x7f800000u ? 0u : d;
  else return d > kBoundMax ? 0u : d;
}

template <int WK>
__device__ __forceinline__ uint32_t bound_low(uint32_t d, uint32_t b) {
  if constexpr (WK == kWeightF32)
    return __float_as_uint(__fsub_rd(__uint_as_float(d), __uint_as_float(b)));
  else
    return min(d, kBoundMax) - b;
}

template <int WK>
__device__ __forceinline__ uint32_t bound_high(uint32_t d, uint32_t b) {
  if constexpr (WK == kWeightF32)
    return __float_as_uint(__fsub_ru(__uint_as_float(d), __uint_as_float(b)));  // inf stays inf
  else
    return d > kBoundMax ? kBoundNone : d - b;
}

template <int WK>
__device__ __forceinline__ uint32_t bound_min(uint32_t a, uint32_t b) {
  if constexpr (WK == kWeightF32)
    return __float_as_uint(fminf(__uint_as_float(a), __uint_as_float(b)));
  else
    return static_cast<uint32_t>(min(static_cast<int32_t>(a), static_cast<int32_t>(b)));
}

template <int WK>
__device__ __forceinline__ uint32_t bound_max(uint32_t a, uint32_t b) {
  if constexpr (WK == kWeightF32)
    return __float_as_uint(fmaxf(__uint_as_float(a), __uint_as_float(b)));
  else
    return static_cast<uint32_t>(max(static_cast<int32_t>(a), static_cast<int32_t>(b)));
}

// Whether a chunk with lower bound lo at the source may improve one with upper
// bound hi at the destination over an edge of raw weight wbits.
template <int WK>
__device__ __forceinline__ bool bound_improves(uint32_t lo, uint32_t hi, uint32_t wbits) {
  if constexpr (WK == kWeightF32) {
    return __fadd_rd(__uint_as_float(lo), __uint_as_float(wbits)) < __uint_as_float(hi);
  } else {
    // no sum of a clamped bound and a clamped weight reaches kBoundNone
    const int32_t w = static_cast<int32_t>(min(WK == kWeightU32 ? wbits : 1u, kBoundMax));
    return lo != kBoundNone && static_cast<int32_t>(lo) + w < static_cast<int32_t>(hi);
  }
}

// Chunks of the source row with lower bounds lo[2W] that may improve the
// destination with upper bounds hi[2W].
template <int W, int WK>
__device__ __forceinline__ uint32_t bound_chunks(const uint32_t* lo, const uint32_t* hi,
                                                 uint32_t wbits) {
  constexpr int N = 2 * W < 4 ? 2 : 4;
  uint32_t cm = 0;
#pragma unroll
  for (int c = 0; c < 2 * W; c += N) {
    uint32_t l[N], h[N];
    load_vec<N>(lo + c, l);
    load_vec<N>(hi + c, h);
#pragma unroll
    for (int k = 0; k < N; ++k)
      cm |= static_cast<uint32_t>(bound_improves<WK>(l[k], h[k], wbits)) << (c + k);
  }
  return cm;
}

// Writes both bounds of every vertex with in-edges at the start of a gather
// level that uses them (a warp per vertex and slice of WS words: one pass over
// their values) and counts the live chunks, as the frontier summary does on
// other levels.  A vertex without in-edges has nothing lowered and is in no
// frontier after the first: its bounds are never written and whatever they
// hold skips or reads rows that change nothing.
template <int W, typename OT, int WK>
__device__ __forceinline__ void gather_bounds(const GroupDev& g, const DevGraph& G, unsigned bid,
                                              unsigned nblk) {
  LevelCtl* ctl = g.ctl;
  if (ctl->done || ctl->sdir != kDirPull || !ctl->bnd_on) return;
  constexpr int WS = W < 4 ? W : 4;
  using GV = GatherVec<WS>;
  constexpr int E = GV::kElem;
  constexpr int P = GV::kParts;
  constexpr int L = GV::kLanesPerHalf;
  constexpr uint32_t kNone = WK == kWeightF32 ? kBoundNoneF32 : kBoundNone;
  constexpr uint32_t kLeast = WK == kWeightF32 ? 0xff800000u : 0x80000000u;
  const LevelView lv = level_view(g);
  const int lane = threadIdx.x & 31;
  const size_t Qg = static_cast<size_t>(g.Qg);
  const int n_light = G.n_plight;
  const int n = n_light + G.n_pheavy;
  const int gw = static_cast<int>((static_cast<long long>(bid) * blockDim.x + threadIdx.x) >> 5);
  const int nwarps = static_cast<int>((static_cast<long long>(nblk) * blockDim.x) >> 5);
  unsigned long long live = 0;
  for (int sl = 0; sl < W / WS; ++sl) {
    const int s0 = sl * 64 * WS;
    uint64_t sel[WS];
#pragma unroll
    for (int i = 0; i < WS; ++i) sel[i] = ctl->gsel[sl * WS + i] & ctl->active[lv.par][sl * WS + i];
    uint32_t pmask, smask;
    gather_vec_masks<WS>(sel, g.Qg - s0, lane, &pmask, &smask);
    uint32_t ref[GV::kSlots];
#pragma unroll
    for (int r = 0; r < P; ++r) {
      if ((pmask >> r) & 1u) {
        load_vec<E>(g.values + static_cast<size_t>(G.hub) * Qg + s0 + (32 * r + lane) * E, &ref[r * E]);
      } else {
#pragma unroll
        for (int k = 0; k < E; ++k) ref[r * E + k] = 0u;
      }
#pragma unroll
      for (int k = 0; k < E; ++k) ref[r * E + k] = bound_ref<WK>(ref[r * E + k]);
    }
    // two vertices per step, every load of both in flight at once; the next
    // step's vertex ids are loaded a step ahead
    constexpr int U = 2;
    auto vertex = [&](int i) { return i < n_light ? G.plight[i] : G.pheavy[i - n_light]; };
    int32_t nv[U];
#pragma unroll
    for (int t = 0; t < U; ++t) nv[t] = gw + t * nwarps < n ? vertex(gw + t * nwarps) : 0;
    for (int i0 = gw; i0 < n; i0 += nwarps * U) {
      int32_t v[U];
      uint32_t d[U][GV::kSlots];
      uint32_t fr[U][P];  // the lane's frontier bits
#pragma unroll
      for (int t = 0; t < U; ++t) {
        v[t] = nv[t];
#pragma unroll
        for (int r = 0; r < P; ++r) {
          const int q = s0 + (32 * r + lane) * E;
          fr[t][r] = static_cast<uint32_t>(lv.fcur[static_cast<size_t>(v[t]) * W + (q >> 6)] >> (q & 63));
          if ((pmask >> r) & 1u) {
            load_vec<E>(g.values + static_cast<size_t>(v[t]) * Qg + q, &d[t][r * E]);
          } else {
#pragma unroll
            for (int k = 0; k < E; ++k) d[t][r * E + k] = 0u;
          }
        }
      }
#pragma unroll
      for (int t = 0; t < U; ++t) {
        const int i = i0 + (U + t) * nwarps;
        if (i < n) nv[t] = vertex(i);
      }
#pragma unroll
      for (int t = 0; t < U; ++t) {
        if (i0 + t * nwarps >= n) break;  // uniform
        uint32_t chunks = 0;
#pragma unroll
        for (int r = 0; r < P; ++r) {
          const uint32_t fs = fr[t][r] & (smask >> (r * E));
          uint32_t lo = kNone, hi = kLeast;
#pragma unroll
          for (int k = 0; k < E; ++k) {
            const uint32_t x = d[t][r * E + k], b = ref[r * E + k];
            const uint32_t xl = (fs >> k) & 1u ? bound_low<WK>(x, b) : kNone;
            const uint32_t xh = (smask >> (r * E + k)) & 1u ? bound_high<WK>(x, b) : kLeast;
            lo = bound_min<WK>(lo, xl);
            hi = bound_max<WK>(hi, xh);
          }
#pragma unroll
          for (int o = L / 2; o > 0; o >>= 1) {
            lo = bound_min<WK>(lo, __shfl_xor_sync(kFull, lo, o));
            hi = bound_max<WK>(hi, __shfl_xor_sync(kFull, hi, o));
          }
          if (lane % L == 0) {
            const size_t at =
                static_cast<size_t>(v[t]) * (2 * W) + sl * 2 * WS + (32 / L) * r + lane / L;
            g.blo[at] = lo;
            g.bhi[at] = hi;
            chunks += lo != kNone ? 1u : 0u;
          }
        }
        if (chunks) live += chunks * degree_of<OT>(G.row, v[t]);
      }
    }
  }
  warp_add(live, &ctl->lc.live_chunks, lane);
}

template <int W, typename OT, int WK>
__global__ void __launch_bounds__(kBlock) k_gather_bounds(GroupDev g, DevGraph G) {
  gather_bounds<W, OT, WK>(g, G, blockIdx.x, gridDim.x);
}

// Gathers in-edges [eb, ee) into best[] (vector layout).  `stage` is this
// warp's 32-entry shared staging array.  All lanes call.
template <int W, int WK, bool kChunks = true>
__device__ __forceinline__ void gather_edges_vec(const GroupDev& g, const DevGraph& G,
                                                 const LevelView& lv, const uint64_t* sb,
                                                 uint32_t pmask, int64_t eb, int64_t ee,
                                                 int lane, int4* stage,
                                                 uint32_t (&best)[GatherVec<W>::kSlots],
                                                 unsigned long long& pairs,
                                                 unsigned& scanned, int screen_qs,
                                                 uint32_t gch, const uint32_t* hi = nullptr) {
  using GV = GatherVec<W>;
  constexpr int E = GV::kElem;
  constexpr int S = GV::kSteps;
  const size_t Qg = static_cast<size_t>(g.Qg);
  const uint32_t* lanebase = g.values + lane * E;
  uint32_t pbit[GV::kParts];
  part_chunks<W>(pmask, lane, pbit);
  // the next batch's columns and weights are in flight while this one is read
  int32_t nu = 0;
  uint32_t nw = 0;
  if (eb + lane < ee) {
    nu = G.pcol[eb + lane];
    nw = weight_bits<WK>(G.pw, eb + lane);
  }
  for (int64_t e0 = eb; e0 < ee; e0 += 32) {
    const int64_t e = e0 + lane;
    int k = 0;
    const int32_t u = nu;
    const uint32_t wb = nw;
    if (e + 32 < ee) {
      nu = G.pcol[e + 32];
      nw = weight_bits<WK>(G.pw, e + 32);
    }
    uint32_t cm = 0xffffffffu;  // 32-slot chunks of the source row to read
    if (e < ee) {
      if (hi != nullptr) {
        // chunks that may improve the vertex, by the bounds
        cm = bound_chunks<W, WK>(g.blo + static_cast<size_t>(u) * (2 * W), hi, wb) & gch;
        k = __popc(cm) << 5;
      } else if (screen_qs < 0 && g.fsum != nullptr) {
        // sparse frontier: skip in-edges whose source has no gathering
        // frontier chunk, and the source row's chunks without one, by the
        // frontier summary (pairs are counted per 32-slot chunk)
        cm = summary_chunks(g.fsum, lv.level, u) & gch;
        k = __popc(cm) << 5;
      } else if (screen_qs < 0) {
        // the same from the source's W-word mask
        uint64_t m[W];
        load_mask<W>(lv.fcur + static_cast<size_t>(u) * W, m);
        // the next batch's source masks move to L2 while this batch's rows load
        if (e + 32 < ee) prefetch_l2(lv.fcur + static_cast<size_t>(nu) * W);
#pragma unroll
        for (int i = 0; i < W; ++i) {
          m[i] &= sb[i];
          k += __popcll(m[i]);
        }
        if constexpr (kChunks) cm = chunk_bits<W>(m);
      } else {
        k = screen_qs;  // dense frontier: every in-edge is gathered (no mask load)
      }
      ++scanned;
    }
    pairs += static_cast<unsigned long long>(k);
    const unsigned lm = __ballot_sync(kFull, k > 0);
    if (k > 0)
      stage[__popc(lm & ((1u << lane) - 1u))] =
          make_int4(u, static_cast<int>(wb), 0, static_cast<int>(cm));
    __syncwarp();
    const int n = __popc(lm);
    int i = 0;
    uint32_t cur[S][GV::kSlots] = {};
    auto relax = [&](int t) {
      const int4 ed = stage[i + t];
      relax_row<W, WK, kChunks>(best, cur[t], static_cast<uint32_t>(ed.y),
                                static_cast<uint32_t>(ed.w), pbit);
    };
    for (; i + S <= n; i += S) {
      load_rows<W, kChunks, true, S>(lanebase, static_cast<unsigned>(Qg), stage, i, n, pbit, cur);
#pragma unroll
      for (int t = 0; t < S; ++t) relax(t);
    }
    if (i < n) {  // the remaining 1 .. S-1 rows in one step
      load_rows<W, kChunks, false, S>(lanebase, static_cast<unsigned>(Qg), stage, i, n, pbit, cur);
#pragma unroll
      for (int t = 0; t < S; ++t) {
        if (i + t >= n) break;
        relax(t);
      }
    }
    __syncwarp();
  }
}

// The same for the warp-per-vertex kernel below, whose register budget (4 blocks
// of 64 registers per SM at W = 4) holds neither a batch loaded ahead nor the
// predicated row loads: loads under branches, 0xffffffff where nothing is read.
// 120 and 200 slots on R-MAT 20, all lists by warps: 39 and 76 ms against 97 and 119
// with gather_edges_vec.
template <int W, int WK>
__device__ __forceinline__ void gather_vertex_edges(const GroupDev& g, const DevGraph& G,
                                                    const LevelView& lv, uint32_t pmask,
                                                    int64_t eb, int64_t ee, int lane, int4* stage,
                                                    uint32_t (&best)[GatherVec<W>::kSlots],
                                                    unsigned long long& pairs, unsigned& scanned,
                                                    int screen_qs, uint32_t gch) {
  using GV = GatherVec<W>;
  constexpr int E = GV::kElem;
  constexpr int S = GV::kSteps;
  const size_t Qg = static_cast<size_t>(g.Qg);
  const uint32_t* lanebase = g.values + lane * E;
  for (int64_t e0 = eb; e0 < ee; e0 += 32) {
    const int64_t e = e0 + lane;
    int k = 0;
    int32_t u = 0;
    uint32_t wb = 0;
    uint32_t cm = 0xffffffffu;  // 32-slot chunks of the source row to read
    if (e < ee) {
      u = G.pcol[e];
      wb = weight_bits<WK>(G.pw, e);
      if (screen_qs < 0) {
        cm = summary_chunks(g.fsum, lv.level, u) & gch;
        k = __popc(cm) << 5;
      } else {
        k = screen_qs;
      }
      ++scanned;
    }
    pairs += static_cast<unsigned long long>(k);
    const unsigned lm = __ballot_sync(kFull, k > 0);
    if (k > 0)
      stage[__popc(lm & ((1u << lane) - 1u))] =
          make_int4(u, static_cast<int>(wb), 0, static_cast<int>(cm));
    __syncwarp();
    const int n = __popc(lm);
    int i = 0;
    for (; i + S <= n; i += S) {
      int4 ed[S];
#pragma unroll
      for (int t = 0; t < S; ++t) ed[t] = stage[i + t];
      uint32_t cur[S][GV::kSlots];
#pragma unroll
      for (int t = 0; t < S; ++t) {
        const uint32_t* row = lanebase + static_cast<size_t>(ed[t].x) * Qg;
#pragma unroll
        for (int r = 0; r < GV::kParts; ++r) {
          if (((pmask >> r) & 1u) && ((static_cast<uint32_t>(ed[t].w) >> (((32 * r + lane) * E) >> 5)) & 1u)) {
            load_vec_cg<E>(row + 32 * E * r, &cur[t][r * E]);
          } else {
#pragma unroll
            for (int q = 0; q < E; ++q) cur[t][r * E + q] = 0xffffffffu;
          }
        }
      }
#pragma unroll
      for (int t = 0; t < S; ++t) {
#pragma unroll
        for (int j = 0; j < GV::kSlots; ++j)
          best[j] = min(best[j], gather_relax<WK>(cur[t][j], static_cast<uint32_t>(ed[t].y)));
      }
    }
    if (i < n) {
      int4 ed[S];
#pragma unroll
      for (int t = 0; t < S; ++t) ed[t] = stage[i + t < n ? i + t : i];
      uint32_t cur[S][GV::kSlots];
#pragma unroll
      for (int t = 0; t < S; ++t) {
        const uint32_t* row = lanebase + static_cast<size_t>(ed[t].x) * Qg;
#pragma unroll
        for (int r = 0; r < GV::kParts; ++r) {
          if (i + t < n && ((pmask >> r) & 1u) && ((static_cast<uint32_t>(ed[t].w) >> (((32 * r + lane) * E) >> 5)) & 1u)) {
            load_vec_cg<E>(row + 32 * E * r, &cur[t][r * E]);
          } else {
#pragma unroll
            for (int q = 0; q < E; ++q) cur[t][r * E + q] = 0xffffffffu;
          }
        }
      }
#pragma unroll
      for (int t = 0; t < S; ++t) {
#pragma unroll
        for (int j = 0; j < GV::kSlots; ++j)
          best[j] = min(best[j], gather_relax<WK>(cur[t][j], static_cast<uint32_t>(ed[t].y)));
      }
    }
    __syncwarp();
  }
}

// Gather level (vectorised), vertices of in-degree <= heavy_degree.
template <int W, typename OT, int WK>
__global__ void __launch_bounds__(kBlock, (W == 4 ? 4 : (W <= 8 ? 3 : 2))) k_sssp_pull_vec(GroupDev g, DevGraph G) {
  using GV = GatherVec<W>;
  constexpr int E = GV::kElem;
  constexpr int P = GV::kParts;
  const LevelCtl* ctl = g.ctl;
  if (ctl->done || ctl->sdir != kDirPull) return;
  __shared__ int4 s_stage[kWarpsPerBlock][32];
  const LevelView lv = level_view(g);
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  uint32_t pmask, smask;
  gather_vec_masks<W>(ctl->gsel, g.Qg, lane, &pmask, &smask);
  const unsigned long long gw = (static_cast<unsigned long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const unsigned long long nwarps = (static_cast<unsigned long long>(gridDim.x) * blockDim.x) >> 5;
  const size_t Qg = static_cast<size_t>(g.Qg);
  uint32_t uacc = 0;
  unsigned long long improved = 0, pairs = 0;
  unsigned scanned = 0, verts = 0;
  int32_t pend_v = 0;  // lane i: i-th vertex waiting to be appended
  int pend_n = 0;      // uniform
  const int screen_qs = gather_screen_qs<W>(g, ctl, lv, G.E);
  const uint32_t gch = gather_chunks<W>(ctl);
  const unsigned long long V = static_cast<unsigned long long>(G.V);
  // the next vertex's offsets are loaded while the current one is gathered
  int64_t nbeg = 0, nend = 0;
  if (gw < V) {
    nbeg = row_at<OT>(G.prow, static_cast<int64_t>(gw));
    nend = row_at<OT>(G.prow, static_cast<int64_t>(gw) + 1);
  }
  for (unsigned long long vv = gw; vv < V; vv += nwarps) {
    const int32_t v = static_cast<int32_t>(vv);
    const int64_t beg = nbeg, end = nend;
    if (vv + nwarps < V) {
      nbeg = row_at<OT>(G.prow, static_cast<int64_t>(vv + nwarps));
      nend = row_at<OT>(G.prow, static_cast<int64_t>(vv + nwarps) + 1);
    }
    if (end == beg || end - beg > G.heavy_degree) continue;
    if (lane == 0) ++verts;  // one count per vertex, not per lane
    uint32_t* row = g.values + static_cast<size_t>(v) * Qg + lane * E;
    uint32_t best[GV::kSlots];
#pragma unroll
    for (int r = 0; r < P; ++r) {
      if ((pmask >> r) & 1u) {
        load_vec<E>(row + 32 * E * r, &best[r * E]);
      } else {
#pragma unroll
        for (int q = 0; q < E; ++q) best[r * E + q] = 0u;
      }
    }
    gather_vertex_edges<W, WK>(g, G, lv, pmask, beg, end, lane, s_stage[wib], best, pairs, scanned,
                               screen_qs, gch);
    // commit (the warp owns v's row this level: the row read above is current)
    uint32_t imp = 0;
#pragma unroll
    for (int r = 0; r < P; ++r) {
      if (!((pmask >> r) & 1u)) continue;
      uint32_t o[E], nv[E];
      load_vec<E>(row + 32 * E * r, o);
      uint32_t b = 0;
#pragma unroll
      for (int q = 0; q < E; ++q) {
        const int j = r * E + q;
        const bool up = ((smask >> j) & 1u) && best[j] < o[q];
        nv[q] = up ? best[j] : o[q];
        b |= static_cast<uint32_t>(up) << q;
      }
      if (b) store_vec<E>(row + 32 * E * r, nv);
      imp |= b << (r * E);
    }
    if (!__any_sync(kFull, imp != 0)) continue;
    improved += __popc(imp);
    uacc |= imp;
    uint64_t words[P];
    gather_vec_words<W>(imp, lane, words);
    // v is this warp's alone during the kernel (earlier kernels of the level
    // are complete, heavy vertices are not in this kernel): its frontier
    // words and stamp need no atomics
#pragma unroll
    for (int r = 0; r < P; ++r) {
      if (words[r]) {
        const int wi = ((32 * r + lane) * E) >> 6;
        lv.fnext[static_cast<size_t>(v) * W + wi] |= words[r];
      }
    }
    if (g.stamp[v] < lv.level + 1) {  // uniform: every lane reads the same word
      __syncwarp();
      if (lane == 0) g.stamp[v] = lv.level + 1;
      // appends are buffered in the lanes and reserved 32 at a time
      if (lane == pend_n) pend_v = v;
      if (++pend_n == 32) {
        flush_appends<OT>(pend_v, pend_n, G, lv, lane);
        pend_n = 0;
      }
    }
  }
  if (pend_n > 0) flush_appends<OT>(pend_v, pend_n, G, lv, lane);
  {
    uint64_t words[P];
    gather_vec_words<W>(uacc, lane, words);
#pragma unroll
    for (int r = 0; r < P; ++r)
      if (words[r]) atomic_or64(lv.nactive + (((32 * r + lane) * E) >> 6), words[r]);
  }
  warp_add(improved, &g.ctl->lc.improved, lane);
  warp_add(pairs, &g.ctl->lc.sssp_pairs, lane);
  warp_add(scanned, &g.ctl->lc.spull_edges, lane);
  warp_add(verts, &g.ctl->lc.spull_vertices, lane);
}

// Owner of in-edge f0 + lane in a chunk whose vertex k starts at prefix
// position pre_k (lane k passes its own pre_k, INT_MAX beyond the chunk;
// every chunk vertex has an in-edge, so the starts are distinct): the last k
// with pre_k <= f0 + lane.  One ballot and one OR-reduction per 32 in-edges
// instead of a binary search per lane.  All lanes call.
__device__ __forceinline__ int chunk_edge_owner(int my_pre, int f0, int lane) {
  const int k0 = __popc(__ballot_sync(kFull, my_pre <= f0)) - 1;
  // bit (pre_k - f0) for the vertices that start inside (f0, f0 + 32)
  const unsigned d = static_cast<unsigned>(my_pre - f0 - 1);
  const unsigned starts = __reduce_or_sync(kFull, d < 31u ? 2u << d : 0u);
  const unsigned upto = lane == 31 ? 0xffffffffu : (2u << lane) - 1u;
  return k0 + __popc(starts & upto);
}

// ORs each 32-slot chunk's improved bits over the lanes that own its slots and
// hands every chunk's word to one lane: `bits` holds the lane's kSlots bits
// (slot r*kElem + k at bit r*kElem + k); the lane that receives a chunk gets
// its index in *chunk (else -1).  With two parts the halves of the lanes swap
// the part they do not keep, so both are reduced in log2(lanes per chunk)
// shuffles together.
template <int W>
__device__ __forceinline__ uint32_t chunk_word(uint32_t bits, int lane, int* chunk) {
  using GV = GatherVec<W>;
  constexpr int E = GV::kElem;
  constexpr int L = GV::kLanesPerHalf;
  constexpr uint32_t kMask = (1u << E) - 1u;
  const int sh = E * (lane % L);
  uint32_t h;
  if constexpr (GV::kParts == 2) {
    const uint32_t h0 = (bits & kMask) << sh, h1 = ((bits >> E) & kMask) << sh;
    const bool odd = lane & 1;
    h = (odd ? h1 : h0) | __shfl_xor_sync(kFull, odd ? h0 : h1, 1);
#pragma unroll
    for (int o = L / 2; o > 1; o >>= 1) h |= __shfl_xor_sync(kFull, h, o);
    *chunk = lane % L < 2 ? (32 / L) * (lane & 1) + lane / L : -1;
  } else {
    static_assert(GV::kParts == 1, "one or two parts per row slice");
    h = (bits & kMask) << sh;
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) h |= __shfl_xor_sync(kFull, h, o);
    *chunk = lane % L == 0 ? lane / L : -1;
  }
  return h;
}

// Gather level (vectorised), vertices of at most kGatherHeavy in-edges: a warp
// takes an item, a run of up to 32 vertices of about the same in-degree with at
// most kGatherHeavy in-edges in all, and walks the item's in-edges 32 at a
// time.  Each lane screens one in-edge (by the bounds, or by the source's
// frontier chunks); what is left goes to the warp's staging list with one
// entry for the vertex's own row before its first live in-edge, and the rows
// are read kSteps at a time, relaxed in registers and committed when the next
// vertex's own row comes up.  A vertex none of whose in-edges is live costs
// its screening only.  The warp owns its vertices' rows (no distance atomics),
// and the next 32 in-edges and the next item's header are in flight while the
// current ones are worked on.  Groups of more than 256 slots are taken in
// slices of 4 words, slice by slice over all items.
//
// What bounds it: reading rows from L2 where every row is read; the chain column
// -> bound -> row where few are.  The form before it, a CTA per 32 vertices with
// row minima merged in shared memory, spent most of its time outside that: 1.4 ms
// for a level of R-MAT 20 that reads 1% of the row chunks.
constexpr int kRowStage = 64;  // 32 in-edges and as many own rows

struct GatherRowSmem {
  int4 stage[kWarpsPerBlock][kRowStage];
  alignas(16) uint32_t hi[kWarpsPerBlock][32][8];
  alignas(16) uint32_t own[kWarpsPerBlock][256];  // the row of the vertex in work as it was
};

template <int W, typename OT, int WK, int WF>
__device__ __forceinline__ void sssp_pull_light_rows(const GroupDev& g, const DevGraph& G,
                                                     unsigned bid, unsigned nblk,
                                                     GatherRowSmem& sm) {
  static_assert(W <= 4, "a slice is at most 256 slots");
  static_assert(WF % W == 0, "a group is a whole number of slices");
  using GV = GatherVec<W>;
  constexpr int E = GV::kElem;
  constexpr int P = GV::kParts;
  constexpr int S = W == 4 ? 4 : 8;
  const LevelCtl* ctl = g.ctl;
  if (ctl->done || ctl->sdir != kDirPull || G.n_gitems == 0) return;
  const LevelView lv = level_view(g);
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  int4* stage = sm.stage[wib];
  uint32_t(*s_hi)[8] = sm.hi[wib];
  uint32_t* own = sm.own[wib] + lane * E;
  const bool bounds = ctl->bnd_on != 0;
  const bool screened = gather_screen_qs<WF>(g, ctl, lv, G.E) < 0;
  // only this kernel adds bits to its vertices' next masks: plain stores
  const bool plain = !ctl->sscatter && !any_bits<WF>(ctl->bfs_bits);
  const unsigned Qg = static_cast<unsigned>(g.Qg);
  const int n_items = G.n_gitems;
  const int total_items = n_items * (WF / W);
  const int gw = static_cast<int>((bid * blockDim.x + threadIdx.x) >> 5);
  const int nwarps = static_cast<int>((nblk * blockDim.x) >> 5);

  int sl = -1;             // current slice
  uint32_t pmask = 0, smask = 0, gch = 0;
  uint32_t pbit[P];
  int qs = 0;              // gathering slots of the slice
  uint32_t uacc = 0;       // union of the slice's improved bits
  unsigned improved = 0, scanned = 0, verts = 0, pairs = 0;  // of this lane
  int32_t pend_v = 0;      // lane i: i-th vertex waiting to be appended
  int pend_n = 0;          // uniform

  auto flush_union_bits = [&]() {
    int c;
    const uint32_t w = chunk_word<W>(uacc, lane, &c);
    if (c >= 0 && w) {
      const int at = sl * 2 * W + c;  // 32-bit halves of the active words
      atomic_or64(lv.nactive + (at >> 1), static_cast<uint64_t>(w) << (32 * (at & 1)));
    }
    uacc = 0;
  };
  auto flush_pending = [&]() {
    bool fresh = false;
    if (lane < pend_n) fresh = atomicMax(g.stamp + pend_v, lv.level + 1) < lv.level + 1;
    warp_append(fresh, pend_v, fresh ? degree_of<OT>(G.row, pend_v) : 0, lv.nlist, lv.ncount,
                lv.nedges, lane);
    pend_n = 0;
  };

  // header of the next item: lane k holds its k-th vertex
  int32_t hv = 0, hpre = 0;
  OT hbeg = 0;
  int hnv = 0;
  auto load_header = [&](int it) {
    const int i = WF > W ? it % n_items : it;
    const int cs = G.gitem_start[i];
    hnv = G.gitem_start[i + 1] - cs;
    if (lane < hnv) {
      hv = G.plight[cs + lane];
      hbeg = static_cast<OT>(G.plight_beg[cs + lane]);
      hpre = G.gitem_pre[cs + lane];
    }
  };
  if (gw < total_items) load_header(gw);
  for (int it = gw; it < total_items; it += nwarps) {
    const int nsl = WF > W ? it / n_items : 0;
    if (nsl != sl) {
      if (sl >= 0) flush_union_bits();
      sl = nsl;
      const uint64_t* sb = ctl->gsel + sl * W;
      gather_vec_masks<W>(sb, g.Qg - sl * 64 * W, lane, &pmask, &smask);
      gch = gather_chunks<W>(sb);
      part_chunks<W>(pmask, lane, pbit);
      qs = 0;
#pragma unroll
      for (int i = 0; i < W; ++i) qs += __popcll(sb[i]);
    }
    const int nv = hnv;
    const int32_t v = hv;
    const int total = __shfl_sync(kFull, hpre, nv - 1);
    int start = __shfl_up_sync(kFull, hpre, 1);
    if (lane == 0) start = 0;
    const OT base = hbeg - start;  // in-edge f of the item: base + f
    if (lane >= nv) start = 0x7fffffff;
    if (it + nwarps < total_items) load_header(it + nwarps);
    if (gch == 0) continue;  // no gathering slot in this slice
    const size_t hoff = static_cast<size_t>(sl) * 2 * W;  // the slice's chunks in the bounds
    if (bounds) {
      constexpr int N = 2 * W < 4 ? 2 : 4;
      if (lane < nv) {
        const uint32_t* hi = g.bhi + static_cast<size_t>(v) * (2 * WF) + hoff;
#pragma unroll
        for (int i = 0; i < 2 * W; i += N) {
          uint32_t x[N];
          load_vec<N>(hi + i, x);
          store_vec<N>(&s_hi[lane][i], x);
        }
      }
      __syncwarp();
    }
    if (sl == 0) {
      verts += lane == 0 ? nv : 0;
      for (int f = lane; f < total; f += 32) ++scanned;
    }
    const uint32_t* lanebase = g.values + sl * 64 * W + lane * E;
    uint32_t best[GV::kSlots];
    int cur_k = -1;     // vertex in work (uniform)
    int32_t cur_v = 0;
    auto commit = [&]() {
      uint32_t imp = 0;
#pragma unroll
      for (int r = 0; r < P; ++r) {
        uint32_t b = 0, o[E];
        load_vec<E>(&own[32 * E * r], o);
#pragma unroll
        for (int q = 0; q < E; ++q) {
          const int j = r * E + q;
          const bool up = ((smask >> j) & 1u) && best[j] < o[q];
          best[j] = up ? best[j] : o[q];
          b |= static_cast<uint32_t>(up) << q;
        }
        if (b) store_vec<E>(const_cast<uint32_t*>(lanebase) + static_cast<uint64_t>(static_cast<uint32_t>(cur_v)) * Qg + 32 * E * r, &best[r * E]);
        imp |= b << (r * E);
      }
      if (!__any_sync(kFull, imp != 0)) return;
      improved += __popc(imp);
      uacc |= imp;
      int c;
      const uint32_t w = chunk_word<W>(imp, lane, &c);
      if (c >= 0 && w) {
        uint32_t* fw = reinterpret_cast<uint32_t*>(lv.fnext + static_cast<size_t>(cur_v) * WF) + hoff + c;
        if (plain) *fw = w;
        else atomicOr(fw, w);
      }
      if (lane == pend_n) pend_v = cur_v;
      if (++pend_n == 32) flush_pending();
    };

    // the staged rows: an own row commits the vertex before it and starts its
    // vertex, the others are relaxed into it
    auto walk = [&](auto chunks, int n) {
      constexpr bool kChunks = decltype(chunks)::value;
      uint32_t cur[S][GV::kSlots] = {};
      int i = 0;
      auto take = [&](int t) {
        const int4 ed = stage[i + t];
        if (ed.z < 0) {  // uniform
          if (cur_k >= 0) commit();
          cur_k = ~ed.z;
          cur_v = ed.x;
#pragma unroll
          for (int j = 0; j < GV::kSlots; ++j) best[j] = cur[t][j];
#pragma unroll
          for (int r = 0; r < P; ++r) store_vec<E>(&own[32 * E * r], &best[r * E]);
        } else {
          relax_row<W, WK, kChunks>(best, cur[t], static_cast<uint32_t>(ed.y),
                                    static_cast<uint32_t>(ed.w), pbit);
        }
      };
      for (; i + S <= n; i += S) {
        load_rows<W, kChunks, true, S>(lanebase, Qg, stage, i, n, pbit, cur);
#pragma unroll
        for (int t = 0; t < S; ++t) take(t);
      }
      if (i < n) {
        load_rows<W, kChunks, false, S>(lanebase, Qg, stage, i, n, pbit, cur);
#pragma unroll
        for (int t = 0; t < S; ++t) {
          if (i + t >= n) break;  // uniform
          take(t);
        }
      }
    };

    // in-edges f0 .. f0 + 31, lane by lane (the next batch is loaded ahead)
    int nk = 0;
    int32_t nu = 0;
    uint32_t nw = 0;
    auto load_batch = [&](int f0) {
      nk = chunk_edge_owner(start, f0, lane);
      const OT e = __shfl_sync(kFull, base, nk) + f0 + lane;
      if (f0 + lane < total) {
        nu = G.pcol[e];
        nw = weight_bits<WK>(G.pw, e);
      }
    };
    load_batch(0);
    for (int f0 = 0; f0 < total; f0 += 32) {
      const int k = nk;
      const int32_t u = nu;
      const uint32_t wb = nw;
      uint32_t cm = 0;
      if (f0 + lane < total) {
        if (bounds)
          cm = bound_chunks<W, WK>(g.blo + static_cast<size_t>(u) * (2 * WF) + hoff, s_hi[k], wb) & gch;
        else if (!screened)
          cm = gch;
        else
          cm = (summary_chunks(g.fsum, lv.level, u) >> hoff) & gch;
      }
      if (f0 + 32 < total) load_batch(f0 + 32);
      const bool live = cm != 0;
      const unsigned lm = __ballot_sync(kFull, live);
      if (lm == 0) continue;
      pairs += (bounds || screened) ? static_cast<unsigned>(__popc(cm)) << 5
                                    : (live ? static_cast<unsigned>(qs) : 0u);
      // the vertex's own row goes before its first live in-edge
      const unsigned lb = lm & below;
      const int kp = __shfl_sync(kFull, k, lb ? 31 - __clz(lb) : lane);
      const bool first = live && k != (lb ? kp : cur_k);
      const unsigned fm = __ballot_sync(kFull, first);
      const int pos = __popc(lb) + __popc(fm & (below | (1u << lane)));
      const int32_t vk = __shfl_sync(kFull, v, k);
      if (live) stage[pos] = make_int4(u, static_cast<int>(wb), k, static_cast<int>(cm));
      if (first) stage[pos - 1] = make_int4(vk, 0, ~k, static_cast<int>(gch));
      __syncwarp();
      const int n = __popc(lm) + __popc(fm);
      if (bounds || screened) walk(std::true_type{}, n);
      else walk(std::false_type{}, n);
      __syncwarp();
    }
    if (cur_k >= 0) commit();
  }
  if (pend_n > 0) flush_pending();
  if (sl >= 0) flush_union_bits();
  warp_add(improved, &g.ctl->lc.improved, lane);
  warp_add(pairs, &g.ctl->lc.sssp_pairs, lane);
  warp_add(scanned, &g.ctl->lc.spull_edges, lane);
  warp_add(verts, &g.ctl->lc.spull_vertices, lane);
}

template <int W, typename OT, int WK, int WF = W>
__global__ void __launch_bounds__(kBlock, 3) k_sssp_pull_rows(GroupDev g, DevGraph G) {
  __shared__ GatherRowSmem sm;
  sssp_pull_light_rows<W, OT, WK, WF>(g, G, blockIdx.x, gridDim.x, sm);
}

// Gather level (vectorised), heavy vertices: CTA per 2048-edge chunk, warps
// min-reduce their slices into shared memory, one atomicMin per slot.
// kMode 0: every gather level, whole source rows; 1: only levels that read
// whole rows (dense entries); 2: only screened levels (sparse entries), with
// the source rows' 32-slot chunks without frontier bits skipped; 3: every
// gather level, skipping as 2 does on screened ones.  Modes 1 and 2
// are launched together (groups of <= 256 slots) so that each level runs the
// variant whose register budget suits it.
template <int W>
struct GatherHeavySmem {
  alignas(16) uint32_t best[64 * W];
  alignas(16) uint32_t hi[2 * W];
  int4 stage[kWarpsPerBlock][32];
};

template <int W, typename OT, int WK, int kMode>
__device__ __forceinline__ void sssp_pull_heavy_chunks(const GroupDev& g, const DevGraph& G,
                                                       unsigned bid, unsigned nblk,
                                                       GatherHeavySmem<W>& sm) {
  uint32_t (&s_best)[64 * W] = sm.best;
  int4 (&s_stage)[kWarpsPerBlock][32] = sm.stage;
  using GV = GatherVec<W>;
  constexpr int E = GV::kElem;
  constexpr int C = 2 * W;
  const LevelCtl* ctl = g.ctl;
  if (ctl->done || ctl->sdir != kDirPull || G.n_sheavy == 0) return;
  const LevelView lv = level_view(g);
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const uint64_t* sb = ctl->gsel;
  uint32_t pmask, smask;
  gather_vec_masks<W>(ctl->gsel, g.Qg, lane, &pmask, &smask);
  const uint32_t lsel = lane_sssp_chunks<W>(ctl, lane);
  const int screen_qs = gather_screen_qs<W>(g, ctl, lv, G.E);
  const uint32_t gch = gather_chunks<W>(ctl);
  const bool bounds = ctl->bnd_on != 0;
  const bool screened = screen_qs < 0 || bounds;
  if ((kMode == 1 && screened) || (kMode == 2 && !screened)) return;
  const size_t Qg = static_cast<size_t>(g.Qg);
  uint64_t uni[W];
#pragma unroll
  for (int i = 0; i < W; ++i) uni[i] = 0;
  unsigned long long improved = 0, pairs = 0;
  unsigned scanned = 0;
  // every heavy vertex is gathered once per launch (all its chunks)
  if (bid == 0 && threadIdx.x == 0)
    atomicAdd(&g.ctl->lc.spull_vertices, static_cast<unsigned long long>(G.n_sheavy));
  // the chunk's vertex and edge range: independent loads, no search, and made
  // a chunk ahead
  int32_t nv = 0;
  int64_t ncb = 0, nce = 0;
  auto header = [&](int64_t ch) {
    nv = G.sheavy[G.sheavy_ch[ch]];
    ncb = G.sheavy_cb[ch];
    nce = G.sheavy_ce[ch];
  };
  if (bid < G.sheavy_chunks) header(bid);
  for (int64_t ch = bid; ch < G.sheavy_chunks; ch += nblk) {
    const int32_t v = nv;
    const int64_t cb = ncb, ce = nce;
    if (ch + nblk < G.sheavy_chunks) header(ch + nblk);
    for (int i = threadIdx.x; i < C * 32; i += blockDim.x) s_best[i] = 0xffffffffu;
    if (bounds && threadIdx.x < C) sm.hi[threadIdx.x] = g.bhi[static_cast<size_t>(v) * C + threadIdx.x];
    __syncthreads();
    const int64_t seg = (ce - cb + kWarpsPerBlock - 1) / kWarpsPerBlock;
    const int64_t wb = cb + wib * seg;
    const int64_t we = min(ce, wb + seg);
    uint32_t best[GV::kSlots];
#pragma unroll
    for (int j = 0; j < GV::kSlots; ++j) best[j] = 0xffffffffu;
    gather_edges_vec<W, WK, (kMode >= 2)>(g, G, lv, sb, pmask, wb, we, lane, s_stage[wib], best,
                                        pairs, scanned, screen_qs, gch, bounds ? sm.hi : nullptr);
#pragma unroll
    for (int j = 0; j < GV::kSlots; ++j) {
      const int q = (32 * (j / E) + lane) * E + (j % E);
      if (((smask >> j) & 1u) && best[j] != 0xffffffffu) atomicMin(&s_best[q], best[j]);
    }
    __syncthreads();
    // commit: warp wib takes 32-slot chunks wib, wib + 8, ... (lane j <-> slot 32c + j)
    bool any = false;
    for (int c = wib; c < C; c += kWarpsPerBlock) {
      const int q = 32 * c + lane;
      bool imp = false;
      if ((lsel >> c) & 1u) {
        const uint32_t b = s_best[q];
        uint32_t* p = g.values + static_cast<size_t>(v) * Qg + q;
        if (b < *p) imp = b < atomicMin(p, b);
      }
      const unsigned m = __ballot_sync(kFull, imp);
      if (m) {
        any = true;
        if (lane == 0) {
          const uint64_t bits = static_cast<uint64_t>(m) << (32 * (c & 1));
          atomic_or64(lv.fnext + static_cast<size_t>(v) * W + (c >> 1), bits);
          uni[c >> 1] |= bits;
          improved += __popc(m);
        }
      }
    }
    bool app = false;
    if (any && lane == 0) app = atomicMax(g.stamp + v, lv.level + 1) < lv.level + 1;
    // one append per improved vertex-chunk: rare, a plain warp append
    warp_append(app, v, app ? degree_of<OT>(G.row, v) : 0, lv.nlist, lv.ncount, lv.nedges, lane);
    __syncthreads();
  }
  flush_union<W>(uni, lv.nactive, lane);
  warp_add(improved, &g.ctl->lc.improved, lane);
  warp_add(pairs, &g.ctl->lc.sssp_pairs, lane);
  warp_add(scanned, &g.ctl->lc.spull_edges, lane);
}

template <int W, typename OT, int WK, int kMode>
__global__ void __launch_bounds__(kBlock, (W <= 4 ? 3 : 2)) k_sssp_pull_heavy_vec(GroupDev g, DevGraph G) {
  __shared__ GatherHeavySmem<W> sm;
  sssp_pull_heavy_chunks<W, OT, WK, kMode>(g, G, blockIdx.x, gridDim.x, sm);
}

// --------------------------------------------------------- level control
__device__ __forceinline__ int32_t decide_dir(const LevelCtl* ctl, unsigned long long count,
                                              unsigned long long edges, bool has_bfs) {
  if (!has_bfs) return kDirPush;
  if (ctl->forced_dir >= 0) return ctl->forced_dir;
  if (ctl->mode == 0) return kDirPush;   // CGP_MODE_PUSH
  if (ctl->mode == 1) return kDirPull;   // CGP_MODE_PULL
  return (edges >= ctl->pull_edge_threshold || count >= ctl->pull_vertex_threshold)
             ? kDirPull : kDirPush;
}

// Group-wide SSSP direction of a level whose frontier has `count` vertices
// and `edges` out-edges.  Hybrid: gather when the edges reach the edge
// threshold and the estimated (edge, slot) pairs a scatter would relax — the
// previous level's improvements x the frontier's mean out-degree — reach
// sssp_pull_pair_unit per SSSP 32-slot chunk: a scatter costs per pair, a
// gather per (in-edge, gathering chunk), so a wide group whose frontier
// carries one or two bits per vertex (a grid's first and last levels) keeps
// scattering although its frontier touches half the edges.
template <int W>
__device__ __forceinline__ int32_t decide_sdir(const LevelCtl* ctl, unsigned long long count,
                                               unsigned long long edges) {
  if (!any_bits<W>(ctl->sssp_bits) || !ctl->sssp_gather) return kDirPush;
  if (ctl->forced_dir >= 0) return ctl->forced_dir;
  if (ctl->mode == 0) return kDirPush;
  if (ctl->mode == 1) return kDirPull;
  if (edges < ctl->sssp_pull_edge_threshold) return kDirPush;
  if (ctl->sssp_pull_pair_unit > 0) {
    int chunks = 0;
    for (int i = 0; i < W; ++i)
      chunks += (static_cast<uint32_t>(ctl->sssp_bits[i]) != 0u) + ((ctl->sssp_bits[i] >> 32) != 0ULL);
    if (ctl->bnd_good) chunks = 1;  // a gather that skips most chunks costs its edge scan
    const double pairs = static_cast<double>(ctl->prev_improved) * static_cast<double>(edges) /
                         static_cast<double>(count > 0 ? count : 1ULL);
    if (pairs < static_cast<double>(ctl->sssp_pull_pair_unit) * chunks) return kDirPush;
  }
  return kDirPull;
}

// Splits the SSSP slots of the next level into gathering (gsel) and
// scattering (ssel) ones.  Group-wide by default (every slot takes
// `group_dir`); with chunk_dir in hybrid mode each 32-slot chunk gathers when
// the out-edges of the next frontier's vertices that carry one of its bits
// (cedges, summed by k_chunk_census) reach the gather threshold and the
// chunk's (edge, slot) pairs (cpairs) reach sssp_pull_pair_unit, so a few
// queries in their dense phase do not make every other slot gather too, and a
// chunk whose last improvements are few scatters them.  Consumes (zeroes)
// cedges and cpairs.
template <int W>
__device__ __forceinline__ void split_sssp_slots(LevelCtl* ctl, int32_t group_dir, int lane) {
  const bool per_chunk = ctl->chunk_dir && ctl->mode == 2 && ctl->forced_dir < 0 &&
                         ctl->sssp_gather;
  // lane c: 32-slot chunk c, half (c & 1) of word c / 2
  uint32_t bits = 0, gat = 0;
  if (lane < 2 * W) {
    bits = reinterpret_cast<const uint32_t*>(ctl->sssp_bits)[lane];
    if (per_chunk) {
      // as the group rule: enough frontier edges, and enough (edge, slot)
      // pairs that a scatter would cost more than the chunk's gather
      if (ctl->cedges[lane] >= ctl->sssp_pull_edge_threshold &&
          (ctl->sssp_pull_pair_unit == 0 || ctl->cpairs[lane] >= ctl->sssp_pull_pair_unit))
        gat = bits;
    } else if (group_dir == kDirPull) {
      gat = bits;
    }
    reinterpret_cast<uint32_t*>(ctl->gsel)[lane] = gat;
    reinterpret_cast<uint32_t*>(ctl->ssel)[lane] = bits & ~gat;
  }
  if (lane < 2 * kMaxW) ctl->cedges[lane] = ctl->cpairs[lane] = 0;
  const unsigned with = __ballot_sync(kFull, bits != 0u);
  const unsigned gathering = __ballot_sync(kFull, gat != 0u);
  const unsigned scattering = __ballot_sync(kFull, (bits & ~gat) != 0u);
  if (lane == 0) {
    ctl->sssp_chunk_levels += __popc(with);
    ctl->gather_chunk_levels += __popc(gathering);
    ctl->sdir = gathering ? kDirPull : kDirPush;
    ctl->sscatter = scattering ? 1 : 0;
  }
  __syncwarp();
}

// Expand mask for `level`: k-hop slots stop once their depth reaches k.  Lane
// j takes slot 32c + j of every 32-slot chunk c (one 16-byte load each, a
// ballot per chunk): a single thread walking the slots paid one dependent
// load per slot, 45 us per level end at 256 slots.
template <int W>
__device__ __forceinline__ void compute_expand(LevelCtl* ctl, const SlotDev* slots, int Qg,
                                               int level, int lane) {
#pragma unroll
  for (int c = 0; c < 2 * W; ++c) {
    const int q = 32 * c + lane;
    bool stop = false;
    if (q < Qg) {
      const int4 s = *reinterpret_cast<const int4*>(slots + q);  // kind, source, k, base
      stop = s.x == 3 && level - s.w >= s.z;
    }
    const unsigned m = __ballot_sync(kFull, stop);
    if (lane == 0) reinterpret_cast<uint32_t*>(ctl->expand)[c] = ~m;
  }
  __syncwarp();
}

// End of a level (one warp, all lanes call): profile, convergence, and the
// set-up of the next level (counter reset, direction, expand mask).
template <int W>
__device__ __forceinline__ void level_end(const GroupDev& g, int lane) {
  LevelCtl* ctl = g.ctl;
  if (ctl->done) return;
  const int l = ctl->level;
  const int par = l & 1;
  const unsigned long long count = ctl->count[par], edges = ctl->edges[par];
  const unsigned long long nextc = ctl->count[par ^ 1], nexte = ctl->edges[par ^ 1];
  const bool gathered = ctl->sdir == kDirPull;
  __syncwarp();
  if (lane < W) ctl->active[par][lane] = 0;
  if (lane == 0) {
    const LevelCounters lc = ctl->lc;
    if (g.prof != nullptr && l < ctl->profile_cap) {
      LevelProfile p;
      p.level = l;
      p.dir = ctl->dir;
      p.frontier = count;
      p.edges = edges;
      p.next = nextc;
      p.active0 = ctl->active[par ^ 1][0];
      p.new_pairs = lc.new_pairs;
      p.pull_vertices = lc.pull_vertices;
      p.pull_edges = lc.pull_edges;
      p.sssp_pairs = lc.sssp_pairs;
      p.sssp_active = lc.sssp_active;
      p.improved = lc.improved;
      p.spull_vertices = lc.spull_vertices;
      p.spull_edges = lc.spull_edges;
      p.sdir = ctl->sdir;
      p.reserved = 0;
      g.prof[l] = p;
    }
    LevelCounters t = ctl->total;
    t.new_pairs += lc.new_pairs;
    t.pull_vertices += lc.pull_vertices;
    t.pull_edges += lc.pull_edges;
    t.sssp_pairs += lc.sssp_pairs;
    t.sssp_active += lc.sssp_active;
    t.improved += lc.improved;
    t.spull_vertices += lc.spull_vertices;
    t.spull_edges += lc.spull_edges;
    ctl->total = t;
    ctl->prev_improved = lc.improved;
    ctl->prev_pull_edges = lc.pull_edges;
    ctl->prev_dir = ctl->dir;
    if (gathered) {
      ctl->gathers++;
      if (ctl->bnd_on) {
        // chunks read against the live ones: a level that kept more than 13/16
        // of them was not worth its pass over the values
        const unsigned long long read = lc.sssp_pairs / 32, live = lc.live_chunks;
        ctl->bnd_good = 2 * read <= live ? 1 : 0;
        const bool fail = 16 * read > 13 * live;
        ctl->bnd_fail = fail ? min(ctl->bnd_fail + 1, 5) : 0;
        ctl->bnd_wait = fail ? 4 << ctl->bnd_fail : 0;
      }
    }
    ctl->lc = LevelCounters{};
    ctl->dense_count = 0;
    ctl->hq_packed = 0;
    ctl->total_frontier += count;
    ctl->total_edges += edges;
    if (ctl->dir == kDirPush) ctl->push_levels++;
    else ctl->pull_levels++;
    ctl->level = l + 1;
    // Set up level l+1 even when it is empty, so that a serving loop can add
    // sources to it and resume.
    ctl->prev_count = count;
    ctl->count[par] = 0;
    ctl->edges[par] = 0;
  }
  __syncwarp();
  if (ctl->khop) compute_expand<W>(ctl, g.slots, g.Qg, l + 1, lane);
  const int32_t dir = decide_dir(ctl, nextc, nexte, any_bits<W>(ctl->bfs_bits));
  split_sssp_slots<W>(ctl, decide_sdir<W>(ctl, nextc, nexte), lane);
  if (lane != 0) return;
  ctl->dir = dir;
  // bounds: not before a first gather level has reached the bulk of the
  // vertices, then on every gather level as long as they skip enough
  if (ctl->bnd_avail && ctl->sdir == kDirPull && ctl->gathers > 0) {
    ctl->bnd_on = ctl->bnd_wait == 0 ? 1 : 0;
    if (ctl->bnd_wait > 0) ctl->bnd_wait--;
  } else {
    ctl->bnd_on = 0;
  }
  if (nextc == 0 || (ctl->max_iterations > 0 && l + 1 >= ctl->max_iterations)) {
    ctl->done = 1;
    return;
  }
  // Pauses (done = 2): depth planes hold depths < 2^num_planes and level l+1
  // writes depth l+2; or the caller asked to stop at halt_level.  The host
  // resumes by clearing `done`.
  if (ctl->num_planes > 0 && ((l + 2) >> ctl->num_planes) != 0) {
    ctl->status |= kStatusPlanesExhausted;
    ctl->done = 2;
  }
  if (ctl->halt_level >= 0 && l + 1 >= ctl->halt_level) ctl->done = 2;
}

template <int W>
__global__ void k_level_end(GroupDev g) {
  level_end<W>(g, static_cast<int>(threadIdx.x));
}

// Per 32-slot chunk, the out-edges of the next frontier's vertices that carry
// an SSSP bit of the chunk (input of the per-chunk direction decision).  Runs
// after the level's kernels, before its level end: each lane takes a vertex
// of the next frontier list, the warp sums its chunks, lane 0 adds them.
template <int W, typename OT>
__device__ __forceinline__ void chunk_census(const GroupDev& g, const DevGraph& G, unsigned bid,
                                             unsigned nblk) {
  LevelCtl* ctl = g.ctl;
  if (ctl->done || !ctl->chunk_dir) return;
  const LevelView lv = level_view(g);
  const unsigned long long n = *lv.ncount;
  const int lane = threadIdx.x & 31;
  unsigned long long acc[2 * W], pacc[2 * W];
#pragma unroll
  for (int c = 0; c < 2 * W; ++c) acc[c] = pacc[c] = 0;
  const unsigned long long stride = static_cast<unsigned long long>(nblk) * blockDim.x;
  for (unsigned long long i0 = static_cast<unsigned long long>(bid) * blockDim.x + (threadIdx.x & ~31);
       i0 < n; i0 += stride) {
    const unsigned long long i = i0 + lane;
    if (i < n) {
      const int32_t v = lv.nlist[i];
      const unsigned long long d = degree_of<OT>(G.row, v);
      uint64_t m[W];
      load_mask<W>(lv.fnext + static_cast<size_t>(v) * W, m);
#pragma unroll
      for (int w = 0; w < W; ++w) {
        const uint64_t x = m[w] & ctl->sssp_bits[w];
        const int lo = __popc(static_cast<uint32_t>(x)), hi = __popc(static_cast<uint32_t>(x >> 32));
        if (lo) acc[2 * w] += d;
        if (hi) acc[2 * w + 1] += d;
        pacc[2 * w] += d * static_cast<unsigned long long>(lo);
        pacc[2 * w + 1] += d * static_cast<unsigned long long>(hi);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 2 * W; ++c) {
    unsigned long long x = acc[c], y = pacc[c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      x += __shfl_xor_sync(kFull, x, o);
      y += __shfl_xor_sync(kFull, y, o);
    }
    if (lane == 0 && x) {
      atomicAdd(&ctl->cedges[c], x);
      atomicAdd(&ctl->cpairs[c], y);
    }
  }
}

template <int W, typename OT>
__global__ void __launch_bounds__(kBlock) k_chunk_census(GroupDev g, DevGraph G) {
  chunk_census<W, OT>(g, G, blockIdx.x, gridDim.x);
}

// Level end inside a device-looped CUDA graph (a WHILE conditional node whose
// body is one level): sets the loop condition from the done flag, so the
// whole traversal runs without the host.  A traversal that is still running
// at `level_cap` levels (more than any converging BFS/SSSP needs) stops with
// kStatusLevelCap instead of looping on.
template <int W>
__global__ void k_level_end_loop(GroupDev g, cudaGraphConditionalHandle loop, int32_t level_cap) {
  level_end<W>(g, static_cast<int>(threadIdx.x));
  if (threadIdx.x != 0) return;
  LevelCtl* ctl = g.ctl;
  if (ctl->done == 0 && ctl->level >= level_cap) {
    ctl->status |= kStatusLevelCap;
    ctl->done = 3;
  }
  cudaGraphSetConditional(loop, ctl->done == 0 ? 1u : 0u);
}

// ------------------------------------------------------- fused level loop
// Barrier over all blocks of a cooperative launch.  The last block to arrive
// runs `last(lane)` with its first warp before it lets the others go, so the
// end of a level costs no barrier of its own.  A wait gives up after
// ctl->bar_limit_ns (the other blocks are co-resident, so this means the device is
// not running them), raises kStatusBarrier and tells every block to leave: wait()
// then returns false in all of them.

__device__ __forceinline__ unsigned load_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void store_release(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

struct GridBarrier {
  LevelCtl* ctl;
  unsigned nblk;
  unsigned epoch;  // barriers passed

  // Every block reads the epoch before it first arrives, so none can miss a
  // release of this launch.
  __device__ __forceinline__ GridBarrier(LevelCtl* c, unsigned n)
      : ctl(c), nblk(n), epoch(load_acquire(&c->bar_release)) {}

  template <typename F>
  __device__ __forceinline__ bool wait(F&& last) {
    __shared__ int s_ok;
    ++epoch;
    __syncthreads();
    if (threadIdx.x < 32) {
      const int lane = static_cast<int>(threadIdx.x);
      unsigned before = 0;
      if (lane == 0) {
        __threadfence();
        before = atomicAdd(&ctl->bar_arrived, 1u);
      }
      before = __shfl_sync(kFull, before, 0);
      bool ok = true;
      if (before == nblk - 1) {
        __threadfence();  // every lane: the other blocks' writes of the phase
        last(lane);
        if (lane == 0) ctl->bar_arrived = 0;
        __threadfence();
        __syncwarp();
        if (lane == 0) store_release(&ctl->bar_release, epoch);
      } else if (lane == 0) {
        unsigned long long t0 = 0;
        for (unsigned spins = 0; load_acquire(&ctl->bar_release) != epoch; ++spins) {
          if ((spins & 255u) != 255u) continue;
          if (load_acquire(&ctl->bar_abort) != 0) {
            ok = false;
            break;
          }
          const unsigned long long t = global_ns();
          if (t0 == 0) t0 = t;
          if (t - t0 > ctl->bar_limit_ns) {
            atomicOr(&ctl->status, kStatusBarrier);
            __threadfence();
            store_release(&ctl->bar_abort, 1u);
            ok = false;
            break;
          }
        }
      }
      if (lane == 0) s_ok = ok ? 1 : 0;
      __threadfence();
    }
    __syncthreads();
    return s_ok != 0;
  }

  __device__ __forceinline__ bool wait() {
    return wait([](int) {});
  }
};

template <int W, bool kSssp>
union TraverseSmem {
  PushSmem<W> push;
  HeavySlotSmem slot;
  PullHeavySmem<W> pull_heavy;
  SsspPushSmem<kSssp ? W : 1> sssp_push;
  SsspListSmem<kSssp ? W : 1> sssp_list;
  SsspHeavySmem<kSssp ? W : 1> sssp_heavy;
  GatherHeavySmem<kSssp ? W : 1> gather_heavy;
  GatherRowSmem gather_light;
};

// Up to `levels` whole levels in one cooperative launch: the phases that are
// kernels of their own in the launched form (see enqueue_level_t) run one
// after another with a grid barrier wherever one reads what another wrote,
// and the level end runs in the last block to reach the level's last barrier.
// A launched level is 10 to 16 dependent kernels, most of which find nothing
// to do; with small graphs and in the first and last levels of deep ones
// their launches are the level's whole time.
template <int W, typename OT, int DEPTH, int WK, bool kSssp>
__global__ void __launch_bounds__(kBlock, 3) k_traverse(GroupDev g, DevGraph G,
                                                        int levels, int flags) {
  static_assert(W <= 4, "wider groups are launched level by level");
  __shared__ TraverseSmem<W, kSssp> sm;
  const unsigned bid = blockIdx.x, nblk = gridDim.x;
  LevelCtl* ctl = g.ctl;
  // held across the levels, a limit or a count of blocks of its own would cost the
  // phases registers they do not have
  GridBarrier bar(ctl, nblk);
  const bool heavy = flags & kTraverseHeavy;
  if ((flags & kTraverseBlockMissing) && bid == 0) return;
  bool swept = false;  // the previous level zeroed its own frontier's masks
  for (int l = 0; l < levels; ++l) {
    if (ctl->done) return;
    const bool bfs = !kSssp || ctl->has_bfs != 0;
    const bool bfs_pull = bfs && ctl->dir == kDirPull;
    const bool gather = kSssp && ctl->sdir == kDirPull;
    const bool scatter = kSssp && ctl->sscatter != 0;
    const bool queue = heavy && ((bfs && !bfs_pull) || scatter);
    const bool queued_lists = scatter && ctl->count[ctl->level & 1] > kInlineLists;
    bool summary = gather;
    if (bfs) summary |= bfs_pull_uses_summary(g, ctl, level_view(g), G.V);
    // what the level's phases read or add to; a pull over whole masks alone
    // rewrites every next mask and needs nothing prepared
    const bool clear = ctl->dir == kDirPush && !swept && ctl->prev_count > 0;
    if (clear || summary || queue) {
      if (clear) clear_next<W>(g, G.E, bid, nblk);
      if (summary) frontier_summary<W, OT>(g, G, bid, nblk);
      if constexpr (kSssp) gather_bounds<W, OT, WK>(g, G, bid, nblk);
      if (queue) heavy_queue_scan<OT>(g, G, bid, nblk);
      if (!bar.wait()) return;
    }
    // A scattering level whose vertices are all expanded by the tiles reads each
    // mask once and can zero it there: the next level has nothing to clear, and
    // a level of a road-like graph is one phase and one barrier.
    const bool sweep = !(bfs && kSssp) && !heavy && !bfs_pull && !gather && !queued_lists;
    swept = sweep;
    if (bfs) {
      if (!bfs_pull) {
        bfs_push_tiles<W, OT, DEPTH>(g, G, bid, nblk, sm.push, sweep);
        if (heavy) {
          __syncthreads();
          bfs_push_chunks<W, OT, DEPTH>(g, G, nblk - 1 - bid, nblk, sm.slot);
        }
      } else {
        bfs_pull_tiles<W, OT, DEPTH>(g, G, bid, nblk);
        bfs_pull_mid<W, OT, DEPTH>(g, G, bid, nblk);
        if (G.n_pheavy > 0) {
          bfs_pull_chunks<W, OT>(g, G, bid, nblk, sm.pull_heavy);
          if (!bar.wait()) return;
          bfs_pull_heavy_commit<W, OT, DEPTH>(g, G, bid, nblk);
        }
        // the pull stores whole next masks: SSSP bits are added afterwards
        if (kSssp && (scatter || gather) && !bar.wait()) return;
      }
      __syncthreads();
    }
    if constexpr (kSssp) {
      if (scatter) {
        sssp_push_tiles<W, OT, WK>(g, G, bid, nblk, sm.sssp_push, sweep);
        if (heavy) {
          __syncthreads();
          sssp_push_chunks<W, OT, WK>(g, G, nblk - 1 - bid, nblk, sm.sssp_heavy);
        }
        if (queued_lists) {
          if (!bar.wait()) return;  // the queue is complete
          sssp_list_vertices<W, OT, WK, 4>(g, G, bid, nblk, sm.sssp_list);
        }
        // a gather stores whole vectors of a row
        if (gather && !bar.wait()) return;
      }
      if (gather) {
        // heavy vertices first: the light ones read their lowered distances
        if (G.n_sheavy > 0)
          sssp_pull_heavy_chunks<W, OT, WK, 3>(g, G, bid, nblk, sm.gather_heavy);
        // The light gather stores whole vectors of a row: depths a push of this
        // level writes into the same vectors must be in place before their row is
        // read.  After a scatter or a pull they are; the heavy gather only lowers
        // its own words and may run beside a push.  (Read again: as values kept over
        // the heavy gather the level's flags cost it spills.)
        const bool pushed = ctl->has_bfs && ctl->dir == kDirPush && !ctl->sscatter;
        if ((G.n_sheavy > 0 || pushed) && !bar.wait()) return;
        sssp_pull_light_rows<W, OT, WK, W>(g, G, bid, nblk, sm.gather_light);
      }
      if (ctl->chunk_dir) {
        if (!bar.wait()) return;
        chunk_census<W, OT>(g, G, bid, nblk);
      }
    }
    if (!bar.wait([&](int lane) { level_end<W>(g, lane); })) return;
  }
}

// Seeds the sources of every slot (one block).  Level 0 starts afterwards.
template <int W, typename OT>
__global__ void k_seed(GroupDev g, DevGraph G) {
  LevelCtl* ctl = g.ctl;
  const int lane = threadIdx.x & 31;
  uint64_t uni[W];
#pragma unroll
  for (int i = 0; i < W; ++i) uni[i] = 0;
  for (int base = threadIdx.x & ~31; base < g.Qg; base += blockDim.x) {
    const int q = base + lane;
    bool app = false;
    int32_t src = 0;
    uint64_t deg = 0;
    if (q < g.Qg) {
      const SlotDev s = g.slots[q];
      if (s.kind != 2 && s.source >= 0) {  // WCC slots are not traversal slots
        src = s.source;
        const uint64_t bit = 1ULL << (q & 63);
        if (s.kind != 1) atomic_or64(g.visited + static_cast<size_t>(src) * W + (q >> 6), bit);
        atomic_or64(g.fbuf0 + static_cast<size_t>(src) * W + (q >> 6), bit);
        if (g.values != nullptr) g.values[static_cast<size_t>(src) * g.Qg + q] = 0u;
        uni[q >> 6] |= bit;
        app = atomicMax(g.stamp + src, 0) < 0;
        deg = degree_of<OT>(G.row, src);
      }
    }
    warp_append(app, src, deg, g.list0, &ctl->count[0], &ctl->edges[0], lane);
  }
  flush_union<W>(uni, ctl->active[0], lane);
  __threadfence();
  __syncthreads();
  if (threadIdx.x < 32) {
    compute_expand<W>(ctl, g.slots, g.Qg, 0, lane);
    const int32_t dir = decide_dir(ctl, ctl->count[0], ctl->edges[0], any_bits<W>(ctl->bfs_bits));
    // the sources' level: every slot starts with the group's direction
    split_sssp_slots<W>(ctl, decide_sdir<W>(ctl, ctl->count[0], ctl->edges[0]), lane);
    if (lane == 0) {
      ctl->dir = dir;
      if (ctl->count[0] == 0) ctl->done = 1;
    }
  }
}

// --------------------------------------------------------------- output
// The buffers a group starts from, each filled with one 32-bit word, in one
// launch (a traversal of a small graph spent more time in seven memsets than
// in a level).
struct FillSpan {
  uint32_t* p;    // 16-byte aligned
  int64_t words;
  uint32_t x;
};
struct FillList {
  FillSpan span[9];
  int n = 0;
  void add(void* p, size_t bytes, uint32_t x) {
    if (bytes == 0) return;
    span[n].p = static_cast<uint32_t*>(p);
    span[n].words = static_cast<int64_t>(bytes / 4);
    span[n++].x = x;
  }
};

static __global__ void __launch_bounds__(kBlock) k_fill_spans(FillList f) {
  const int64_t t0 = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int i = 0; i < f.n; ++i) {
    const FillSpan s = f.span[i];
    const uint4 x = make_uint4(s.x, s.x, s.x, s.x);
    const int64_t vecs = s.words / 4;
    for (int64_t k = t0; k < vecs; k += stride) reinterpret_cast<uint4*>(s.p)[k] = x;
    if (t0 < s.words - 4 * vecs) s.p[4 * vecs + t0] = s.x;
  }
}

// Fills the working values with each slot's "unreached" marker, or with
// `uniform` everywhere when it is nonzero (the serving layout, where a slot
// changes kind between requests).  Warp per vertex row, lanes over slots.
static __global__ void k_fill_values(uint32_t* values, const SlotDev* slots, int Qg,
                                     int64_t V, uint32_t f32_inf_for_sssp, uint32_t uniform) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t v = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; v < V;
       v += warps) {
    uint32_t* row = values + static_cast<size_t>(v) * Qg;
    for (int q = lane; q < Qg; q += 32) {
      uint32_t x = uniform;
      if (!uniform) {
        const int kind = slots[q].kind;
        x = kind == 1 ? f32_inf_for_sssp : (kind == 2 ? 0u : 0x7fffffffu);
      }
      row[q] = x;
    }
  }
}

// Depth planes -> int32 depths (INT32_MAX where the visited bit is clear).
// Vertex-major output: warp per vertex, lanes over queries (coalesced row
// writes).  Query-major output: blockIdx.y walks queries, threads walk
// vertices (coalesced column writes).
template <int W>
__device__ __forceinline__ uint32_t plane_depth(const uint64_t* visited, const uint64_t* planes,
                                                int K, int64_t V, int64_t v, int q) {
  const size_t word = static_cast<size_t>(v) * W + (q >> 6);
  const uint64_t bit = 1ULL << (q & 63);
  if (!(visited[word] & bit)) return 0x7fffffffu;
  uint32_t d = 0;
  for (int b = 0; b < K; ++b)
    if (planes[static_cast<size_t>(b) * V * W + word] & bit) d |= 1u << b;
  return d;
}

// Bits 0 .. 3 of x to the lowest bits of four bytes (the shifted copies of the
// nibble do not overlap, so the product carries nothing).
__device__ __forceinline__ uint32_t spread_nibble(uint32_t x) {
  return ((x & 0xfu) * 0x00204081u) & 0x01010101u;
}

template <int W>
__global__ void k_materialize_planes(const uint64_t* visited, const uint64_t* planes,
                                     int K, int64_t V, int Qg, OutMap om, int query_major) {
  if (query_major) {
    for (int q = blockIdx.y; q < Qg; q += gridDim.y) {
      uint32_t* col = om.out + om.col(q) * om.sq;
      for (int64_t v = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; v < V;
           v += static_cast<int64_t>(gridDim.x) * blockDim.x)
        col[v * om.sv] = plane_depth<W>(visited, planes, K, V, v, q);
    }
    return;
  }
  if (blockIdx.y != 0) return;
  // vertex-major: each lane owns 4 consecutive queries of a 128-query block, so
  // a warp's store is 512 contiguous bytes; the depths are put together a byte
  // per query (bit by bit the kernel was bound by its instructions: 0.34 ms for
  // 1 GB against 0.17 ms at the copy rate)
  const int lane = threadIdx.x & 31;
  const int64_t warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  const bool vec = om.qmap == nullptr && (om.sv % 4 == 0) && om.sq == 1 && (om.q0 % 4 == 0) &&
                   (reinterpret_cast<uintptr_t>(om.out) & 15) == 0;
  const uint32_t* vis32 = reinterpret_cast<const uint32_t*>(visited);
  const uint32_t* planes32 = reinterpret_cast<const uint32_t*>(planes);
  const size_t plane = static_cast<size_t>(V) * W * 2;  // 32-bit words per plane
  for (int64_t v = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; v < V;
       v += warps) {
    uint32_t* row = om.out + v * om.sv;
    for (int q0 = 4 * lane; q0 < Qg; q0 += 128) {
      const size_t word = static_cast<size_t>(v) * (2 * W) + (q0 >> 5);
      const int sh = q0 & 31;
      // the first 4 planes are loaded together with the visited word
      const uint32_t vis = vis32[word] >> sh;
      uint32_t pw[4];
#pragma unroll
      for (int b = 0; b < 4; ++b) pw[b] = b < K ? planes32[b * plane + word] : 0u;
      uint32_t bytes = 0;  // depth bits 0 .. 7, a byte per query
#pragma unroll
      for (int b = 0; b < 4; ++b) bytes |= spread_nibble(pw[b] >> sh) << b;
      for (int b = 4; b < K && b < 8; ++b) bytes |= spread_nibble(planes32[b * plane + word] >> sh) << b;
      uint32_t d[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) d[j] = (bytes >> (8 * j)) & 0xffu;
      for (int b = 8; b < K; ++b) {
        const uint32_t pl = planes32[b * plane + word] >> sh;
#pragma unroll
        for (int j = 0; j < 4; ++j) d[j] |= ((pl >> j) & 1u) << b;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (!((vis >> j) & 1u)) d[j] = 0x7fffffffu;
      if (vec && q0 + 4 <= Qg) {
        *reinterpret_cast<uint4*>(row + om.col(q0)) = make_uint4(d[0], d[1], d[2], d[3]);
      } else {
        for (int j = 0; j < 4 && q0 + j < Qg; ++j) row[om.col(q0 + j) * om.sq] = d[j];
      }
    }
  }
}

// Working values (rows of Qg slots) of slots 0 .. n-1 -> output mapping (skips
// WCC slots); same mappings.
static __global__ void k_copy_values(const uint32_t* values, const SlotDev* slots, int64_t V,
                                     int n, int Qg, OutMap om, int query_major) {
  if (query_major) {
    for (int q = blockIdx.y; q < n; q += gridDim.y) {
      if (slots[q].kind == 2) continue;
      uint32_t* col = om.out + om.col(q) * om.sq;
      for (int64_t v = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; v < V;
           v += static_cast<int64_t>(gridDim.x) * blockDim.x)
        col[v * om.sv] = values[static_cast<size_t>(v) * Qg + q];
    }
    return;
  }
  if (blockIdx.y != 0) return;
  const int lane = threadIdx.x & 31;
  const int64_t warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t v = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; v < V;
       v += warps) {
    const uint32_t* src = values + static_cast<size_t>(v) * Qg;
    uint32_t* row = om.out + v * om.sv;
    for (int q = lane; q < n; q += 32)
      if (slots[q].kind != 2) row[om.col(q) * om.sq] = src[q];
  }
}

}  // namespace dev
}  // namespace cgp
