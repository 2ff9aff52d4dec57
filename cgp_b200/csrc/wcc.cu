// Weakly connected components by min-label hooking (union-find).
//
// The reference runs WCC as label propagation inside the frontier loop
// (init_wcc_all_vertices_kernel, hybrid_engine.hxx:95-123, min-reduce push),
// which needs O(diameter) levels.  Its fixpoint is the minimum vertex id of
// each component (cpu_wcc, puercgp/examples/mtx_loader.hxx:328-356).  Here the
// same labels come from one union-find pass: roots are always linked under
// the smaller root, so every root is its component's minimum id, followed by
// a pointer-jumping pass that writes label[v] = root(v).
#include "engine.h"

namespace cgp {
namespace {

using namespace dev;

__global__ void k_uf_self(int32_t* parent, int64_t V) {
  for (int64_t v = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; v < V;
       v += static_cast<int64_t>(gridDim.x) * blockDim.x)
    parent[v] = static_cast<int32_t>(v);
}

// Every vertex starts below its first neighbour if that has the smaller id (a
// forest: parents are smaller), else as its own root: the first link of each
// vertex costs no atomic.
template <typename OT>
__global__ void k_uf_init(const void* row, const int32_t* col, int32_t* parent, int64_t V) {
  for (int64_t v = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; v < V;
       v += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t beg = row_at<OT>(row, v);
    int32_t p = static_cast<int32_t>(v);
    if (row_at<OT>(row, v + 1) > beg) p = min(p, col[beg]);
    parent[v] = p;
  }
}

// Points every vertex at its root.  All vertices jump at once, each past what
// the others have shortened already, so long chains take a logarithmic number
// of steps.  Runs alone (no links are made meanwhile).
__global__ void k_uf_compress(int32_t* parent, int64_t V) {
  volatile int32_t* p = parent;
  for (int64_t v = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; v < V;
       v += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int32_t cur = p[v];
    for (;;) {
      const int32_t next = p[cur];
      if (next == cur) break;
      p[v] = next;
      cur = next;
    }
  }
}

// Root of x; shortens the path on the way (parent[x] < x for non-roots, so
// racing shortcuts only ever point further up the same tree).
__device__ __forceinline__ int32_t uf_find(int32_t* parent, int32_t x) {
  volatile int32_t* p = parent;
  int32_t cur = p[x];
  if (cur == x) return x;
  int32_t prev = x;
  for (;;) {
    const int32_t next = p[cur];
    if (next == cur) break;
    p[prev] = next;
    prev = cur;
    cur = next;
  }
  return cur;
}

// Joins the sets of a and b, linking the larger root under the smaller.
__device__ __forceinline__ void uf_union(int32_t* parent, int32_t a, int32_t b) {
  int32_t ra = uf_find(parent, a);
  int32_t rb = uf_find(parent, b);
  while (ra != rb) {
    if (ra < rb) {
      const int32_t t = ra;
      ra = rb;
      rb = t;
    }
    // ra > rb: try to hang ra below rb
    const int32_t old = atomicCAS(parent + ra, ra, rb);
    if (old == ra) return;
    ra = uf_find(parent, old);
    rb = uf_find(parent, rb);
  }
}

// Every CSR entry u->v joins u and v.  On a symmetric CSR each undirected
// edge is visited once (v < u).  Warp per tile of 32 vertices; vertices with
// more than 32 entries are walked by the whole warp.
template <typename OT>
__global__ void __launch_bounds__(kBlock) k_uf_hook(const void* row, const int32_t* col,
                                                    int32_t* parent, int64_t V, int symmetric) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t tile = gw; tile * 32 < V; tile += nw) {
    const int64_t u = tile * 32 + lane;
    int64_t beg = 0, end = 0;
    if (u < V) {
      beg = row_at<OT>(row, u);
      end = row_at<OT>(row, u + 1);
    }
    if (end - beg <= 32) {
      for (int64_t e = beg; e < end; ++e) {
        const int32_t v = col[e];
        if (!symmetric || v < u) uf_union(parent, static_cast<int32_t>(u), v);
      }
    }
    unsigned big = __ballot_sync(kFull, end - beg > 32);
    while (big) {
      const int src = __ffs(big) - 1;
      big &= big - 1;
      const int64_t bu = __shfl_sync(kFull, u, src);
      const int64_t bb = __shfl_sync(kFull, beg, src);
      const int64_t be = __shfl_sync(kFull, end, src);
      for (int64_t e = bb + lane; e < be; e += 32) {
        const int32_t v = col[e];
        if (!symmetric || v < bu) uf_union(parent, static_cast<int32_t>(bu), v);
      }
    }
  }
}

// Joins every step-th vertex with its second neighbour.  A first pass over few
// vertices and a compression come before the pass over all: without them all
// vertices at once meet at a few roots.  With and without, the whole of WCC: R-MAT
// 15, 18 and 20 67 against 140, 130 against 800 and 240 against 625 us, a directed
// graph of 2.4M entries 140 against 810; 8 copies of R-MAT 14 196 against 285.
// Regular graphs pay the two launches for nothing: a 26-neighbour stencil 71
// against 62, a band of 8 neighbours 73 against 63.
template <typename OT>
__global__ void k_uf_second(const void* row, const int32_t* col, int32_t* parent, int64_t V,
                            int64_t step) {
  for (int64_t v = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) * step; v < V;
       v += static_cast<int64_t>(gridDim.x) * blockDim.x * step) {
    const int64_t beg = row_at<OT>(row, v);
    if (row_at<OT>(row, v + 1) > beg + 1) uf_union(parent, static_cast<int32_t>(v), col[beg + 1]);
  }
}

// The root most of kSamples vertices spread over the graph have (one block):
// in most graphs that of the component two links per vertex have already
// gathered the bulk of.
constexpr int kSamples = 256;

__global__ void k_uf_sample(const int32_t* parent, int64_t V, int32_t* most) {
  __shared__ int32_t s_root[kSamples];
  __shared__ int s_best;
  const int t = threadIdx.x;
  // odd multiplier: samples of a power-of-two id space are spread evenly
  const int64_t v = static_cast<int64_t>((static_cast<uint64_t>(t) * 2654435761ULL) % static_cast<uint64_t>(V));
  s_root[t] = parent[v];
  if (t == 0) s_best = 0;
  __syncthreads();
  int c = 0;
  for (int i = 0; i < kSamples; ++i) c += s_root[i] == s_root[t] ? 1 : 0;
  atomicMax(&s_best, (c << 8) | (kSamples - 1 - t));
  __syncthreads();
  if (t == kSamples - 1 - (s_best & 255)) *most = s_root[t];
}

// Joins u and v unless v already points at `root`, an ancestor of u; `root` is u's
// root afterwards.
__device__ __forceinline__ void uf_join(int32_t* parent, int32_t u, int32_t v, int32_t& root) {
  if (static_cast<volatile int32_t*>(parent)[v] == root) return;
  uf_union(parent, u, v);
  root = uf_find(parent, u);
}

// The entries of the vertices outside the sampled component: each joins its
// endpoints.  An entry between it and another component is found from the
// other end, on a directed graph through the transpose (second call).  The
// skipped vertices hold almost all entries of a small-world graph, so the pass
// reads the offsets, a root per vertex and few lists.  Where many vertices are
// left (no component holds most), most of their entries lead to vertices that
// already point at the same root: one load each, with the root at hand (10,000
// cliques of 33: the pass over all entries once per edge 99 us in all, with two
// finds per entry here 118, with this test 96).  Warp per tile of 32 vertices;
// vertices with more than 32 entries are walked by the whole warp.
template <typename OT>
__global__ void __launch_bounds__(kBlock) k_uf_rest(const void* row, const int32_t* col,
                                                    int32_t* parent, int64_t V,
                                                    const int32_t* most) {
  const int32_t skip = *most;
  const int lane = threadIdx.x & 31;
  const int64_t gw = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t tile = gw; tile * 32 < V; tile += nw) {
    const int64_t u = tile * 32 + lane;
    int64_t beg = 0, end = 0;
    int32_t root = skip;  // an ancestor of u (its root, as far as this lane knows)
    if (u < V) root = static_cast<volatile int32_t*>(parent)[u];
    if (root != skip) {
      beg = row_at<OT>(row, u);
      end = row_at<OT>(row, u + 1);
    }
    if (end - beg <= 32) {
      for (int64_t e = beg; e < end; ++e) uf_join(parent, static_cast<int32_t>(u), col[e], root);
    }
    unsigned big = __ballot_sync(kFull, end - beg > 32);
    while (big) {
      const int src = __ffs(big) - 1;
      big &= big - 1;
      const int64_t bu = __shfl_sync(kFull, u, src);
      const int64_t bb = __shfl_sync(kFull, beg, src);
      const int64_t be = __shfl_sync(kFull, end, src);
      int32_t br = __shfl_sync(kFull, root, src);
      for (int64_t e = bb + lane; e < be; e += 32) uf_join(parent, static_cast<int32_t>(bu), col[e], br);
    }
  }
}

// Root of x without shortening the path.  The label pass writes roots into
// the parent array itself, so it must not also store shortcuts: a late
// shortcut store to parent[y] could replace y's finished label (its root)
// with an intermediate ancestor.
__device__ __forceinline__ int32_t uf_root(const int32_t* parent, int32_t x) {
  const volatile int32_t* p = parent;
  int32_t cur = x;
  for (;;) {
    const int32_t next = p[cur];
    if (next == cur) return cur;
    cur = next;
  }
}

// labels[v] = root(v), in place over the parent array: each entry is written
// once, by its own thread, with an ancestor of v, so concurrent readers still
// follow valid parent chains.
__global__ void k_uf_labels(int32_t* parent, int64_t V) {
  for (int64_t v = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; v < V;
       v += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int32_t r = uf_root(parent, static_cast<int32_t>(v));
    reinterpret_cast<volatile int32_t*>(parent)[v] = r;
  }
}

__global__ void k_broadcast(const uint32_t* labels, int64_t V, OutMap om, int colidx) {
  for (int64_t v = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; v < V;
       v += static_cast<int64_t>(gridDim.x) * blockDim.x)
    om.out[v * om.sv + static_cast<int64_t>(colidx) * om.sq] = labels[v];
}

}  // namespace

namespace {

// Entries per vertex from which neighbours are sampled.  Below, two links per
// vertex are a good part of all entries and the passes between them cost more
// than they save: on 1100 x 1300 grids (3.6 entries) sampling took 264 to 304 us
// for most and 536 and 1040 us for two of ten, all entries at once 356 to 424;
// on R-MAT 18 (29 entries) 130 to 240 us against 890 to 2700.
constexpr int64_t kSampleDegree = 8;

template <typename OT>
int link_all(GraphImpl* g, int32_t* parent, int32_t* most, int blocks, cudaStream_t s) {
  const int64_t V = g->V;
  const int32_t* col = g->col.as<int32_t>();
  if (g->E < kSampleDegree * V) {
    k_uf_self<<<blocks, kBlock, 0, s>>>(parent, V);
    k_uf_hook<OT><<<blocks, kBlock, 0, s>>>(g->row.p, col, parent, V, g->symmetric ? 1 : 0);
    return 2;
  }
  k_uf_init<OT><<<blocks, kBlock, 0, s>>>(g->row.p, col, parent, V);
  k_uf_compress<<<blocks, kBlock, 0, s>>>(parent, V);
  k_uf_second<OT><<<blocks, kBlock, 0, s>>>(g->row.p, col, parent, V, 61);
  k_uf_compress<<<blocks, kBlock, 0, s>>>(parent, V);
  k_uf_second<OT><<<blocks, kBlock, 0, s>>>(g->row.p, col, parent, V, 1);
  k_uf_compress<<<blocks, kBlock, 0, s>>>(parent, V);
  k_uf_sample<<<1, kSamples, 0, s>>>(parent, V, most);
  k_uf_rest<OT><<<blocks, kBlock, 0, s>>>(g->row.p, col, parent, V, most);
  if (g->symmetric) return 8;
  k_uf_rest<OT><<<blocks, kBlock, 0, s>>>(g->trow.p, g->tcol.as<int32_t>(), parent, V, most);
  return 9;
}

}  // namespace

// Union-find with neighbour sampling (Sutton, Ben-Nun, Barak: Optimizing
// parallel graph connectivity computation via subgraph sampling, 2018): two
// links per vertex, then only the vertices outside the component most of them
// have ended up in visit their lists; graphs of low degree link every entry.
// Visiting every entry took 0.86 ms on R-MAT 17, where the finds and links of
// 1.9M edges meet at a few roots; sampling takes 0.1.
int wcc_labels(GraphImpl* g, uint32_t* labels, cudaStream_t s) {
  // parent array lives in `labels` itself (int32 view), the sampled root
  // behind it; the final pass rewrites every entry with its root.
  int32_t* parent = reinterpret_cast<int32_t*>(labels);
  const int blocks = g->num_sms * 8;
  const int n = g->offset_bytes == 8 ? link_all<int64_t>(g, parent, parent + g->V, blocks, s)
                                     : link_all<int32_t>(g, parent, parent + g->V, blocks, s);
  k_uf_labels<<<blocks, kBlock, 0, s>>>(parent, g->V);
  ck(cudaGetLastError(), "wcc");
  return n + 1;
}

void broadcast_labels(const uint32_t* labels, int64_t V, OutMap om, int col, cudaStream_t s) {
  k_broadcast<<<256, kBlock, 0, s>>>(labels, V, om, col);
  ck(cudaGetLastError(), "wcc broadcast");
}

}  // namespace cgp
