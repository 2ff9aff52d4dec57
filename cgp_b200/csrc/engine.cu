// Multi-query traversal engine: graph upload, cached device workspaces, the
// device-driven level loop (replayed as CUDA graphs) and output writing.
//
// Replaces the host loops of frontier_engine::run
// (puercgp/include/puercgp/engine/frontier_engine.hxx:2203-3139) and
// hybrid_frontier_engine::run (hybrid_engine.hxx:793-1141).  The reference
// copies one or two counters to the host and synchronises after every level;
// here the direction decision, counter resets and convergence test run in one
// warp at the end of each level, and the host only looks at the control block
// once per chunk of levels or once per launch of the fused loop.
#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstring>
#include <numeric>

#include "engine.h"
#include "kernels.cuh"
#include "levels.h"

namespace cgp {

using namespace dev;

// --------------------------------------------------- traversals per device
OnDevice::Load OnDevice::loads_[OnDevice::kDevices];

static int64_t steady_ns() {
  return std::chrono::duration_cast<std::chrono::nanoseconds>(
             std::chrono::steady_clock::now().time_since_epoch()).count();
}

OnDevice::OnDevice(int device) : load_(loads_[device % kDevices]) {
  if (++load_.running > 1) load_.shared_until = steady_ns() + kSharedNs;
}

int OnDevice::callers(int device) {
  const Load& l = loads_[device % kDevices];
  const int n = l.running;
  return n < 2 && steady_ns() < l.shared_until ? 2 : n;
}

// ------------------------------------------------------------- buffers
namespace {
// Fault-injection hook for tests: >= 0 counts down the device allocations
// still allowed before one fails as if the device were out of memory; -1 off.
std::atomic<int64_t> g_fail_alloc_countdown{-1};
std::atomic<int32_t> g_grid_failure{CGP_GRID_OK};
// A grid barrier's wait, on a device that runs every block of the launch; and
// where a block is missing on purpose.
constexpr unsigned long long kBarrierNs = 20ULL * 1000 * 1000 * 1000;
constexpr unsigned long long kInjectedBarrierNs = 50ULL * 1000 * 1000;

bool injected_alloc_failure() {
  int64_t c = g_fail_alloc_countdown.load();
  while (c >= 0) {
    if (g_fail_alloc_countdown.compare_exchange_weak(c, c - 1)) return c == 0;
  }
  return false;
}
}  // namespace

DevBuf::~DevBuf() {
  if (p) cudaFree(p);
}

bool DevBuf::ensure(size_t need) {
  if (need <= bytes && p) return false;
  if (p) cudaFree(p);
  p = nullptr;
  bytes = 0;
  size_t alloc = std::max<size_t>(need, 256);
  if (injected_alloc_failure())
    throw ApiError{CGP_ERR_OOM, "cudaMalloc of " + std::to_string(alloc) +
                                    " bytes failed (injected by cgp_debug_fail_allocations)"};
  cudaError_t e = cudaMalloc(&p, alloc);
  if (e != cudaSuccess) {
    cudaGetLastError();
    p = nullptr;
    throw ApiError{CGP_ERR_OOM, "cudaMalloc of " + std::to_string(alloc) + " bytes failed"};
  }
  bytes = alloc;
  return true;
}

bool DevBuf::offer(size_t need, bool* moved) {
  if (need <= bytes && p) return true;
  size_t free_b = 0, total_b = 0;
  if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess || need > free_b / 8) {
    cudaGetLastError();
    return false;
  }
  if (p) cudaFree(p);
  p = nullptr;
  bytes = 0;
  *moved = true;  // the old block is gone either way
  if (cudaMalloc(&p, need) != cudaSuccess) {
    cudaGetLastError();
    p = nullptr;
    return false;
  }
  bytes = need;
  return true;
}

Workspace::Workspace(int dev) : device(dev) {
  ck(cudaHostAlloc(reinterpret_cast<void**>(&hctl), 2 * sizeof(LevelCtl), cudaHostAllocDefault),
     "cudaHostAlloc(ctl)");
  const size_t start_bytes = kSlotsOffset + kMaxWords * 64 * sizeof(SlotDev);
  ck(cudaHostAlloc(reinterpret_cast<void**>(&hstart), start_bytes, cudaHostAllocDefault),
     "cudaHostAlloc(start)");
  ck(cudaEventCreateWithFlags(&uploaded, cudaEventDisableTiming), "cudaEventCreate");
  ck(cudaEventCreate(&t0), "cudaEventCreate");
  ck(cudaEventCreate(&t1), "cudaEventCreate");
  ck(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking), "cudaStreamCreate");
  ck(cudaStreamCreateWithFlags(&capture, cudaStreamNonBlocking), "cudaStreamCreate");
  ck(cudaStreamCreateWithFlags(&copy, cudaStreamNonBlocking), "cudaStreamCreate");
  ck(cudaEventCreateWithFlags(&out_ready, cudaEventDisableTiming), "cudaEventCreate");
  for (auto& e : ev) ck(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "cudaEventCreate");
  ctl.ensure(start_bytes);
}

void Workspace::clear_graphs() {
  for (auto& kv : graphs) cudaGraphExecDestroy(kv.second.exec);
  graphs.clear();
}

Workspace::~Workspace() {
  clear_graphs();
  if (hctl) cudaFreeHost(hctl);
  if (hstart) cudaFreeHost(hstart);
  if (uploaded) cudaEventDestroy(uploaded);
  if (t0) cudaEventDestroy(t0);
  if (t1) cudaEventDestroy(t1);
  if (stream) cudaStreamDestroy(stream);
  if (capture) cudaStreamDestroy(capture);
  if (copy) cudaStreamDestroy(copy);
  if (out_ready) cudaEventDestroy(out_ready);
  for (auto& e : ev)
    if (e) cudaEventDestroy(e);
}

KernelTimer::KernelTimer() {
  for (auto& e : ev) ck(cudaEventCreate(&e), "cudaEventCreate");
}

KernelTimer::~KernelTimer() {
  for (auto& e : ev)
    if (e) cudaEventDestroy(e);
}

void KernelTimer::mark(int c, cudaStream_t s) {
  if (n == kMaxMarks) flush();
  ck(cudaEventRecord(ev[n], s), "timer event");
  cls[n] = c;
  ++n;
  if (c >= 0) ++count[c];
}

void KernelTimer::flush() {
  if (n == 0) return;
  ck(cudaEventSynchronize(ev[n - 1]), "timer sync");
  for (int i = 0; i + 1 < n; ++i) {
    if (cls[i] < 0) continue;
    float t = 0;
    ck(cudaEventElapsedTime(&t, ev[i], ev[i + 1]), "timer elapsed");
    ms[cls[i]] += t;
  }
  // keep the last mark open across flushes
  if (cls[n - 1] >= 0) {
    cudaEvent_t last = ev[n - 1];
    int lc = cls[n - 1];
    ev[n - 1] = ev[0];
    ev[0] = last;
    cls[0] = lc;
    n = 1;
  } else {
    n = 0;
  }
}

// --------------------------------------------------------------- graph
DevGraph GraphImpl::dev_graph(int64_t h, bool light_items) {
  const HeavyPair& hp = heavy_for(h);
  DevGraph d;
  d.row = row.p;
  d.col = col.as<int32_t>();
  d.w = w.p;
  d.prow = pull_row();
  d.pcol = pull_col();
  d.pw = pull_w();
  d.V = V;
  d.E = E;
  d.heavy = hp.heavy.vertices.as<int32_t>();
  d.n_heavy = hp.heavy.n;
  d.heavy_chunks = hp.heavy.chunks;
  d.pheavy = hp.pheavy.vertices.as<int32_t>();
  d.pheavy_ch = hp.pheavy.chunk_h.as<int32_t>();
  d.pheavy_cb = hp.pheavy.chunk_beg.as<int64_t>();
  d.pheavy_ce = hp.pheavy.chunk_end.as<int64_t>();
  d.n_pheavy = hp.pheavy.n;
  d.pheavy_chunks = hp.pheavy.chunks;
  d.plight = hp.plight.vertices.as<int32_t>();
  d.plight_chunk_start = hp.plight.chunk_start.as<int32_t>();
  d.plight_beg = hp.plight.beg.as<int64_t>();
  d.n_plight = hp.plight.n;
  d.n_plight_chunks = hp.plight.chunks;
  d.n_pmid = hp.plight.n_mid;
  d.mid_degree = hp.plight.mid_degree;
  d.gitem_start = hp.plight.item_start.as<int32_t>();
  d.gitem_pre = hp.plight.item_pre.as<int32_t>();
  d.n_gitems = hp.plight.items;
  const HeavyTable& sh = light_items ? hp.gheavy : hp.pheavy;
  d.sheavy = sh.vertices.as<int32_t>();
  d.sheavy_ch = sh.chunk_h.as<int32_t>();
  d.sheavy_cb = sh.chunk_beg.as<int64_t>();
  d.sheavy_ce = sh.chunk_end.as<int64_t>();
  d.n_sheavy = sh.n;
  d.sheavy_chunks = sh.chunks;
  d.heavy_degree = h;
  d.hub = hub;
  return d;
}

namespace {

// Host copies kept for table building.
struct HostCsr {
  std::vector<int64_t> row, trow;
};
std::mutex g_host_mu;
std::map<const GraphImpl*, HostCsr> g_host;

void build_heavy(const std::vector<int64_t>& row, int64_t V, int64_t h, HeavyTable& t) {
  std::vector<int32_t> vs;
  std::vector<int64_t> cs{0};
  for (int64_t v = 0; v < V; ++v) {
    int64_t d = row[v + 1] - row[v];
    if (d > h) {
      vs.push_back(static_cast<int32_t>(v));
      cs.push_back(cs.back() + (d + kHeavyChunk - 1) / kHeavyChunk);
    }
  }
  t.n = static_cast<int32_t>(vs.size());
  t.chunks = cs.back();
  // per chunk: its vertex's table index and its edge range, so that a CTA
  // finds its work with three independent loads instead of a binary search
  std::vector<int32_t> ch(static_cast<size_t>(t.chunks));
  std::vector<int64_t> cb(static_cast<size_t>(t.chunks)), ce(static_cast<size_t>(t.chunks));
  for (size_t i = 0; i < vs.size(); ++i) {
    const int64_t b = row[vs[i]], e = row[vs[i] + 1];
    for (int64_t c = cs[i]; c < cs[i + 1]; ++c) {
      ch[c] = static_cast<int32_t>(i);
      cb[c] = b + (c - cs[i]) * kHeavyChunk;
      ce[c] = std::min(e, cb[c] + kHeavyChunk);
    }
  }
  t.vertices.ensure(std::max<size_t>(vs.size(), 1) * sizeof(int32_t));
  t.chunk_h.ensure(std::max<size_t>(ch.size(), 1) * sizeof(int32_t));
  t.chunk_beg.ensure(std::max<size_t>(cb.size(), 1) * sizeof(int64_t));
  t.chunk_end.ensure(std::max<size_t>(ce.size(), 1) * sizeof(int64_t));
  if (!vs.empty()) {
    ck(cudaMemcpy(t.vertices.p, vs.data(), vs.size() * sizeof(int32_t), cudaMemcpyHostToDevice),
       "upload heavy");
    ck(cudaMemcpy(t.chunk_h.p, ch.data(), ch.size() * sizeof(int32_t), cudaMemcpyHostToDevice),
       "upload heavy chunk vertices");
    ck(cudaMemcpy(t.chunk_beg.p, cb.data(), cb.size() * sizeof(int64_t), cudaMemcpyHostToDevice),
       "upload heavy chunk starts");
    ck(cudaMemcpy(t.chunk_end.p, ce.data(), ce.size() * sizeof(int64_t), cudaMemcpyHostToDevice),
       "upload heavy chunk ends");
  }
}

void build_light_chunks(const std::vector<int64_t>& row, int64_t V, int64_t h, int sms,
                        LightChunks& t) {
  // light vertices by in-degree, largest first (ties by id): CTAs take chunks
  // roughly in this order, so within a gather level the better-connected
  // vertices settle first and the rest read their lowered distances
  // (a counting sort by in-degree)
  std::vector<int64_t> at(static_cast<size_t>(h) + 2, 0);
  for (int64_t v = 0; v < V; ++v) {
    const int64_t d = row[v + 1] - row[v];
    if (d > 0 && d <= h) ++at[h - d + 1];
  }
  for (int64_t i = 0; i <= h; ++i) at[i + 1] += at[i];
  std::vector<int32_t> order(static_cast<size_t>(at[h + 1]));
  for (int64_t v = 0; v < V; ++v) {
    const int64_t d = row[v + 1] - row[v];
    if (d > 0 && d <= h) order[at[h - d]++] = static_cast<int32_t>(v);
  }
  std::vector<int32_t> vs;
  std::vector<int32_t> cs{0};
  int cur_v = 0;
  int64_t cur_e = 0;
  for (const int32_t v : order) {
    const int64_t d = row[v + 1] - row[v];
    if (cur_v > 0 && (cur_v == dev::kLightChunkVerts || cur_e + d > dev::kLightChunkEdges)) {
      cs.push_back(static_cast<int32_t>(vs.size()));
      cur_v = 0;
      cur_e = 0;
    }
    vs.push_back(static_cast<int32_t>(v));
    ++cur_v;
    cur_e += d;
  }
  if (cur_v > 0) cs.push_back(static_cast<int32_t>(vs.size()));
  t.n = static_cast<int32_t>(vs.size());
  t.chunks = static_cast<int32_t>(cs.size()) - 1;
  // BFS pull: a warp per vertex above mid_degree in-edges, a lane below.  Where
  // the warps of the GPU hold every vertex of more than 8 at once, those get
  // one each: a lane walks 32 in-edges in 8 dependent steps, a warp in one.
  const int64_t warps = 24 * static_cast<int64_t>(sms);
  auto above = [&](int64_t d) {
    int32_t n = 0;
    while (n < t.n && row[vs[n] + 1] - row[vs[n]] > d) ++n;
    return n;
  };
  t.n_mid = above(8);
  t.mid_degree = 8;
  if (t.n_mid > 2 * warps) {
    t.n_mid = above(32);
    t.mid_degree = 32;
  }
  // per entry: its first in-edge; and the row gather's items with their
  // in-edge prefixes, so that an item's header is three independent loads
  std::vector<int64_t> beg(vs.size());
  std::vector<int32_t> pre(vs.size()), is;
  int32_t run = 0, acc = 0;
  // two items for each warp of the GPU at least: a 96 x 97 grid in items of 32
  // vertices is 290 warps' serial work
  int64_t edges = 0;
  for (const int32_t v : vs) edges += std::min<int64_t>(row[v + 1] - row[v], dev::kGatherHeavy);
  const int32_t most_v = static_cast<int32_t>(
      std::min<int64_t>(32, std::max<int64_t>(1, static_cast<int64_t>(vs.size()) / (2 * warps))));
  const int64_t most_e =
      std::min<int64_t>(dev::kGatherHeavy, std::max<int64_t>(32, edges / (2 * warps)));
  for (size_t i = 0; i < vs.size(); ++i) {
    beg[i] = row[vs[i]];
    const int64_t d = row[vs[i] + 1] - row[vs[i]];
    if (d > dev::kGatherHeavy) continue;
    if (is.empty() || run == most_v || acc + d > most_e) {
      is.push_back(static_cast<int32_t>(i));
      run = 0;
      acc = 0;
    }
    ++run;
    acc += static_cast<int32_t>(d);
    pre[i] = acc;
  }
  t.items = static_cast<int32_t>(is.size());
  is.push_back(static_cast<int32_t>(vs.size()));
  t.vertices.ensure(std::max<size_t>(vs.size(), 1) * sizeof(int32_t));
  t.chunk_start.ensure(cs.size() * sizeof(int32_t));
  t.beg.ensure(std::max<size_t>(vs.size(), 1) * sizeof(int64_t));
  t.item_start.ensure(is.size() * sizeof(int32_t));
  t.item_pre.ensure(std::max<size_t>(vs.size(), 1) * sizeof(int32_t));
  if (!vs.empty()) {
    ck(cudaMemcpy(t.vertices.p, vs.data(), vs.size() * sizeof(int32_t), cudaMemcpyHostToDevice),
       "upload light vertices");
    ck(cudaMemcpy(t.beg.p, beg.data(), beg.size() * sizeof(int64_t), cudaMemcpyHostToDevice),
       "upload light offsets");
    ck(cudaMemcpy(t.item_pre.p, pre.data(), pre.size() * sizeof(int32_t), cudaMemcpyHostToDevice),
       "upload light prefixes");
  }
  ck(cudaMemcpy(t.chunk_start.p, cs.data(), cs.size() * sizeof(int32_t), cudaMemcpyHostToDevice),
     "upload light chunks");
  ck(cudaMemcpy(t.item_start.p, is.data(), is.size() * sizeof(int32_t), cudaMemcpyHostToDevice),
     "upload gather items");
}

}  // namespace

const HeavyPair& GraphImpl::heavy_for(int64_t h) {
  std::lock_guard<std::mutex> lk(heavy_mu);
  auto it = heavy_cache.find(h);
  if (it != heavy_cache.end()) return *it->second;
  auto hp = std::make_unique<HeavyPair>();
  {
    std::lock_guard<std::mutex> hl(g_host_mu);
    HostCsr& hc = g_host[this];
    build_heavy(hc.row, V, h, hp->heavy);
    build_heavy(hc.trow.empty() ? hc.row : hc.trow, V, h, hp->pheavy);
    build_heavy(hc.trow.empty() ? hc.row : hc.trow, V, std::min<int64_t>(h, dev::kGatherHeavy),
                hp->gheavy);
    build_light_chunks(hc.trow.empty() ? hc.row : hc.trow, V, h, num_sms, hp->plight);
  }
  return *heavy_cache.emplace(h, std::move(hp)).first->second;
}

std::unique_ptr<Workspace> GraphImpl::acquire() {
  std::lock_guard<std::mutex> lk(mu);
  if (!pool.empty()) {
    auto ws = std::move(pool.back());
    pool.pop_back();
    return ws;
  }
  return std::make_unique<Workspace>(device);
}

void GraphImpl::release(std::unique_ptr<Workspace> ws) {
  std::lock_guard<std::mutex> lk(mu);
  pool.push_back(std::move(ws));
}

void GraphImpl::copy_out(const std::vector<HostSegment>& segs, cudaStream_t s) {
  std::unique_ptr<HostCopier> c;
  {
    std::lock_guard<std::mutex> lk(mu);
    if (!copiers.empty()) {
      c = std::move(copiers.back());
      copiers.pop_back();
    }
  }
  if (!c) c = std::make_unique<HostCopier>(device);
  c->copy(segs, s);  // a copier that failed is dropped
  std::lock_guard<std::mutex> lk(mu);
  copiers.push_back(std::move(c));
}

cgp_status translate_exception() {
  try {
    throw;
  } catch (const ApiError& e) {
    return set_error(e.code, e.msg);
  } catch (const CudaError& e) {
    cudaError_t c = e.code;
    return set_error(c == cudaErrorMemoryAllocation ? CGP_ERR_OOM : CGP_ERR_CUDA,
                     e.where + ": " + cudaGetErrorString(c));
  } catch (const std::bad_alloc&) {
    return set_error(CGP_ERR_OOM, "host allocation failed");
  } catch (const std::exception& e) {
    return set_error(CGP_ERR_INVALID_ARG, e.what());
  } catch (...) {
    return set_error(CGP_ERR_INVALID_ARG, "unknown error");
  }
}

// -------------------------------------------------------------- groups
int choose_words(int n, int requested) {
  if (requested > 0) {
    int w = 1;
    while (w < requested) w <<= 1;
    return std::min(w, kMaxWords);
  }
  int need = std::max(1, (n + 63) / 64);
  int w = 1;
  while (w < need) w <<= 1;
  return std::min(w, kMaxWords);
}

GroupSpec make_group(const cgp_query* q, int n, int W, int depth_mode) {
  GroupSpec g;
  g.W = W;
  g.n = n;
  g.Qg = n;
  g.slots.resize(n);
  for (int i = 0; i < n; ++i) {
    g.slots[i].kind = q[i].kind;
    g.slots[i].source = q[i].source;
    g.slots[i].k = q[i].k;
    g.slots[i].base = 0;
    if (q[i].kind == CGP_KIND_SSSP) g.has_sssp = true;
    if (q[i].kind == CGP_KIND_BFS || q[i].kind == CGP_KIND_KHOP) g.has_bfs = true;
    if (q[i].kind == CGP_KIND_WCC) g.has_wcc = true;
  }
  if (depth_mode == CGP_DEPTH_PLANES && !g.has_sssp) g.depth_mode = kDepthPlanes;
  else if (depth_mode == CGP_DEPTH_DIRECT || g.has_sssp) g.depth_mode = kDepthDirect;
  else g.depth_mode = (n >= 16) ? kDepthPlanes : kDepthDirect;  // auto
  return g;
}

static constexpr int kInitialPlanes = 8;  // depth planes allocated at first
static constexpr int kStartPlanes = 4;    // ... and zeroed: depths up to 15

int64_t group_state_bytes(const GraphImpl* g, int W, int Qg, int depth_mode) {
  const int64_t V = g->V;
  int64_t b = 3 * V * W * 8 + 3 * V * 4;
  if (depth_mode == kDepthPlanes) b += static_cast<int64_t>(kInitialPlanes) * V * W * 8;
  else b += V * static_cast<int64_t>(Qg) * 4;
  return b;
}

namespace {

template <int W>
Dispatch pick_ot(int ob, int depth, int wk) {
  return ob == 8 ? pick_depth<W, int64_t>(depth, wk) : pick_depth<W, int32_t>(depth, wk);
}

Dispatch dispatch(int W, int ob, int depth, int wk) {
  switch (W) {
    case 1: return pick_ot<1>(ob, depth, wk);
    case 2: return pick_ot<2>(ob, depth, wk);
    case 4: return pick_ot<4>(ob, depth, wk);
    case 8: return pick_ot<8>(ob, depth, wk);
    default: return pick_ot<16>(ob, depth, wk);
  }
}

GroupDev group_dev(Workspace* ws, const GroupSpec& spec, bool profiles) {
  GroupDev g{};
  g.visited = ws->visited.as<uint64_t>();
  g.fbuf0 = ws->fbuf0.as<uint64_t>();
  g.fbuf1 = ws->fbuf1.as<uint64_t>();
  g.list0 = ws->list0.as<int32_t>();
  g.list1 = ws->list1.as<int32_t>();
  g.stamp = ws->stamp.as<int32_t>();
  g.planes = spec.depth_mode == kDepthPlanes ? ws->planes.as<uint64_t>() : nullptr;
  g.values = spec.depth_mode == kDepthPlanes
                 ? nullptr
                 : (spec.external_values ? spec.external_values : ws->values.as<uint32_t>());
  g.hacc = ws->hacc.as<uint64_t>();
  g.fsum = ws->fsum.as<uint64_t>();
  if (spec.bounds) {
    g.blo = ws->bounds.as<uint32_t>();
    g.bhi = g.blo + ws->bounds.bytes / 8;
  }
  g.dense_list = ws->dense.as<int32_t>();
  g.hq_vertex = ws->hq_vertex.as<int32_t>();
  g.hq_start = ws->hq_start.as<int64_t>();
  g.hq_cap = static_cast<int64_t>(ws->hq_start.bytes / sizeof(int64_t));
  g.ctl = ws->ctl.as<LevelCtl>();
  g.prof = profiles ? ws->prof.as<LevelProfile>() : nullptr;
  g.slots = ws->slots_dev();
  g.Qg = spec.Qg;
  return g;
}

constexpr int kProfileCap = 1 << 16;

// SSSP levels may gather (pull) when the pull CSR exists and the options
// allow it: always in pull mode, by frontier edges in hybrid mode.
bool sssp_gather_on(const GraphImpl* g, const cgp_options& o) {
  if (!g->can_gather() || o.traversal_mode == CGP_MODE_PUSH) return false;
  return o.traversal_mode == CGP_MODE_PULL || o.sssp_pull_edge_ratio > 0;
}

// SSSP direction per 32-slot chunk: asked for, or by default in serving
// groups (whose slots are in every phase of their traversals at once).
bool sssp_chunk_dir(const GroupSpec& spec, const cgp_options& o) {
  if (!spec.has_sssp || o.traversal_mode != CGP_MODE_HYBRID) return false;
  return o.sssp_chunk_direction > 0 || (o.sssp_chunk_direction == 0 && spec.serving);
}

// Slots per vector load of the gather kernels (GatherVec::kElem).
int row_vector(int W) { return W == 1 ? 2 : 4; }

// Rows the vectorised gather can read: whole vectors, aligned.
bool vector_rows(const GroupSpec& spec, const uint32_t* values) {
  const int elem = row_vector(spec.W);
  return values != nullptr && spec.Qg % elem == 0 &&
         reinterpret_cast<uintptr_t>(values) % (4 * elem) == 0;
}

}  // namespace

bool pad_rows(const GraphImpl* g, const Workspace* ws, GroupSpec& spec, const cgp_options& o,
              bool external) {
  const int elem = row_vector(spec.W);
  if (!spec.has_sssp || spec.n % elem == 0 || !sssp_gather_on(g, o)) return false;
  const int padded = (spec.n + elem - 1) / elem * elem;
  const size_t need = static_cast<size_t>(g->V) * padded * 4;
  if (ws->values.bytes < need) {
    size_t free_b = 0, total_b = 0;
    ck(cudaMemGetInfo(&free_b, &total_b), "cudaMemGetInfo");
    // all that group_prepare may still allocate: the group's state, and up to 32
    // bytes per vertex of lists and summaries
    const size_t state = static_cast<size_t>(group_state_bytes(g, spec.W, padded, spec.depth_mode)) +
                         static_cast<size_t>(g->V) * 32;
    if (external ? need > free_b / 4 : state > free_b) return false;
  }
  spec.Qg = padded;
  spec.slots.resize(padded, dev::SlotDev{-1, -1, 0, 0});
  return true;
}

void group_prepare(GraphImpl* g, Workspace* ws, GroupSpec& spec, const cgp_options& o,
                   cudaStream_t s) {
  const int64_t V = g->V;
  const int W = spec.W;
  const int64_t hth = heavy_threshold(o);
  const HeavyPair& hp = g->heavy_for(hth);
  bool moved = false;
  spec.depth_bits = 0;
  const size_t mask_bytes = static_cast<size_t>(V) * W * 8;
  try {
    moved |= ws->visited.ensure(mask_bytes);
    moved |= ws->fbuf0.ensure(mask_bytes);
    moved |= ws->fbuf1.ensure(mask_bytes);
    moved |= ws->list0.ensure(static_cast<size_t>(V) * 4);
    moved |= ws->list1.ensure(static_cast<size_t>(V) * 4);
    moved |= ws->stamp.ensure(static_cast<size_t>(V) * 4);
    moved |= ws->hacc.ensure(static_cast<size_t>(std::max(1, hp.pheavy.n)) * W * 8);
    moved |= ws->fsum.ensure(static_cast<size_t>(V) * 8);
    // heavy-queue capacity: every heavy vertex, and every vertex of out-degree
    // > 32 (small or skewed frontiers queue those)
    const size_t hq_cap = std::max<size_t>(std::max<int64_t>(1, hp.heavy.n), g->n_deg32);
    moved |= ws->hq_vertex.ensure(hq_cap * 4);
    moved |= ws->hq_start.ensure(hq_cap * 8);
    if (spec.has_sssp) moved |= ws->dense.ensure(static_cast<size_t>(V) * 4);
    if (spec.depth_mode == kDepthPlanes) {
      moved |= ws->planes.ensure(static_cast<size_t>(kInitialPlanes) * mask_bytes);
    } else if (spec.external_values == nullptr) {
      moved |= ws->values.ensure(static_cast<size_t>(V) * spec.Qg * 4);
    }
    if (o.profile_iterations) moved |= ws->prof.ensure(kProfileCap * sizeof(LevelProfile));
    // Bounds for the default gather kernels.  A serving group decides gather
    // or scatter per 32-slot chunk and its slots are in every phase at once.
    spec.bounds = spec.has_sssp && !spec.serving && sssp_gather_on(g, o) &&
                  !sssp_chunk_dir(spec, o) && o.light_chunks >= 0 &&
                  vector_rows(spec, spec.external_values ? spec.external_values
                                                         : ws->values.as<uint32_t>()) &&
                  ws->bounds.offer(static_cast<size_t>(V) * W * 16, &moved);
  } catch (...) {
    // a failed ensure() has already freed its old block: graphs captured with
    // the old pointers must never be replayed
    ws->generation++;
    ws->clear_graphs();
    throw;
  }
  if (moved) {
    ws->generation++;
    ws->clear_graphs();
  }
  const uint32_t sssp_inf = g->weight_kind == CGP_WEIGHT_F32 ? 0x7f800000u : 0xffffffffu;
  uint32_t* values = group_dev(ws, spec, false).values;
  // one marker for every slot: all of one kind, or the serving layout
  const bool one_kind = !(spec.has_bfs && spec.has_sssp) && !spec.has_wcc;
  uint32_t marker = spec.uniform_inf;
  if (marker == 0 && one_kind) marker = spec.has_sssp ? sssp_inf : 0x7fffffffu;
  // only 4 planes are zeroed: group_enact adds planes when a depth needs them
  const size_t planes_bytes = static_cast<size_t>(kStartPlanes) * mask_bytes;
  FillList fill;
  bool fill_late = false;
  fill.add(ws->visited.p, mask_bytes, 0);
  fill.add(ws->fbuf0.p, mask_bytes, 0);
  fill.add(ws->fbuf1.p, mask_bytes, 0);
  fill.add(ws->stamp.p, static_cast<size_t>(V) * 4, 0xffffffffu);
  fill.add(ws->hacc.p, static_cast<size_t>(std::max(1, hp.pheavy.n)) * W * 8, 0);
  fill.add(ws->fsum.p, static_cast<size_t>(V) * 8, 0);
  if (spec.depth_mode == kDepthPlanes) {
    fill.add(ws->planes.p, planes_bytes, 0);
  } else if (marker != 0 && reinterpret_cast<uintptr_t>(values) % 16 == 0) {
    fill.add(values, static_cast<size_t>(V) * spec.Qg * 4, marker);
  } else {
    fill_late = true;
  }

  // slots and control block, one upload (the last one has left the buffer)
  ck(cudaEventSynchronize(ws->uploaded), "slot upload");
  std::memcpy(ws->hstart + Workspace::kSlotsOffset, spec.slots.data(),
              spec.slots.size() * sizeof(SlotDev));
  LevelCtl& c = *reinterpret_cast<LevelCtl*>(ws->hstart);
  std::memset(&c, 0, sizeof(c));
  for (int q = 0; q < spec.Qg; ++q) {
    const int k = spec.slots[q].kind;
    if (k == CGP_KIND_BFS || k == CGP_KIND_KHOP) c.bfs_bits[q >> 6] |= 1ULL << (q & 63);
    if (k == CGP_KIND_SSSP) c.sssp_bits[q >> 6] |= 1ULL << (q & 63);
    if (k == CGP_KIND_KHOP) c.khop = 1;
  }
  for (int i = 0; i < kMaxW; ++i) c.expand[i] = ~0ULL;
  c.forced_dir = -1;
  c.halt_level = -1;
  c.max_iterations = o.max_iterations;
  int mode = o.traversal_mode;
  if (!g->can_gather()) mode = CGP_MODE_PUSH;
  c.mode = mode;
  c.num_planes = spec.depth_mode == kDepthPlanes ? kStartPlanes : 0;
  c.profile_cap = o.profile_iterations ? kProfileCap : 0;
  c.pull_vertex_threshold = static_cast<unsigned long long>(
      std::max(1.0, o.pull_frontier_ratio * static_cast<double>(V)));
  c.pull_edge_threshold = static_cast<unsigned long long>(
      std::max(1.0, o.pull_edge_ratio * static_cast<double>(g->E)));
  c.sssp_gather = sssp_gather_on(g, o) ? 1 : 0;
  c.chunk_dir = sssp_chunk_dir(spec, o) ? 1 : 0;
  c.bfs_chunked = (spec.has_bfs && (o.bfs_pull_form == 1 || o.bfs_pull_form == 2) &&
                   hp.plight.chunks > 0) ? o.bfs_pull_form : 0;
  c.has_bfs = spec.has_bfs ? 1 : 0;
  c.bnd_avail = spec.bounds ? 1 : 0;
  c.bar_limit_ns = g_grid_failure.load() == CGP_GRID_BLOCK_MISSING ? kInjectedBarrierNs : kBarrierNs;
  c.prev_dir = kDirPush;
  c.sssp_pull_edge_threshold = static_cast<unsigned long long>(
      std::max(1.0, o.sssp_pull_edge_ratio * static_cast<double>(g->E)));
  c.sssp_pull_pair_unit = o.sssp_pull_pair_ratio > 0
                              ? static_cast<unsigned long long>(
                                    std::max(1.0, o.sssp_pull_pair_ratio * static_cast<double>(g->E)))
                              : 0ULL;
  ck(cudaMemcpyAsync(ws->ctl.p, ws->hstart,
                     Workspace::kSlotsOffset + spec.slots.size() * sizeof(SlotDev),
                     cudaMemcpyHostToDevice, s), "upload ctl");
  ck(cudaEventRecord(ws->uploaded, s), "event");
  int64_t words = 0;
  for (int i = 0; i < fill.n; ++i) words += fill.span[i].words;
  const int blocks = static_cast<int>(std::min<int64_t>(g->num_sms * 8, words / (4 * kBlock) + 1));
  k_fill_spans<<<blocks, kBlock, 0, s>>>(fill);
  spec.launches++;
  if (fill_late) {  // per-slot markers: reads the uploaded slots
    k_fill_values<<<g->num_sms * 8, kBlock, 0, s>>>(values, ws->slots_dev(), spec.Qg, V, sssp_inf,
                                                    spec.uniform_inf);
    spec.launches++;
  }
  ck(cudaGetLastError(), "group start");
  Dispatch d = dispatch(W, g->offset_bytes, spec.depth_mode, g->weight_kind);
  d.seed(group_dev(ws, spec, o.profile_iterations != 0), g->dev_graph(hth), s);
  ck(cudaGetLastError(), "seed");
  spec.launches++;
}

namespace {

// What one level of the group launches under options o.
LevelLaunch level_launch(GraphImpl* g, Workspace* ws, const GroupSpec& spec, const cgp_options& o,
                         const Dispatch& d) {
  LevelLaunch L;
  L.g = group_dev(ws, spec, o.profile_iterations != 0);
  L.G = g->dev_graph(heavy_threshold(o), o.light_chunks >= 0);
  L.gr = d.grids(g->num_sms);
  L.has_bfs = spec.has_bfs;
  L.has_sssp = spec.has_sssp;
  int mode = o.traversal_mode;
  if (!g->can_gather()) mode = CGP_MODE_PUSH;
  L.pull = mode != CGP_MODE_PUSH;
  L.heavy_push = L.G.n_heavy > 0 || g->max_degree > 32;
  L.bfs_chunked = L.pull && spec.has_bfs && L.G.n_plight_chunks > 0 && o.bfs_pull_form == 1;
  L.spull = spec.has_sssp && sssp_gather_on(g, o);
  L.gvec = vector_rows(spec, L.g.values);
  L.lchunks = o.light_chunks >= 0;
  L.bounds = spec.bounds;
  L.dense_unroll = o.dense_unroll == 2 ? 2 : 1;
  L.chunk_dir = L.spull && sssp_chunk_dir(spec, o);
  L.kt = nullptr;
  return L;
}

// Edges x mask words up to which SSSP levels run fused: below the line the
// launches weigh more (mixed R-MAT 17, 48 slots, 3.7M: 1.33 ms fused against
// 1.72 launched; directed 200K, 100 slots, 4.8M: 3.4 against 3.6), above it the
// launched kernels' own register budgets do (R-MAT 20, 256 slots, 126M: 12.7
// against 12.3; a 1024-slot grid, 36M: 253 against 209).
constexpr int64_t kFusedWork = 1 << 24;
// Edges x slots up to which groups that only scatter run fused (see fused_loop).
constexpr int64_t kFusedScatter = 1 << 21;

// Blocks of a fused launch: one per 256 vertices and entries, as far as the GPU
// holds them all at once.
int fused_blocks(const GraphImpl* g, int most) {
  return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(most, (g->E + g->V) / 256)));
}

// Whether the group's levels run as the fused loop: the automatic loop form,
// with the kernel variants the loop holds (the default ones).
bool fused_loop(const GraphImpl* g, const GroupSpec& spec, const cgp_options& o,
                const Dispatch& d, const LevelLaunch& L) {
  if (spec.W > 4 || (spec.has_sssp && L.G.E * spec.W > kFusedWork)) return false;
  if (o.level_loop != CGP_LOOP_AUTO || !o.use_cuda_graph || o.bfs_pull_form != 0) return false;
  // serving groups on streams of their own: launched levels of different
  // groups overlap on the device, cooperative launches take all of it in turn
  if (spec.serving && (o.serve_groups > 1 || o.serve_admission == 2)) return false;
  const int most = d.traverse(spec.has_sssp).per_sm * g->num_sms;
  if (most < 1) return false;
  const int64_t work = L.G.E * spec.W;
  const bool short_lists = !L.heavy_push;  // no list above 32 edges: many levels as a rule
  // Scatter levels want more warps per SM than the loop's register budget leaves:
  // groups that only scatter run fused while launches weigh more.  Push mode, 64
  // slots on 150K vertices of 10 out-edges: 5.2 ms fused, 4.1 launched; one slot
  // 0.67 against 0.72.  (Gathering, 100 slots on 200K vertices: 3.2 against 3.4.)
  if (spec.has_sssp && !L.spull && short_lists && L.G.E * spec.n > kFusedScatter) return false;
  // Beside other traversals only tiny groups, and others as far as their launches
  // do not queue up: cooperative launches that do not fit next to each other run in
  // turn, each leaving the GPU idle at its barriers, where launched levels
  // interleave.  Calls/s of 2, 4 and 8 callers, fused against launched: 256 BFS on
  // R-MAT 20 557, 559, 563 against 586, 646, 656; mixed R-MAT 17 801, 836, 845
  // against 830, 1051, 1117; 16 SSSP on a 96 x 97 grid (a third of the GPU's blocks)
  // 997, 1024, 1014 against 650, 966, 1121; but one BFS on R-MAT 11 14152, 26189,
  // 25108 against 6328, 10429, 8878, and on R-MAT 12 12305, 12096, 12202 against
  // 6252, 10734, 11703: a traversal of a few levels on so small a graph is over
  // before the next call's launch.  One BFS on R-MAT 12 beside the R-MAT 20 batch
  // took 400 us (90%: 1590) when both were fused, 184 (359) by this rule.
  const int callers = OnDevice::callers(g->device), blocks = fused_blocks(g, most);
  if (callers > 1 && work > (spec.has_sssp ? 1 << 15 : 1 << 16)) {
    if (2 * callers * blocks > 5 * most) return false;
    const bool quick = !spec.has_sssp && !short_lists && work <= 1 << 18;
    if (5 * blocks > 3 * most && !quick) return false;
  }
  if (spec.has_sssp && (L.dense_unroll == 2 || (L.spull && !(L.gvec && L.lchunks)))) return false;
  return true;
}

// Levels per launch of the fused loop: enough that the launches between are
// nothing, few enough that a traversal that cannot converge (negative
// weights) keeps coming back to the host.
constexpr int kFusedLevels = 256;

// Enqueues up to `levels` levels as one cooperative launch; 0 when it does not fit.
int enqueue_fused(GraphImpl* g, const GroupSpec& spec, const Dispatch& d, LevelLaunch& L,
                  cudaStream_t s, int levels) {
  const TraverseKernel k = d.traverse(spec.has_sssp);
  const int blocks = fused_blocks(g, k.per_sm * g->num_sms);
  const int32_t injected = g_grid_failure.load();
  if (injected == CGP_GRID_DOES_NOT_FIT) return 0;
  int flags = L.heavy_push ? kTraverseHeavy : 0;
  if (injected == CGP_GRID_BLOCK_MISSING && blocks > 1) flags |= kTraverseBlockMissing;
  void* args[] = {&L.g, &L.G, &levels, &flags};
  const cudaError_t e = cudaLaunchCooperativeKernel(k.fn, dim3(blocks), dim3(kBlock), args, 0, s);
  if (e == cudaErrorCooperativeLaunchTooLarge) {  // part of the GPU is reserved: launch the levels
    cudaGetLastError();
    return 0;
  }
  ck(e, "fused level loop");
  return 1;
}

// Enqueues `levels` levels as one launch of the fused loop (`fused`), as a replayed
// CUDA graph or as plain launches, and returns the kernels launched; levels < 0:
// the whole traversal as one device-looped graph (a WHILE conditional node
// around one level, the condition set by the level's last kernel from the done
// flag).  A fused launch that does not fit becomes at most 8 launched levels:
// `levels` is then what was enqueued.
int enqueue_levels(GraphImpl* g, Workspace* ws, const GroupSpec& spec, const cgp_options& o,
                   cudaStream_t s, int& levels, KernelTimer* kt, bool fused) {
  Dispatch d = dispatch(spec.W, g->offset_bytes, spec.depth_mode, g->weight_kind);
  LevelLaunch L = level_launch(g, ws, spec, o, d);
  if (fused) {
    const int n = enqueue_fused(g, spec, d, L, s, levels);
    if (n > 0) return n;
    levels = std::min(levels, 8);
  }
  L.kt = kt;
  if (!o.use_cuda_graph || kt != nullptr) {
    int n = 0;
    for (int i = 0; i < levels; ++i) n += d.enqueue(L, s);
    ck(cudaGetLastError(), "level launch");
    return n;
  }
  L.kt = nullptr;
  const bool loop = levels < 0;
  auto key = std::make_tuple(spec.W, g->offset_bytes, spec.depth_mode, g->weight_kind,
                             (spec.has_bfs ? 1 : 0) | (spec.has_sssp ? 2 : 0) | (L.pull ? 4 : 0) |
                                 (o.profile_iterations ? 8 : 0) | (L.dense_unroll == 2 ? 16 : 0) |
                                 (L.spull ? 32 : 0) | (L.lchunks ? 64 : 0) | (loop ? 128 : 0) |
                                 (L.chunk_dir ? 256 : 0) | (L.bfs_chunked ? 512 : 0) |
                                 (L.bounds ? 1024 : 0),
                             levels, spec.Qg, static_cast<int>(L.G.heavy_degree), ws->generation,
                             reinterpret_cast<uint64_t>(L.g.values));
  auto it = ws->graphs.find(key);
  if (it == ws->graphs.end()) {
    cudaGraph_t graph = nullptr;
    int n = 0;
    if (loop) {
      ck(cudaGraphCreate(&graph, 0), "graph create");
      try {
        cudaGraphConditionalHandle h = 0;
        ck(cudaGraphConditionalHandleCreate(&h, graph, 1, cudaGraphCondAssignDefault),
           "conditional handle");
        cudaGraphNodeParams p{};
        p.type = cudaGraphNodeTypeConditional;
        p.conditional.handle = h;
        p.conditional.type = cudaGraphCondTypeWhile;
        p.conditional.size = 1;
        cudaGraphNode_t node = nullptr;
        ck(cudaGraphAddNode(&node, graph, nullptr, 0, &p), "conditional node");
        cudaGraph_t body = p.conditional.phGraph_out[0];
        L.device_loop = true;
        L.loop = h;
        L.level_cap = static_cast<int32_t>(std::min<int64_t>(g->V + 2, INT32_MAX - 1));
        ck(cudaStreamBeginCaptureToGraph(ws->capture, body, nullptr, nullptr, 0,
                                         cudaStreamCaptureModeThreadLocal),
           "begin capture");
        n = d.enqueue(L, ws->capture);
        cudaError_t le = cudaGetLastError();
        cudaError_t ce = cudaStreamEndCapture(ws->capture, &body);
        ck(le, "capture launch");
        ck(ce, "end capture");
      } catch (...) {
        cudaGraphDestroy(graph);
        throw;
      }
    } else {
      ck(cudaStreamBeginCapture(ws->capture, cudaStreamCaptureModeThreadLocal), "begin capture");
      for (int i = 0; i < levels; ++i) n += d.enqueue(L, ws->capture);
      cudaError_t le = cudaGetLastError();
      cudaError_t ce = cudaStreamEndCapture(ws->capture, &graph);
      ck(le, "capture launch");
      ck(ce, "end capture");
    }
    cudaGraphExec_t exec = nullptr;
    cudaError_t ie = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    ck(ie, "instantiate");
    it = ws->graphs.emplace(key, CachedGraph{exec, n}).first;
  }
  ck(cudaGraphLaunch(it->second.exec, s), "graph launch");
  return it->second.launches;
}

}  // namespace

void group_enact(GraphImpl* g, Workspace* ws, GroupSpec& spec, const cgp_options& o,
                 cudaStream_t s, GroupRun* out, int max_levels, KernelTimer* kt) {
  bool fused = false;
  if (kt == nullptr) {
    const Dispatch d = dispatch(spec.W, g->offset_bytes, spec.depth_mode, g->weight_kind);
    fused = fused_loop(g, spec, o, d, level_launch(g, ws, spec, o, d));
  }
  const int per_chunk = kt ? 1 : (o.levels_per_sync > 0 ? o.levels_per_sync
                                                        : (fused ? kFusedLevels : 8));
  int enqueued = 0;
  int chunk = 0;
  LevelCtl* snap = ws->hctl;
  int last = -1;  // snapshot of the last levels enqueued
  // A run to convergence without per-level timing is one device-looped graph:
  // the host waits once.  (The launch count of such a run is that of one
  // level; the per-level count is reported with the level count below.)
  const bool device_loop = kt == nullptr && max_levels <= 0 && o.use_cuda_graph &&
                           o.level_loop == CGP_LOOP_DEVICE;
  if (device_loop) {
    int whole = -1;
    const int per_level = enqueue_levels(g, ws, spec, o, s, whole, nullptr, false);
    ck(cudaStreamSynchronize(s), "device level loop");
    ck(cudaMemcpy(&snap[0], ws->ctl.p, sizeof(LevelCtl), cudaMemcpyDeviceToHost), "read ctl");
    last = 0;
    const LevelCtl& c = snap[0];
    spec.launches += static_cast<uint64_t>(per_level) * static_cast<uint64_t>(std::max(1, c.level));
  }
  for (;;) {
    if (device_loop) break;
    int n = per_chunk;
    if (max_levels > 0) n = std::min(n, max_levels - enqueued);
    if (n <= 0) break;
    // level time = the level kernels' classes (the open init interval of the
    // group is charged to its own class when the first level's marks flush)
    auto level_sum = [](const KernelTimer* t) {
      double x = 0;
      for (int c = 0; c < kNumClasses; ++c)
        if (c != kClassInit && c != kClassOutput && c != kClassWcc) x += t->ms[c];
      return x;
    };
    const double before = kt ? level_sum(kt) : 0.0;
    spec.launches += enqueue_levels(g, ws, spec, o, s, n, kt, fused);
    enqueued += n;
    ck(cudaMemcpyAsync(&snap[chunk & 1], ws->ctl.p, sizeof(LevelCtl), cudaMemcpyDeviceToHost, s),
       "read ctl");
    last = chunk & 1;
    ck(cudaEventRecord(ws->ev[chunk & 1], s), "event");
    bool stop = false;
    if (kt) {
      kt->flush();
      ck(cudaEventSynchronize(ws->ev[chunk & 1]), "sync level");
      out->level_ms.push_back(static_cast<float>(level_sum(kt) - before));
      stop = snap[chunk & 1].done != 0;
    } else if (fused) {
      // one launch is a whole traversal as a rule: nothing is kept in flight
      ck(cudaEventSynchronize(ws->ev[chunk & 1]), "sync levels");
      const LevelCtl& c = snap[chunk & 1];
      stop = c.done != 0 || (c.status & kStatusBarrier) != 0;
    } else if (chunk > 0) {
      ck(cudaEventSynchronize(ws->ev[(chunk - 1) & 1]), "sync chunk");
      const LevelCtl& c = snap[(chunk - 1) & 1];
      stop = c.done != 0;
    }
    if (stop) break;
    ++chunk;
  }
  if (!fused || last < 0) ck(cudaStreamSynchronize(s), "level loop");
  if (last < 0) {
    ck(cudaMemcpy(&snap[0], ws->ctl.p, sizeof(LevelCtl), cudaMemcpyDeviceToHost), "read ctl");
    last = 0;
  }
  LevelCtl c = snap[last];
  if (c.status & kStatusBarrier)
    throw ApiError{CGP_ERR_DEVICE, "grid barrier timed out at level " + std::to_string(c.level)};
  if (c.status & kStatusLevelCap)
    throw ApiError{CGP_ERR_DEVICE, "traversal did not converge within " +
                                       std::to_string(c.level) + " levels"};
  if (c.done == 2 && (c.status & kStatusPlanesExhausted)) {
    // Deeper than the depth planes can hold: add planes and resume.
    const size_t mask_bytes = static_cast<size_t>(g->V) * spec.W * 8;
    const int K = c.num_planes;
    const int K2 = std::min(kMaxPlanes, K < kInitialPlanes ? kInitialPlanes : K + 8);
    if (K2 == K) throw ApiError{CGP_ERR_DEVICE, "BFS depth exceeds 2^24 levels"};
    if (static_cast<size_t>(K2) * mask_bytes > ws->planes.bytes) {
      DevBuf bigger;
      bigger.ensure(static_cast<size_t>(K2) * mask_bytes);
      ck(cudaMemcpyAsync(bigger.p, ws->planes.p, static_cast<size_t>(K) * mask_bytes,
                         cudaMemcpyDeviceToDevice, s), "grow planes");
      ck(cudaStreamSynchronize(s), "grow planes");
      std::swap(ws->planes.p, bigger.p);
      std::swap(ws->planes.bytes, bigger.bytes);
      ws->generation++;
      ws->clear_graphs();
    }
    ck(cudaMemsetAsync(static_cast<char*>(ws->planes.p) + static_cast<size_t>(K) * mask_bytes, 0,
                       static_cast<size_t>(K2 - K) * mask_bytes, s), "zero planes");
    c.num_planes = K2;
    c.status &= ~kStatusPlanesExhausted;
    c.done = 0;
    ck(cudaMemcpyAsync(ws->ctl.p, &c, sizeof(LevelCtl), cudaMemcpyHostToDevice, s), "resume");
    ck(cudaStreamSynchronize(s), "resume");
    if (max_levels <= 0 || enqueued < max_levels) {
      group_enact(g, ws, spec, o, s, out, max_levels > 0 ? max_levels - enqueued : 0, kt);
      return;
    }
  }
  spec.depth_bits = 0;  // depths written are at most c.level
  while (spec.depth_bits < c.num_planes && (c.level >> spec.depth_bits) != 0) ++spec.depth_bits;
  out->iterations = c.level;
  out->push_levels = c.push_levels;
  out->pull_levels = c.pull_levels;
  out->frontier_vertices = c.total_frontier;
  out->frontier_edges = c.total_edges;
  out->status = c.status;
  out->counters = c.total;
  if (o.profile_iterations) {
    int n = std::min(c.level, kProfileCap);
    out->profiles.resize(n);
    if (n > 0)
      ck(cudaMemcpy(out->profiles.data(), ws->prof.p, n * sizeof(LevelProfile),
                    cudaMemcpyDeviceToHost), "read profiles");
  }
}

void group_enqueue_levels(GraphImpl* g, Workspace* ws, GroupSpec& spec, const cgp_options& o,
                          cudaStream_t s, int levels) {
  const Dispatch d = dispatch(spec.W, g->offset_bytes, spec.depth_mode, g->weight_kind);
  const bool fused = fused_loop(g, spec, o, d, level_launch(g, ws, spec, o, d));
  spec.launches += enqueue_levels(g, ws, spec, o, s, levels, nullptr, fused);
}

void group_write_output(GraphImpl* g, Workspace* ws, GroupSpec& spec, OutMap om,
                        int query_major, cudaStream_t s) {
  spec.launches++;
  const dim3 grid(g->num_sms * 8, query_major ? std::min(spec.n, 65535) : 1);
  if (spec.depth_mode == kDepthPlanes) {
    switch (spec.W) {
#define CGP_MAT(WW) case WW: k_materialize_planes<WW><<<grid, kBlock, 0, s>>>(ws->visited.as<uint64_t>(), ws->planes.as<uint64_t>(), spec.depth_bits, g->V, spec.n, om, query_major); break;
      CGP_MAT(1) CGP_MAT(2) CGP_MAT(4) CGP_MAT(8) CGP_MAT(16)
#undef CGP_MAT
    }
  } else {
    k_copy_values<<<grid, kBlock, 0, s>>>(group_dev(ws, spec, false).values, ws->slots_dev(),
                                          g->V, spec.n, spec.Qg, om, query_major);
  }
  ck(cudaGetLastError(), "write output");
}

}  // namespace cgp

// ======================================================================
//                                C ABI
// ======================================================================
using namespace cgp;

namespace {

// Symmetry check on a host CSR with sorted rows.
bool csr_is_symmetric(const std::vector<int64_t>& row, const int32_t* col, int64_t V) {
  for (int64_t u = 0; u < V; ++u) {
    for (int64_t e = row[u]; e < row[u + 1]; ++e) {
      int32_t v = col[e];
      const int32_t* b = col + row[v];
      const int32_t* en = col + row[v + 1];
      bool sorted = std::is_sorted(b, en);
      bool found = sorted ? std::binary_search(b, en, static_cast<int32_t>(u))
                          : std::find(b, en, static_cast<int32_t>(u)) != en;
      if (!found) return false;
    }
  }
  return true;
}

thread_local std::vector<LevelProfile> t_profiles;
thread_local std::vector<float> t_level_ms;  // per-level kernel time (profile_kernels)
thread_local cgp_kernel_profile t_kernel_profile;

}  // namespace

extern "C" {

cgp_status cgp_graph_create(const void* row_offsets, int32_t offset_bytes,
                            const int32_t* col_indices, const void* weights,
                            int32_t weight_kind, int64_t num_vertices, int64_t num_edges,
                            int32_t flags, cgp_graph** out) {
  clear_error();
  if (out == nullptr) return set_error(CGP_ERR_INVALID_ARG, "out is NULL");
  *out = nullptr;
  if (row_offsets == nullptr || (num_edges > 0 && col_indices == nullptr))
    return set_error(CGP_ERR_INVALID_ARG, "row_offsets/col_indices is NULL");
  if (offset_bytes != 4 && offset_bytes != 8)
    return set_error(CGP_ERR_INVALID_ARG, "offset_bytes must be 4 or 8");
  if (num_vertices <= 0 || num_vertices >= INT32_MAX || num_edges < 0)
    return set_error(CGP_ERR_INVALID_ARG, "vertex count must be in [1, 2^31-1)");
  if (weight_kind != CGP_WEIGHT_NONE && weight_kind != CGP_WEIGHT_U32 && weight_kind != CGP_WEIGHT_F32)
    return set_error(CGP_ERR_INVALID_ARG, "unknown weight_kind");
  if (weight_kind != CGP_WEIGHT_NONE && weights == nullptr)
    return set_error(CGP_ERR_INVALID_ARG, "weights is NULL");
  auto* g = new (std::nothrow) cgp_graph();
  if (!g) return set_error(CGP_ERR_OOM, "host allocation failed");
  try {
    GraphImpl& G = g->impl;
    ck(cudaGetDevice(&G.device), "cudaGetDevice");
    ck(cudaDeviceGetAttribute(&G.num_sms, cudaDevAttrMultiProcessorCount, G.device), "attr");
    G.V = num_vertices;
    G.E = num_edges;
    G.weight_kind = weight_kind;
    const bool on_dev = (flags & CGP_GRAPH_DEVICE_POINTERS) != 0;
    const cudaMemcpyKind kind = on_dev ? cudaMemcpyDeviceToHost : cudaMemcpyHostToHost;
    // host copies: 64-bit offsets and (for validation / transpose) columns
    std::vector<int64_t> hrow(num_vertices + 1);
    if (offset_bytes == 8) {
      ck(cudaMemcpy(hrow.data(), row_offsets, (num_vertices + 1) * 8, kind), "read offsets");
    } else {
      std::vector<int32_t> r32(num_vertices + 1);
      ck(cudaMemcpy(r32.data(), row_offsets, (num_vertices + 1) * 4, kind), "read offsets");
      for (int64_t i = 0; i <= num_vertices; ++i) hrow[i] = r32[i];
    }
    if (hrow[0] != 0 || hrow[num_vertices] != num_edges)
      throw ApiError{CGP_ERR_INVALID_ARG, "row_offsets must start at 0 and end at num_edges"};
    for (int64_t v = 0; v < num_vertices; ++v) {
      if (hrow[v + 1] < hrow[v]) throw ApiError{CGP_ERR_INVALID_ARG, "row_offsets not monotone"};
      G.max_degree = std::max(G.max_degree, hrow[v + 1] - hrow[v]);
      G.n_deg32 += hrow[v + 1] - hrow[v] > 32 ? 1 : 0;
    }
    std::vector<int32_t> hcol(num_edges);
    if (num_edges > 0)
      ck(cudaMemcpy(hcol.data(), col_indices, num_edges * 4, kind), "read columns");
    for (int64_t e = 0; e < num_edges; ++e)
      if (hcol[e] < 0 || hcol[e] >= num_vertices)
        throw ApiError{CGP_ERR_INVALID_ARG, "column index out of range at edge " + std::to_string(e)};
    // device offsets: 32-bit unless asked for 64 or the edge count needs it
    const bool off64 = (flags & CGP_GRAPH_OFFSETS64) != 0 || num_edges >= INT32_MAX;
    G.offset_bytes = off64 ? 8 : 4;
    G.row.ensure((num_vertices + 1) * G.offset_bytes);
    if (off64) {
      ck(cudaMemcpy(G.row.p, hrow.data(), (num_vertices + 1) * 8, cudaMemcpyHostToDevice), "upload offsets");
    } else {
      std::vector<int32_t> r32(hrow.begin(), hrow.end());
      ck(cudaMemcpy(G.row.p, r32.data(), (num_vertices + 1) * 4, cudaMemcpyHostToDevice), "upload offsets");
    }
    G.col.ensure(std::max<int64_t>(num_edges, 1) * 4);
    if (num_edges > 0)
      ck(cudaMemcpy(G.col.p, hcol.data(), num_edges * 4, cudaMemcpyHostToDevice), "upload columns");
    if (weight_kind != CGP_WEIGHT_NONE) {
      G.w.ensure(std::max<int64_t>(num_edges, 1) * 4);
      if (num_edges > 0)
        ck(cudaMemcpy(G.w.p, weights, num_edges * 4,
                      on_dev ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice), "upload weights");
    }
    G.symmetric = (flags & CGP_GRAPH_SYMMETRIC) != 0 || csr_is_symmetric(hrow, hcol.data(), num_vertices);
    // Pull CSR.  A directed graph needs its transpose.  A symmetric one can be
    // pulled over directly, except that an SSSP gather also needs, per entry
    // (v, u), the weight of u -> v: the transpose (counting sort by
    // destination, sources ascending) gives it, and when its columns equal
    // the CSR's (sorted lists, no multi-edge mismatch) only the weights are
    // kept, or nothing when they equal w.
    std::vector<int64_t> trow;
    const bool weighted = weight_kind != CGP_WEIGHT_NONE;
    if (!G.symmetric || weighted) {
      std::vector<uint32_t> hw;
      if (weighted) {
        hw.resize(num_edges);
        if (num_edges > 0)
          ck(cudaMemcpy(hw.data(), weights, num_edges * 4, kind), "read weights");
      }
      trow.assign(num_vertices + 1, 0);
      for (int64_t e = 0; e < num_edges; ++e) trow[hcol[e] + 1]++;
      for (int64_t v = 0; v < num_vertices; ++v) trow[v + 1] += trow[v];
      std::vector<int64_t> cur(trow.begin(), trow.end() - 1);
      std::vector<int32_t> tcol(num_edges);
      std::vector<uint32_t> tw(weighted ? num_edges : 0);
      for (int64_t u = 0; u < num_vertices; ++u)
        for (int64_t e = hrow[u]; e < hrow[u + 1]; ++e) {
          const int64_t p = cur[hcol[e]]++;
          tcol[p] = static_cast<int32_t>(u);
          if (weighted) tw[p] = hw[e];
        }
      const bool aligned = G.symmetric && trow == hrow && tcol == hcol;
      if (aligned) {
        trow.clear();
        if (tw != hw) {
          G.tw.ensure(std::max<int64_t>(num_edges, 1) * 4);
          ck(cudaMemcpy(G.tw.p, tw.data(), num_edges * 4, cudaMemcpyHostToDevice), "upload t-weights");
        }
      } else {
        G.trow.ensure((num_vertices + 1) * G.offset_bytes);
        if (off64) {
          ck(cudaMemcpy(G.trow.p, trow.data(), (num_vertices + 1) * 8, cudaMemcpyHostToDevice), "upload t-offsets");
        } else {
          std::vector<int32_t> r32(trow.begin(), trow.end());
          ck(cudaMemcpy(G.trow.p, r32.data(), (num_vertices + 1) * 4, cudaMemcpyHostToDevice), "upload t-offsets");
        }
        G.tcol.ensure(std::max<int64_t>(num_edges, 1) * 4);
        if (num_edges > 0)
          ck(cudaMemcpy(G.tcol.p, tcol.data(), num_edges * 4, cudaMemcpyHostToDevice), "upload t-columns");
        if (weighted) {
          G.tw.ensure(std::max<int64_t>(num_edges, 1) * 4);
          if (num_edges > 0)
            ck(cudaMemcpy(G.tw.p, tw.data(), num_edges * 4, cudaMemcpyHostToDevice), "upload t-weights");
        }
      }
    }
    {
      const std::vector<int64_t>& in = trow.empty() ? hrow : trow;
      for (int64_t v = 1; v < num_vertices; ++v)
        if (in[v + 1] - in[v] > in[G.hub + 1] - in[G.hub]) G.hub = static_cast<int32_t>(v);
    }
    {
      std::lock_guard<std::mutex> lk(g_host_mu);
      HostCsr& hc = g_host[&G];
      hc.row = std::move(hrow);
      hc.trow = std::move(trow);
    }
    *out = g;
    return CGP_OK;
  } catch (...) {
    cgp_status st = translate_exception();
    delete g;
    return st;
  }
}

cgp_status cgp_graph_destroy(cgp_graph* g) {
  clear_error();
  if (g == nullptr) return CGP_OK;
  {
    std::lock_guard<std::mutex> lk(g_host_mu);
    g_host.erase(&g->impl);
  }
  cudaDeviceSynchronize();
  delete g;
  return CGP_OK;
}

cgp_status cgp_graph_info(const cgp_graph* g, int64_t* V, int64_t* E, int32_t* wk, int32_t* sym) {
  if (g == nullptr) return set_error(CGP_ERR_INVALID_ARG, "graph is NULL");
  if (V) *V = g->impl.V;
  if (E) *E = g->impl.E;
  if (wk) *wk = g->impl.weight_kind;
  if (sym) *sym = g->impl.symmetric ? 1 : 0;
  return CGP_OK;
}

cgp_status cgp_last_profiles(cgp_level_profile* out, int32_t cap, int32_t* count) {
  if (count == nullptr) return set_error(CGP_ERR_INVALID_ARG, "count is NULL");
  int n = static_cast<int>(t_profiles.size());
  *count = n;
  if (out != nullptr) {
    for (int i = 0; i < std::min(n, cap); ++i) {
      out[i].iteration = t_profiles[i].level;
      out[i].mode = t_profiles[i].dir;
      out[i].frontier_size = t_profiles[i].frontier;
      out[i].frontier_edges = t_profiles[i].edges;
      out[i].next_size = t_profiles[i].next;
      out[i].query_convergence_mask = t_profiles[i].active0;
      out[i].new_pairs = t_profiles[i].new_pairs;
      out[i].pull_vertices = t_profiles[i].pull_vertices;
      out[i].pull_edges = t_profiles[i].pull_edges;
      out[i].sssp_pairs = t_profiles[i].sssp_pairs;
      out[i].sssp_active = t_profiles[i].sssp_active;
      out[i].improved = t_profiles[i].improved;
      out[i].sssp_pull_vertices = t_profiles[i].spull_vertices;
      out[i].sssp_pull_edges = t_profiles[i].spull_edges;
      out[i].sssp_mode = t_profiles[i].sdir;
      out[i].kernel_ms = i < static_cast<int>(t_level_ms.size()) ? t_level_ms[i] : 0.0f;
    }
  }
  return CGP_OK;
}

cgp_status cgp_debug_fail_allocations(int64_t after) {
  g_fail_alloc_countdown.store(after < 0 ? -1 : after);
  return CGP_OK;
}

cgp_status cgp_debug_grid_launches(int32_t failure) {
  clear_error();
  if (failure < CGP_GRID_OK || failure > CGP_GRID_BLOCK_MISSING)
    return set_error(CGP_ERR_INVALID_ARG, "unknown grid launch failure");
  g_grid_failure.store(failure);
  return CGP_OK;
}

cgp_status cgp_last_kernel_profile(cgp_kernel_profile* out) {
  if (out == nullptr) return set_error(CGP_ERR_INVALID_ARG, "out is NULL");
  *out = t_kernel_profile;
  return CGP_OK;
}

cgp_status cgp_batch_run(cgp_graph* graph, const cgp_query* queries, int32_t nq,
                         const cgp_options* opts, void* out, int32_t out_layout,
                         int32_t out_on_device, cgp_stats* stats) {
  clear_error();
  if (graph == nullptr) return set_error(CGP_ERR_INVALID_ARG, "graph is NULL");
  if (queries == nullptr || nq <= 0)
    return set_error(CGP_ERR_INVALID_ARG, "query batch must be non-empty");
  if (out == nullptr) return set_error(CGP_ERR_INVALID_ARG, "out is NULL");
  if (out_layout != CGP_LAYOUT_VERTEX_MAJOR && out_layout != CGP_LAYOUT_QUERY_MAJOR)
    return set_error(CGP_ERR_INVALID_ARG, "unknown out_layout");
  cgp_options o;
  if (opts) o = *opts;
  else cgp_options_init(&o);
  if (o.max_queries > 0 && nq > o.max_queries)
    return set_error(CGP_ERR_INVALID_ARG, "query batch exceeds max_queries");
  GraphImpl* g = &graph->impl;
  for (int i = 0; i < nq; ++i) {
    const cgp_query& q = queries[i];
    if (q.kind < CGP_KIND_BFS || q.kind > CGP_KIND_KHOP)
      return set_error(CGP_ERR_INVALID_ARG, "unknown query kind at index " + std::to_string(i));
    if (q.kind != CGP_KIND_WCC && (q.source < 0 || q.source >= g->V))
      return set_error(CGP_ERR_INVALID_ARG, "query source out of range at index " + std::to_string(i));
    if (q.kind == CGP_KIND_KHOP && q.k < 0)
      return set_error(CGP_ERR_INVALID_ARG, "k-hop bound must be non-negative");
  }
  std::unique_ptr<Workspace> ws;
  std::unique_ptr<KernelTimer> kt;
  try {
    ck(cudaSetDevice(g->device), "cudaSetDevice");
    ws = g->acquire();
    if (o.profile_kernels) kt = std::make_unique<KernelTimer>();
    cudaStream_t s = o.stream ? static_cast<cudaStream_t>(o.stream) : ws->stream;
    auto wall0 = std::chrono::steady_clock::now();
    const cudaEvent_t t0 = ws->t0, t1 = ws->t1;
    ck(cudaEventRecord(t0, s), "event");
    const int64_t V = g->V;
    const bool qmajor = out_layout == CGP_LAYOUT_QUERY_MAJOR;
    // output target on the device
    uint32_t* dout = static_cast<uint32_t*>(out);
    if (!out_on_device) {
      ws->stage.ensure(static_cast<size_t>(V) * nq * 4);
      dout = ws->stage.as<uint32_t>();
    }
    OutMap om;
    om.out = dout;
    om.sv = qmajor ? 1 : nq;
    om.sq = qmajor ? V : 1;
    om.qmap = nullptr;
    om.q0 = 0;
    // WCC queries: one union-find pass, labels broadcast to every WCC column
    std::vector<int> wcc_idx, trav_idx;
    for (int i = 0; i < nq; ++i) (queries[i].kind == CGP_KIND_WCC ? wcc_idx : trav_idx).push_back(i);
    GroupRun total;
    uint64_t launches = 0;
    int groups = 0;
    int W0 = 0, depth0 = 0;
    t_profiles.clear();
    t_level_ms.clear();
    if (!wcc_idx.empty()) {
      if (kt) kt->mark(kClassWcc, s);
      ws->wcc.ensure(static_cast<size_t>(V + 1) * 4);
      launches += wcc_labels(g, ws->wcc.as<uint32_t>(), s);
      for (int i : wcc_idx) broadcast_labels(ws->wcc.as<uint32_t>(), V, om, i, s);
      launches += wcc_idx.size();
      if (kt) kt->mark(-1, s);
    }
    // Traversal groups of up to 64*W queries, in submission order.  A batch
    // with many BFS-like and many SSSP queries is split by kind first (each
    // kind then gets its own groups): the kinds share no state, a pure BFS
    // group keeps its depths in bit-planes, and a pure SSSP group reads no
    // BFS slots in its gathers.  Small mixed batches share one group, as in
    // the reference's hybrid batch.
    std::vector<std::vector<int>> classes;
    {
      std::vector<int> bfs_like, sssp_q;
      for (int i : trav_idx) (queries[i].kind == CGP_KIND_SSSP ? sssp_q : bfs_like).push_back(i);
      if (bfs_like.size() >= 64 && sssp_q.size() >= 64) classes = {bfs_like, sssp_q};
      else if (!trav_idx.empty()) classes = {trav_idx};
    }
    struct GroupPlan {
      const std::vector<int>* cls;
      size_t begin;
      int n;
      int W;
    };
    std::vector<GroupPlan> plan;
    for (const auto& cls : classes) {
      const int Wc = choose_words(static_cast<int>(cls.size()), o.mask_words);
      const int per_group = 64 * Wc;
      for (size_t b = 0; b < cls.size(); b += per_group) {
        const int n = static_cast<int>(std::min<size_t>(per_group, cls.size() - b));
        plan.push_back(GroupPlan{&cls, b, n, choose_words(n, o.mask_words)});
      }
    }
    const bool single = plan.size() == 1;
    // Host output: each group's result block is copied to the host on the
    // copy stream as soon as it is written, overlapping the next group's
    // traversal, when its destination is one contiguous block (query-major
    // rows, or a run of vertex-major columns as a 2D copy).
    // Pageable outputs are copied once at the end by several threads
    // (HostCopier): R-MAT 18, 90 k-hop queries, 94 MB into a new array.
    const bool host_out = !out_on_device && !o.discard_results;
    const bool staged_out = host_out && !HostCopier::direct(out);
    bool copied_all = host_out;
    std::vector<char> col_copied(host_out ? nq : 0, 0);
    for (const GroupPlan& gp : plan) {
      const int n = gp.n;
      std::vector<cgp_query> gq(n);
      for (int i = 0; i < n; ++i) gq[i] = queries[(*gp.cls)[gp.begin + i]];
      GroupSpec spec = make_group(gq.data(), n, gp.W, o.depth_mode);
      // A device vertex-major output holding exactly this group's columns is
      // used directly as the working value matrix (no copy at the end).
      bool in_place = out_on_device && !qmajor && single && wcc_idx.empty() &&
                      spec.depth_mode != kDepthPlanes;
      if (pad_rows(g, ws.get(), spec, o, in_place)) in_place = false;
      if (in_place) spec.external_values = dout;
      const OnDevice running(g->device);
      if (kt) kt->mark(kClassInit, s);
      group_prepare(g, ws.get(), spec, o, s);
      GroupRun r;
      group_enact(g, ws.get(), spec, o, s, &r, 0, kt.get());
      if (r.status != 0) throw ApiError{CGP_ERR_DEVICE, "device status " + std::to_string(r.status)};
      if (!in_place) {
        if (kt) kt->mark(kClassOutput, s);
        std::vector<int32_t> qmap(n);
        for (int i = 0; i < n; ++i) qmap[i] = (*gp.cls)[gp.begin + i];
        bool run = true;  // consecutive columns
        for (int i = 1; i < n; ++i) run = run && qmap[i] == qmap[0] + i;
        OutMap m = om;
        m.q0 = qmap[0];
        // sized with the group, so that a later batch in another order does
        // not allocate between its traversal and its output
        ws->qmap.ensure(static_cast<size_t>(n) * 4);
        if (!run) {
          ck(cudaMemcpyAsync(ws->qmap.p, qmap.data(), static_cast<size_t>(n) * 4,
                             cudaMemcpyHostToDevice, s), "upload query map");
          m.qmap = ws->qmap.as<int32_t>();
        }
        group_write_output(g, ws.get(), spec, m, qmajor, s);
        if (kt) kt->mark(-1, s);
        if (host_out && !staged_out && run && wcc_idx.empty()) {
          ck(cudaEventRecord(ws->out_ready, s), "event");
          ck(cudaStreamWaitEvent(ws->copy, ws->out_ready, 0), "wait");
          const size_t q0 = static_cast<size_t>(qmap[0]);
          char* hbase = static_cast<char*>(out);
          const char* dbase = reinterpret_cast<const char*>(dout);
          if (qmajor) {
            const size_t off = q0 * static_cast<size_t>(V) * 4;
            ck(cudaMemcpyAsync(hbase + off, dbase + off, static_cast<size_t>(n) * V * 4,
                               cudaMemcpyDeviceToHost, ws->copy), "copy out");
          } else {
            ck(cudaMemcpy2DAsync(hbase + q0 * 4, static_cast<size_t>(nq) * 4, dbase + q0 * 4,
                                 static_cast<size_t>(nq) * 4, static_cast<size_t>(n) * 4, V,
                                 cudaMemcpyDeviceToHost, ws->copy), "copy out");
          }
          for (int i = 0; i < n; ++i) col_copied[qmap[i]] = 1;
        }
      }
      launches += spec.launches;
      total.iterations = std::max(total.iterations, r.iterations);
      total.push_levels += r.push_levels;
      total.pull_levels += r.pull_levels;
      total.frontier_vertices += r.frontier_vertices;
      total.frontier_edges += r.frontier_edges;
      total.counters.new_pairs += r.counters.new_pairs;
      total.counters.pull_vertices += r.counters.pull_vertices;
      total.counters.pull_edges += r.counters.pull_edges;
      total.counters.sssp_pairs += r.counters.sssp_pairs;
      total.counters.sssp_active += r.counters.sssp_active;
      total.counters.improved += r.counters.improved;
      total.counters.spull_vertices += r.counters.spull_vertices;
      total.counters.spull_edges += r.counters.spull_edges;
      if (groups == 0) {
        W0 = spec.W;
        depth0 = spec.depth_mode;
        t_profiles = r.profiles;
        t_level_ms = r.level_ms;
      }
      ++groups;
    }
    ck(cudaEventRecord(t1, s), "event");
    for (char c : col_copied) copied_all = copied_all && c;
    if (staged_out) {
      g->copy_out({{out, dout, static_cast<size_t>(V) * nq * 4}}, s);
    } else if (host_out && !copied_all)
      ck(cudaMemcpyAsync(out, dout, static_cast<size_t>(V) * nq * 4, cudaMemcpyDeviceToHost, s),
         "copy out");
    ck(cudaStreamSynchronize(s), "batch");
    if (host_out) ck(cudaStreamSynchronize(ws->copy), "copy out");
    float ms = 0;
    cudaEventElapsedTime(&ms, t0, t1);
    if (kt) {
      kt->flush();
      std::memset(&t_kernel_profile, 0, sizeof(t_kernel_profile));
      for (int c = 0; c < kNumClasses; ++c) {
        t_kernel_profile.ms[c] = kt->ms[c];
        t_kernel_profile.launches[c] = kt->count[c];
      }
    }
    if (stats) {
      std::memset(stats, 0, sizeof(*stats));
      stats->iterations = total.iterations;
      stats->push_levels = total.push_levels;
      stats->pull_levels = total.pull_levels;
      stats->groups = groups;
      stats->gpu_time_ms = ms;
      stats->wall_time_ms = std::chrono::duration<float, std::milli>(
                                std::chrono::steady_clock::now() - wall0).count();
      stats->frontier_vertices = total.frontier_vertices;
      stats->frontier_edges = total.frontier_edges;
      stats->mask_words = W0;
      stats->depth_mode = depth0 == kDepthPlanes ? CGP_DEPTH_PLANES : CGP_DEPTH_DIRECT;
      stats->kernel_launches = launches;
      stats->new_pairs = total.counters.new_pairs;
      stats->pull_vertices = total.counters.pull_vertices;
      stats->pull_edges = total.counters.pull_edges;
      stats->sssp_pairs = total.counters.sssp_pairs;
      stats->sssp_active = total.counters.sssp_active;
      stats->improved = total.counters.improved;
      stats->sssp_pull_vertices = total.counters.spull_vertices;
      stats->sssp_pull_edges = total.counters.spull_edges;
    }
    g->release(std::move(ws));
    return CGP_OK;
  } catch (...) {
    cgp_status st = translate_exception();
    if (ws) {
      cudaStreamSynchronize(ws->stream);
      g->release(std::move(ws));
    }
    return st;
  }
}

}  // extern "C"
