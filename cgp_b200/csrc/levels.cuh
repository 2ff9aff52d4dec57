// Kernel launches of one traversal level, by mask width (included by levels_w*.cu).
#pragma once

#include <algorithm>

#include "kernels.cuh"
#include "levels.h"

namespace cgp {

using namespace dev;

namespace {

template <typename K>
int occupancy_grid(K kernel, int sms) {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kBlock, 0) != cudaSuccess) {
    cudaGetLastError();
    per_sm = 2;
  }
  return std::max(1, per_sm) * sms;
}

// Enqueues one level; returns the number of kernels launched.
template <int W, typename OT, int DEPTH, int WK>
int enqueue_level_t(const LevelLaunch& L, cudaStream_t s) {
  const int t = L.gr.tile, h = L.gr.heavy, c = L.gr.clear;
  KernelTimer* kt = L.kt;
  int n = 0;
  if (kt) kt->mark(kClassClear, s);
  k_clear_next<W><<<c, kBlock, 0, s>>>(L.g, L.G.E);
  ++n;
  if (L.g.fsum != nullptr && (L.pull || L.spull)) {
    k_frontier_summary<W, OT><<<c, kBlock, 0, s>>>(L.g, L.G);
    ++n;
  }
  if (L.bounds) {
    k_gather_bounds<W, OT, WK><<<t, kBlock, 0, s>>>(L.g, L.G);
    ++n;
  }
  if (L.heavy_push) {
    k_heavy_queue<OT><<<c, kBlock, 0, s>>>(L.g, L.G);
    ++n;
  }
  if (L.has_bfs) {
    if (kt) kt->mark(kClassBfsPush, s);
    k_bfs_push<W, OT, DEPTH><<<t, kBlock, 0, s>>>(L.g, L.G);
    ++n;
    if (L.heavy_push) {
      k_bfs_push_heavy<W, OT, DEPTH><<<h, kBlock, 0, s>>>(L.g, L.G);
      ++n;
    }
    if (L.pull) {
      if (kt) kt->mark(kClassBfsPull, s);
      k_bfs_pull<W, OT, DEPTH><<<t, kBlock, 0, s>>>(L.g, L.G);
      ++n;
      if (L.G.n_pmid > 0) {  // in-degree 33 .. heavy_degree: warp per vertex
        k_bfs_pull_mid<W, OT, DEPTH><<<L.gr.bfs_mid, kBlock, 0, s>>>(L.g, L.G);
        ++n;
      }
      if (L.bfs_chunked) {  // each of the two forms returns at once on the other's levels
        k_bfs_pull_chunked<W, OT, DEPTH><<<L.gr.bfs_chunked, kBlock, 0, s>>>(L.g, L.G);
        ++n;
      }
      if (L.G.n_pheavy) {
        k_bfs_pull_heavy<W, OT><<<h, kBlock, 0, s>>>(L.g, L.G);
        k_bfs_pull_heavy_commit<W, OT, DEPTH><<<std::max(1, (L.G.n_pheavy + kBlock - 1) / kBlock), kBlock, 0, s>>>(L.g, L.G);
        n += 2;
      }
    }
  }
  if (L.has_sssp) {
    if (kt) kt->mark(kClassSsspPush, s);
    k_sssp_push<W, OT, WK><<<t, kBlock, 0, s>>>(L.g, L.G);
    if (kt) kt->mark(kClassSsspDense, s);
    if (L.dense_unroll == 2)
      k_sssp_list<W, OT, WK, 8><<<L.gr.dense2, kBlock, 0, s>>>(L.g, L.G);
    else
      k_sssp_list<W, OT, WK, 4><<<L.gr.dense, kBlock, 0, s>>>(L.g, L.G);
    n += 2;
    if (L.heavy_push) {
      if (kt) kt->mark(kClassSsspHeavy, s);
      k_sssp_push_heavy<W, OT, WK><<<h, kBlock, 0, s>>>(L.g, L.G);
      ++n;
    }
    if (L.spull) {
      if (kt) kt->mark(kClassSsspPull, s);
      // heavy vertices first: the light vertices' gathers of the same level
      // then read the hubs' lowered distances (the level is Gauss-Seidel)
      if (L.gvec ? L.G.n_sheavy : L.G.n_pheavy) {
        if (L.gvec && W <= 4) {
          // whole-row and chunk-skipping variants; each returns at once on the
          // other's levels
          k_sssp_pull_heavy_vec<W, OT, WK, 1><<<L.gr.gather_heavy_vec, kBlock, 0, s>>>(L.g, L.G);
          k_sssp_pull_heavy_vec<W, OT, WK, 2><<<L.gr.gather_heavy_vec2, kBlock, 0, s>>>(L.g, L.G);
          ++n;
        } else if (L.gvec) {
          k_sssp_pull_heavy_vec<W, OT, WK, 0><<<L.gr.gather_heavy_vec, kBlock, 0, s>>>(L.g, L.G);
        } else {
          k_sssp_pull_heavy<W, OT, WK><<<L.gr.gather_heavy, kBlock, 0, s>>>(L.g, L.G);
        }
        ++n;
      }
      if constexpr (W <= 4) {
        if (L.gvec && L.lchunks) {
          k_sssp_pull_rows<W, OT, WK><<<L.gr.gather_rows, kBlock, 0, s>>>(L.g, L.G);
        } else if (L.gvec) {
          k_sssp_pull_vec<W, OT, WK><<<L.gr.gather_vec, kBlock, 0, s>>>(L.g, L.G);
        } else {
          k_sssp_pull<W, OT, WK><<<L.gr.gather, kBlock, 0, s>>>(L.g, L.G);
        }
      } else if (L.gvec && L.lchunks) {
        k_sssp_pull_rows<4, OT, WK, W><<<L.gr.gather_rows, kBlock, 0, s>>>(L.g, L.G);
      } else if (L.gvec) {
        k_sssp_pull_vec<W, OT, WK><<<L.gr.gather_vec, kBlock, 0, s>>>(L.g, L.G);
      } else {
        k_sssp_pull<W, OT, WK><<<L.gr.gather, kBlock, 0, s>>>(L.g, L.G);
      }
      ++n;
    }

  }
  if (kt) kt->mark(kClassLevelEnd, s);
  if (L.chunk_dir) {
    k_chunk_census<W, OT><<<c, kBlock, 0, s>>>(L.g, L.G);
    ++n;
  }
  if (L.device_loop) k_level_end_loop<W><<<1, 32, 0, s>>>(L.g, L.loop, L.level_cap);
  else k_level_end<W><<<1, 32, 0, s>>>(L.g);
  ++n;
  if (kt) kt->mark(-1, s);
  return n;
}

template <int W, typename OT, int DEPTH, int WK>
Grids grids_t(int sms) {
  static int tile = 0, heavy = 0, dense = 0, dense2 = 0, gather = 0, gather_heavy = 0;
  static int gather_vec = 0, gather_heavy_vec = 0, gather_rows = 0, gather_heavy_vec2 = 0;
  static int bfs_chunked = 0, bfs_mid = 0;
  if (tile == 0) {
    bfs_chunked = occupancy_grid(k_bfs_pull_chunked<W, OT, DEPTH>, sms);
    bfs_mid = occupancy_grid(k_bfs_pull_mid<W, OT, DEPTH>, sms);
    gather_rows = occupancy_grid(k_sssp_pull_rows<(W < 4 ? W : 4), OT, WK, W>, sms);
    gather_vec = occupancy_grid(k_sssp_pull_vec<W, OT, WK>, sms);
    gather_heavy_vec = occupancy_grid(k_sssp_pull_heavy_vec<W, OT, WK, (W <= 4 ? 1 : 0)>, sms);
    gather_heavy_vec2 = occupancy_grid(k_sssp_pull_heavy_vec<W, OT, WK, 2>, sms);
    gather = occupancy_grid(k_sssp_pull<W, OT, WK>, sms);
    gather_heavy = occupancy_grid(k_sssp_pull_heavy<W, OT, WK>, sms);
    dense = occupancy_grid(k_sssp_list<W, OT, WK, 4>, sms);
    dense2 = occupancy_grid(k_sssp_list<W, OT, WK, 8>, sms);
    int a = occupancy_grid(k_bfs_push<W, OT, DEPTH>, sms);
    int b = occupancy_grid(k_bfs_pull<W, OT, DEPTH>, sms);
    int c = occupancy_grid(k_sssp_push<W, OT, WK>, sms);
    tile = std::min(a, std::min(b, c));
    heavy = std::min(occupancy_grid(k_bfs_pull_heavy<W, OT>, sms),
                     occupancy_grid(k_sssp_push_heavy<W, OT, WK>, sms));
  }
  Grids g;
  g.tile = tile;
  g.heavy = heavy;
  g.clear = sms * 4;
  g.dense = dense;
  g.dense2 = dense2;
  g.gather = gather;
  g.gather_heavy = gather_heavy;
  g.gather_vec = gather_vec;
  g.gather_heavy_vec = gather_heavy_vec;
  g.gather_rows = gather_rows;
  g.gather_heavy_vec2 = gather_heavy_vec2;
  g.bfs_chunked = bfs_chunked;
  g.bfs_mid = bfs_mid;
  return g;
}

template <int W, typename OT>
void seed_t(const GroupDev& g, const DevGraph& G, cudaStream_t s) {
  k_seed<W, OT><<<1, kBlock, 0, s>>>(g, G);
}

template <int W, typename OT, int DEPTH, int WK, bool kSssp>
TraverseKernel traverse_kernel() {
  auto* fn = k_traverse<W, OT, DEPTH, WK, kSssp>;
  static const int per_sm = [&] {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, kBlock, 0) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    return n;
  }();
  return {reinterpret_cast<const void*>(fn), per_sm};
}

template <int W, typename OT, int DEPTH, int WK>
TraverseKernel traverse_t(bool has_sssp) {
  // wider groups: a level's work outweighs its launches (see fused_loop)
  if constexpr (W > 4) return {nullptr, 0};
  else if (!has_sssp) return traverse_kernel<W, OT, DEPTH, kWeightNone, false>();
  else if constexpr (DEPTH == kDepthPlanes) {
    return {nullptr, 0};  // planes hold BFS depths only
  } else {
    return traverse_kernel<W, OT, DEPTH, WK, true>();
  }
}

template <int W, typename OT, int DEPTH, int WK>
Dispatch dispatch_of() {
  return {enqueue_level_t<W, OT, DEPTH, WK>, grids_t<W, OT, DEPTH, WK>, seed_t<W, OT>,
          traverse_t<W, OT, DEPTH, WK>};
}

template <int W, typename OT, int DEPTH>
Dispatch pick_wk(int wk) {
  switch (wk) {
    case kWeightU32: return dispatch_of<W, OT, DEPTH, kWeightU32>();
    case kWeightF32: return dispatch_of<W, OT, DEPTH, kWeightF32>();
    default: return dispatch_of<W, OT, DEPTH, kWeightNone>();
  }
}

}  // namespace

template <int W, typename OT>
Dispatch pick_depth(int depth, int wk) {
  return depth == kDepthPlanes ? pick_wk<W, OT, kDepthPlanes>(wk) : pick_wk<W, OT, kDepthDirect>(wk);
}

}  // namespace cgp
