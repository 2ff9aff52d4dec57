// Launch layer of one traversal level: what a level's launches need, and the
// per-mask-width entry points (each levels_w*.cu instantiates the kernels of
// one width and offset type, so that they compile side by side).
#pragma once

#include "engine.h"

namespace cgp {

using dev::DevGraph;
using dev::GroupDev;

struct Grids {
  int tile;   // tile kernels (grid-stride)
  int heavy;
  int clear;
  int dense;
  int dense2;
  int gather;
  int gather_heavy;
  int gather_vec;
  int gather_heavy_vec;
  int gather_rows;
  int gather_heavy_vec2;
  int bfs_chunked;
  int bfs_mid;
};

struct LevelLaunch {
  GroupDev g{};
  DevGraph G;
  Grids gr;
  bool has_bfs;
  bool has_sssp;
  bool pull;
  bool bounds = false;  // gather levels may screen by bounds
  bool spull;        // SSSP gather kernels are part of the level
  bool gvec;         // rows allow the vectorised gather (alignment, width)
  bool lchunks;      // light vertices gathered by items (in 4-word slices above W = 4)
  int dense_unroll;  // edges per step of the SSSP list kernel (1: 4, 2: 8)
  KernelTimer* kt;   // per-class event timing (non-graph runs only)
  bool heavy_push = false;                // heavy-queue push kernels are part of a level
  bool bfs_chunked = false;               // chunked light-vertex BFS pull is part of a pull level
  bool chunk_dir = false;                 // census of per-chunk frontier edges
  bool device_loop = false;               // level end sets a WHILE node's condition
  cudaGraphConditionalHandle loop = 0;    // ... this one
  int32_t level_cap = 0;                  // ... and stops at this many levels
};

using EnqueueFn = int (*)(const LevelLaunch&, cudaStream_t);
using GridsFn = Grids (*)(int);
using SeedFn = void (*)(const GroupDev&, const DevGraph&, cudaStream_t);


// The fused level loop (of BFS groups or of groups with SSSP slots), and how many of its blocks an SM
// holds (0: not available).
struct TraverseKernel {
  const void* fn;
  int per_sm;
};
using TraverseFn = TraverseKernel (*)(bool has_sssp);

struct Dispatch {
  EnqueueFn enqueue;
  GridsFn grids;
  SeedFn seed;
  TraverseFn traverse;
};

// Entry points for mask width W (1, 2, 4, 8, 16), offset type OT (int32_t or
// int64_t), depth mode and weight kind; one levels_w*.cu per (W, OT).
template <int W, typename OT>
Dispatch pick_depth(int depth, int wk);

}  // namespace cgp
