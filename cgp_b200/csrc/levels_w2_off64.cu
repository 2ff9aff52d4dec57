// Level kernels of groups with 2 mask words (128 slots), 64-bit offsets.
#include "levels.cuh"

namespace cgp {

template Dispatch pick_depth<2, int64_t>(int depth, int wk);

}  // namespace cgp
