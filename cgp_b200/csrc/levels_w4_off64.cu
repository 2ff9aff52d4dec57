// Level kernels of groups with 4 mask words (256 slots), 64-bit offsets.
#include "levels.cuh"

namespace cgp {

template Dispatch pick_depth<4, int64_t>(int depth, int wk);

}  // namespace cgp
