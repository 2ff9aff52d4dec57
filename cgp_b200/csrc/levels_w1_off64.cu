// Level kernels of groups with 1 mask word (64 slots), 64-bit offsets.
#include "levels.cuh"

namespace cgp {

template Dispatch pick_depth<1, int64_t>(int depth, int wk);

}  // namespace cgp
