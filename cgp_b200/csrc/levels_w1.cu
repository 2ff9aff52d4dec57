// Level kernels of groups with 1 mask word (64 slots), 32-bit offsets.
#include "levels.cuh"

namespace cgp {

template Dispatch pick_depth<1, int32_t>(int depth, int wk);

}  // namespace cgp
