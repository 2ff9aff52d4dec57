// Level kernels of groups with 16 mask words (1024 slots), 32-bit offsets.
#include "levels.cuh"

namespace cgp {

template Dispatch pick_depth<16, int32_t>(int depth, int wk);

}  // namespace cgp
