// Level kernels of groups with 8 mask words (512 slots), 32-bit offsets.
#include "levels.cuh"

namespace cgp {

template Dispatch pick_depth<8, int32_t>(int depth, int wk);

}  // namespace cgp
