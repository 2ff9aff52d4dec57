// Level kernels of groups with 8 mask words (512 slots), 64-bit offsets.
#include "levels.cuh"

namespace cgp {

template Dispatch pick_depth<8, int64_t>(int depth, int wk);

}  // namespace cgp
