// Instantiates the selective-scan forward by warp roles for f32 storage.
#include "m1_fwd16_kernel.cuh"

namespace mb200 {
void fwd16_f32(Fwd16Table* t) { build_fwd16<float>(t); }
}  // namespace mb200
