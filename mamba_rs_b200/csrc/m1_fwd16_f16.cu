// Instantiates the selective-scan forward by warp roles for f16 storage.
#include "m1_fwd16_kernel.cuh"

namespace mb200 {
void fwd16_f16(Fwd16Table* t) { build_fwd16<__half>(t); }
}  // namespace mb200
