// Instantiates the selective-scan forward by warp roles for bf16 storage.
#include "m1_fwd16_kernel.cuh"

namespace mb200 {
void fwd16_bf16(Fwd16Table* t) { build_fwd16<__nv_bfloat16>(t); }
}  // namespace mb200
