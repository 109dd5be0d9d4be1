// Instantiates the two-lane selective-scan backward kernels for bf16 storage.
#include "m1_bwd2_kernel.cuh"

namespace mb200 {
void bwd2_kernels_bf16(BwdKernelFn* fn, size_t* smem) { fill_bwd2<__nv_bfloat16>(fn, smem); }
}  // namespace mb200
