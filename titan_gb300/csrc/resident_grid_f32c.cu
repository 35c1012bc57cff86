// resident_grid_f32c.cu -- the resident grid's kernels (resident_grid.cuh) of
// one precision form, compiled and loaded by themselves.
#include "resident_grid.cuh"

namespace tg {

const void *grid_kernel_f32c(int integ, int stage, int shape) { return rg_kernel<P_FP32C, false>(integ, stage, shape); }

}  // namespace tg
