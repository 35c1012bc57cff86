// resident_grid_f32.cu -- the resident grid's kernels (resident_grid.cuh) of
// one precision form, compiled and loaded by themselves.
#include "resident_grid.cuh"

namespace tg {

const void *grid_kernel_f32(int integ, int stage, int shape) { return rg_kernel<P_FP32, false>(integ, stage, shape); }

}  // namespace tg
