// resident_grid_f64_lanes.cu -- the resident grid's kernels (resident_grid.cuh) of
// one precision form, compiled and loaded by themselves.
#include "resident_grid.cuh"

namespace tg {

const void *grid_kernel_f64_lanes(int integ, int stage, int shape) { return rg_kernel<P_FP64, true>(integ, stage, shape); }

}  // namespace tg
