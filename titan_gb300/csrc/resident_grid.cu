// resident_grid.cu -- launches of the resident grid (resident_grid.cuh).  Its
// kernels are compiled in a file per precision form, so that a process loads
// only those it uses (all of them in one file took 16 ms of a first launch)
// and the build compiles them side by side.
#include "resident_grid.cuh"

namespace tg {

const void *grid_kernel_f64(int integ, int stage, int shape);
const void *grid_kernel_f64_lanes(int integ, int stage, int shape);
const void *grid_kernel_f32(int integ, int stage, int shape);
const void *grid_kernel_f32c(int integ, int stage, int shape);

namespace {

// max_nm: the largest tile's masses.  A lane per component serves FP64 tiles
// of at most kLaneWarps warps of masses (20^3 lattice, 53 masses: 12.5 us per
// step against 12.9; 24^3, 91 masses: equal, with spills against none)
const void *grid_kernel(int precision, int integ, int stage, int shape, int max_nm) {
    if (precision == P_FP64)
        return grid_resident_lanes(precision, shape, max_nm) ? grid_kernel_f64_lanes(integ, stage, shape)
                                                             : grid_kernel_f64(integ, stage, shape);
    return precision == P_FP32 ? grid_kernel_f32(integ, stage, shape) : grid_kernel_f32c(integ, stage, shape);
}

}  // namespace

size_t grid_resident_smem_bytes(int precision, const TileInfo &ti, int stage) {
    return (size_t)rg_layout(precision, ti, stage).total;
}
int grid_resident_threads(int shape) { return kShapes[shape].threads; }
int grid_resident_exchange_bytes(int precision) { return precision == P_FP32 ? 32 : 64; }

int grid_resident_ctas(int shape) { return kShapes[shape].ctas; }
bool grid_resident_lanes(int precision, int shape, int max_nm) {
    const int warps = kShapes[shape].threads / 32;
    return precision == P_FP64 && max_nm <= kLaneMasses * (warps < kLaneWarps ? warps : kLaneWarps);
}

cudaError_t grid_resident_prepare(int precision, int integ, const GridResArgs &r, int shape, size_t smem, int *ctas_per_sm) {
    const void *f = grid_kernel(precision, integ, r.stage, shape, r.max_nm);
    const cudaError_t e = raise_smem_limit(f, smem);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas_per_sm, f, kShapes[shape].threads, smem);
}

cudaError_t launch_grid_resident(int precision, int integ, const StepArgs &a, const GridResArgs &r, int shape,
                                 size_t smem, int parity, int64_t nsteps, int write_acc, cudaStream_t s) {
    const void *f = grid_kernel(precision, integ, r.stage, shape, r.max_nm);
    const cudaError_t e = raise_smem_limit(f, smem);
    if (e != cudaSuccess) return e;
    int64_t passes = nsteps * (integ == INTEG_RK2 ? 2 : 1);
    void *args[] = {const_cast<StepArgs *>(&a), const_cast<GridResArgs *>(&r), &parity, &passes, &write_acc};
    return cudaLaunchCooperativeKernel(f, dim3(r.ntiles), dim3(kShapes[shape].threads), args, smem, s);
}

cudaError_t launch_grid_single(int precision, int integ, const StepArgs &a, const GridResArgs &r, int shape,
                               size_t smem, int parity, int half, int write_acc, cudaStream_t s, bool programmatic) {
    if (precision == P_FP64) return cudaErrorInvalidValue;
    const void *f = grid_kernel(precision, integ, r.stage, shape, r.max_nm);
    const cudaError_t e = raise_smem_limit(f, smem);
    if (e != cudaSuccess) return e;
    GridResArgs one = r;
    one.half = half;
    one.single = 1;
    int64_t passes = 1;
    void *args[] = {const_cast<StepArgs *>(&a), &one, &parity, &passes, &write_acc};
    return launch_programmatic(f, dim3(r.ntiles), dim3(kShapes[shape].threads), args, smem, s, programmatic);
}

}  // namespace tg
