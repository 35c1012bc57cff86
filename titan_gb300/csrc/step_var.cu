// step_var.cu -- register-capped launch-bound variants of the per-tile step
// kernel (a separate translation unit so that the build compiles them in
// parallel with step.cu).  FP32 forms, Euler integrator:
//   variant 1: __launch_bounds__(256, 3)  <= 85 registers per thread
//   variant 2: __launch_bounds__(256, 4)  <= 64 registers per thread
// FP64, every integrator, where more than two CTAs per SM are needed:
//   variant 3: __launch_bounds__(256, 3).  A step is bound by the FP64 pipe
//   in the mass phase and by the integer units in the entry phase (about 60 %
//   and 45 % busy), and three CTAs at different phases share them better than
//   one: 80^3 lattice 496 us per step with 256-mass tiles and one 512-thread
//   CTA per SM, 449 with 96-mass tiles and three of 256 threads (80
//   registers, 54 bytes of spills); four of 192 threads 478, two of 384 also
//   478.
#include "step_kernel.cuh"

namespace tg {

const void *step_kernel_capped(int precision, int variant, int integ) {
    if (precision == P_FP32) {
        if (variant == 1) return (const void *)k_step<P_FP32, 256, 3, INTEG_EULER>;
        if (variant == 2) return (const void *)k_step<P_FP32, 256, 4, INTEG_EULER>;
    } else if (precision == P_FP32C) {
        if (variant == 1) return (const void *)k_step<P_FP32C, 256, 3, INTEG_EULER>;
        if (variant == 2) return (const void *)k_step<P_FP32C, 256, 4, INTEG_EULER>;
    } else if (variant == 3) {
        if (integ == INTEG_VERLET) return (const void *)k_step<P_FP64, 256, 3, INTEG_VERLET>;
        if (integ == INTEG_RK2) return (const void *)k_step<P_FP64, 256, 3, INTEG_RK2>;
        return (const void *)k_step<P_FP64, 256, 3, INTEG_EULER>;
    }
    return nullptr;
}

}  // namespace tg
