/*
 * swehr_wide_f32.cu -- the mixed kernels of runs whose divisors may be subnormal
 * (DevParams::mixed_ok == 0: no film or one below 2^-40, constants of extreme
 * size).  4096^2 in ponded flow without a film: 1.66 ms a step in the ordinary
 * kernels, whose quotients by such divisors were infinite, 2.38 here.
 */
#include "swehr_launch.cuh"

namespace swehr {

WideKernels wide_kernels_f32() { return FormLauncher<PolicyF32, float>::wide_kernels(); }

}  // namespace swehr
