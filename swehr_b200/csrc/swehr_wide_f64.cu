/*
 * swehr_wide_f64.cu -- the FP64 kernels of runs whose constants the branch-free
 * sequences do not take (DevParams::fast_ok == 0: a bulk density above 2^50, a
 * stream-power fraction above 2^100 and the like): the plain operators
 * throughout, once (4096^2 in ponded flow with J = 2^101: 19.6 ms a step in the
 * ordinary kernels, which formed every cell both ways, 6.4 here).
 */
#include "swehr_launch.cuh"

namespace swehr {

WideKernels wide_kernels_f64() { return FormLauncher<PolicyF64, double>::wide_kernels(); }

}  // namespace swehr
