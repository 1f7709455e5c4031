/*
 * swehr_wide16_f64.cu -- the kernels of swehr_wide_f64.cu for the pool's 16 x 16-
 * cell tiles.
 */
#define SWEHR_TILE_I 16
#define SWEHR_TILE_J 16
#define SWEHR_TILE_NS t16x16
#include "swehr_launch.cuh"

namespace swehr {

WideKernels wide_kernels_f64_t16() { return FormLauncher<PolicyF64, double>::wide_kernels(); }

}  // namespace swehr
