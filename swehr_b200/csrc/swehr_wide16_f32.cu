/*
 * swehr_wide16_f32.cu -- the kernels of swehr_wide_f32.cu for the pool's 16 x 16-
 * cell tiles.
 */
#define SWEHR_TILE_I 16
#define SWEHR_TILE_J 16
#define SWEHR_TILE_NS t16x16
#include "swehr_launch.cuh"

namespace swehr {

WideKernels wide_kernels_f32_t16() { return FormLauncher<PolicyF32, float>::wide_kernels(); }

}  // namespace swehr
