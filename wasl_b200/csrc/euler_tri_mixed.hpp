// The mixed form's kernels by polynomial order and volume rule: one explicit
// instantiation per object (euler_tri_mixed_kernels.cu compiled with WASL_P and
// WASL_R), dispatched by euler_tri_mixed.cu.
#pragma once

#include <cstddef>

#include <cuda_runtime.h>

#include "kernels.hpp"

namespace wasl_b200 {

// Launch shapes of the tile kernels (elements per CTA, register budget):
//   0: 128 elements, <= 128 registers (4 CTAs / 16 warps per SM)
//   1: 128 elements, no register cap
//   2: 256 elements, <= 128 registers (2 CTAs per SM)
//   3:  64 elements, <= 128 registers (8 CTAs per SM)
// and of the shared-face tile kernel:
//   4:  64 elements, sized for 7 CTAs per SM (14 warps)
//   5:  96 elements, sized for 5 CTAs per SM (15 warps)
//   6: 128 elements, sized for 4 CTAs per SM (16 warps)
//   7: 128 elements, sized for 3 CTAs per SM
// and of the patch kernel:
//   8: 256 elements, <= 128 registers (2 CTAs per SM)
//   9: 128 elements, sized for 5 CTAs per SM
//  10:  64 elements, sized for 8 CTAs per SM
//  11: 192 elements, sized for 3 CTAs per SM
// (larger patches have fewer faces to outside elements, which both patches
// evaluate: P3 at 500,000 triangles 341 us a stage in shape 8 against 371 with
// 128 elements at the same registers (310 with the point loops rolled), at 45,602 triangles 37 us in shape 11
// against 45; 64 elements suit meshes that larger patches leave SMs idle on)
// and of the patch kernel with its volume term on the tensor cores:
//  12: 128 elements, <= 128 registers
//  13: 128 elements, sized for 5 CTAs per SM
// and of the persistent tile kernel (one wave of resident CTAs looping over
// the tiles of the mesh or of the batch's work list):
//  14: 128 elements, <= 128 registers
//  15: 256 elements, <= 128 registers
constexpr int kTileShapes = kTileShapeCount;
constexpr int kTileElements[kTileShapes] = {128, 128, 256, 64, 64, 96, 128, 128,
                                            256, 128, 64, 192, 128, 128, 128, 256};
constexpr int kFirstPatchShape = 8, kPatchShapeEnd = 14;

// R: the volume rule's order, or 0 for the symmetric rule.
template <int P, int R> struct MixedForm {
  static void upload();
  static void stage(const StageArgs &a, cudaStream_t s);
  static void stage_tile(int shape, const StageArgs &a, cudaStream_t s);
  static void prepare_tile();
  static std::size_t face_record_bytes();
};

extern template struct MixedForm<1, 0>;
extern template struct MixedForm<1, 1>;
extern template struct MixedForm<1, 2>;
extern template struct MixedForm<1, 3>;
extern template struct MixedForm<2, 0>;
extern template struct MixedForm<2, 2>;
extern template struct MixedForm<2, 3>;
extern template struct MixedForm<2, 4>;
extern template struct MixedForm<3, 0>;
extern template struct MixedForm<3, 3>;
extern template struct MixedForm<3, 4>;
extern template struct MixedForm<3, 5>;

} // namespace wasl_b200
