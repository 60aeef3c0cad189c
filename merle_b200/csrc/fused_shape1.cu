// fused_shape1.cu - the fused kernels of op shape 1 (query template 1): see
// fused_warp.cuh and shape.cuh.  One file per shape, so that they compile side by side.
#include "fused_warp.cuh"

namespace mb {
mb_status fused_shape1(const DevPrg &P, const ShapeArgs &A, const ShapeLaunch &L) {
  return fused_shape_launch<0>(P, A, L);
}
}  // namespace mb
