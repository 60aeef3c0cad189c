// bitmap_planes_join.cu - the plane kernels of dimensions of 1 and 2 bytes behind a foreign key: see bitmap_planes.cuh.
#include "bitmap_planes.cuh"

namespace mb {
mb_status planes_join(const PlanePass &P) {
  return P.src->width == 1 ? launch_planes_fine<4, true, 1>(P) : launch_planes_fine<4, true, 2>(P);
}
}  // namespace mb
