// bitmap_planes_wide.cu - the plane kernels of 8-byte columns, and of dimensions of 4 and 8 bytes: see bitmap_planes.cuh.
#include "bitmap_planes.cuh"

namespace mb {
mb_status planes_wide(const PlanePass &P) {
  if (!P.src->fk) return launch_planes_fine<8, false, 1>(P);
  return P.src->width == 4 ? launch_planes_fine<4, true, 4>(P) : launch_planes_fine<4, true, 8>(P);
}
}  // namespace mb
