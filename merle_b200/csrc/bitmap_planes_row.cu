// bitmap_planes_row.cu - the plane kernels of columns of 1, 2 and 4 bytes: see bitmap_planes.cuh.
#include "bitmap_planes.cuh"

namespace mb {
mb_status planes_row(int mode, const PlanePass &P) {
  switch (P.src->width) {
  case 1:
    return mode == BP_DIRECT ? launch_planes_k<1, false, 1, BP_DIRECT, true, 0>(P) : launch_planes_fine<1, false, 1>(P);
  case 2: return launch_planes_fine<2, false, 1>(P);
  default: return launch_planes_fine<4, false, 1>(P);
  }
}
}  // namespace mb
