// bitmap_planes_any_row.cu - the plane kernels of any levels of a column: see bitmap_planes.cuh.
#include "bitmap_planes.cuh"

namespace mb {
mb_status planes_any_row(int mode, const PlanePass &P) {
  switch (P.src->width) {
  case 1: return launch_planes_any<1, false, 1>(mode, P);
  case 2: return launch_planes_any<2, false, 1>(mode, P);
  case 4: return launch_planes_any<4, false, 1>(mode, P);
  default: return launch_planes_any<8, false, 1>(mode, P);
  }
}
}  // namespace mb
