// bitmap_planes_any_join.cu - the plane kernels of any levels of a dimension behind a foreign key: see bitmap_planes.cuh.
#include "bitmap_planes.cuh"

namespace mb {
mb_status planes_any_join(int mode, const PlanePass &P) {
  switch (P.src->width) {
  case 1: return launch_planes_any<4, true, 1>(mode, P);
  case 2: return launch_planes_any<4, true, 2>(mode, P);
  case 4: return launch_planes_any<4, true, 4>(mode, P);
  default: return launch_planes_any<4, true, 8>(mode, P);
  }
}
}  // namespace mb
