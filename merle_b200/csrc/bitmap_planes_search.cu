// bitmap_planes_search.cu - the plane kernels of one level over a wide domain: see bitmap_planes.cuh.
#include "bitmap_planes.cuh"

namespace mb {
mb_status planes_search(const PlanePass &P) {
  if (!P.src->fk) {
    switch (P.src->width) {
    case 1: return launch_planes_k<1, false, 1, BP_SEARCH, true, 0>(P);
    case 2: return launch_planes_k<2, false, 1, BP_SEARCH, true, 0>(P);
    case 4: return launch_planes_k<4, false, 1, BP_SEARCH, true, 0>(P);
    default: return launch_planes_k<8, false, 1, BP_SEARCH, true, 0>(P);
    }
  }
  switch (P.src->width) {  // the column read by row is the 4-byte key; width is the dimension's
  case 1: return launch_planes_k<4, true, 1, BP_SEARCH, true, 0>(P);
  case 2: return launch_planes_k<4, true, 2, BP_SEARCH, true, 0>(P);
  case 4: return launch_planes_k<4, true, 4, BP_SEARCH, true, 0>(P);
  default: return launch_planes_k<4, true, 8, BP_SEARCH, true, 0>(P);
  }
}
}  // namespace mb
