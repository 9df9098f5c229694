// Instantiations of the x pass for the rest of the reference's weak-scaling
// grids (inputs/config.yaml:71-106): 80, 160 and 200 (x lines of M = Nx/2 =
// 40, 80, 100 complex points, plans 8 x 5, 16 x 5, 10 x 10) and 102 (M = 51,
// plan 3 x 17).  The first variant that fits is the default; the autotuner
// picks among them.
#include "pf_internal.h"

namespace pf {

int x_variants_r5(int nx, XKernels* out, int n) {
  switch (nx) {
    case 80:
      n = add_x<80, 16, 256, 3>(out, n, ",3/SM");
      n = add_x<80, 8, 256>(out, n);
      n = add_x<80, 4, 256>(out, n);
      break;
    case 160:
      n = add_x<160, 16, 256, 2>(out, n, ",2/SM");
      n = add_x<160, 16, 512>(out, n);
      n = add_x<160, 8, 512>(out, n);
      n = add_x<160, 4, 256>(out, n);
      break;
    case 200:  // 10 warps: one to each column of the 10 x 10 lines (x pass of 17 fields 495 us with 8 or 16 warps, 429)
      n = add_x<200, 8, 320, 2>(out, n, ",2/SM");
      n = add_x<200, 8, 256, 3>(out, n, ",3/SM");
      n = add_x<200, 4, 320>(out, n);
      n = add_x<200, 2, 256>(out, n);
      break;
    case 102:  // 6 warps: two to each column of the 3 x 17 lines (5 fields 30.8 -> 26.7 us)
      n = add_x<102, 6, 192, 3>(out, n, ",3/SM");
      n = add_x<102, 17, 192, 3>(out, n, ",3/SM");
      n = add_x<102, 3, 256>(out, n);
      n = add_x<102, 2, 256>(out, n);
      break;
    default: break;
  }
  return n;
}

}  // namespace pf
