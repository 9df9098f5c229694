// yz-pass instantiations for the rest of the reference's weak-scaling grids:
// 80^2, 160^2, 200^2 planes (lines of 16 x 5, 16 x 10 and 20 x 10) and 102^2
// (lines of 6 x 17).  80^2, 102^2 and 160^2 planes fit one CTA (54, 97 and
// 218 KB); 200^2 planes are shared by clusters of 5 CTAs (71 KB each), whose
// thread count is a multiple of both run lengths of a line and of the warp
// size.
#include "pf_internal.h"

namespace pf {

int yz_variants_r5(int ny, int nz, YZKernels* out, int n) {
  // 80^2: 64 registers, four CTAs per SM, k-space values four at a time: yz pass of 13 fields 29.0 -> 26.5 us
  if (ny == 80 && nz == 80) n = add_yz1<80, 80, 256, true, 4, 4>(out, n);
  if (ny == 160 && nz == 160) n = add_yz1<160, 160, 512, true>(out, n);
  if (ny == 102 && nz == 102) {  // two CTAs per SM (72 registers): yz pass of 13 fields 104.7 -> 84.0 us
    n = add_yz1<102, 102, 448, false, 2>(out, n);
    n = add_yz1<102, 102, 256, false>(out, n);
  }
  // two clusters' CTAs per SM, one buffer each and k-space values ten at a time: yz pass of 7 fields
  // 614 -> 432 us against separate A and B buffers (135 KB, one CTA per SM); clusters of 2 x 800
  // threads and of 10 x 160 were 2 to 5 % slower
  if (ny == 200 && nz == 200) n = add_yz<200, 200, 5, 320, 2, 10>(out, n);
  return n;
}

}  // namespace pf
