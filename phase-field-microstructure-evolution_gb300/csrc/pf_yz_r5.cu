// yz-pass instantiations for the rest of the reference's weak-scaling grids:
// 80^2, 160^2, 200^2 planes (lines of 16 x 5, 16 x 10 and 20 x 10) and 102^2
// (lines of 6 x 17).  80^2 and 102^2 planes have one CTA each (54 and 97 KB);
// 160^2 and 200^2 are shared by clusters of 4 and 5 (54 and 67 KB), whose thread
// count is a multiple of the y run and of the warp size.
#include "pf_internal.h"

namespace pf {

int yz_variants_r5(int ny, int nz, YZKernels* out, int n) {
  // 80^2: yz pass of 13 fields 26.5 -> 24.9 us (160 threads), of 51 fields 95 -> 90 us (256; 94 with 160)
  // against one transform stage a pass
  if (ny == 80 && nz == 80) {
    n = add_yz<80, 80, 1, 256, true, 5, 2, 1, 3>(out, n);
    n = add_yz<80, 80, 1, 160, true, 1, 1, 10, 4>(out, n);
  }
  // 160^2: 21 fields 385 -> 350 us, 7 fields 138 -> 127 us against one CTA per plane (200 KB, 512 threads);
  // clusters of two (320 threads) 1 to 3 % slower than of four
  if (ny == 160 && nz == 160) n = add_yz<160, 160, 4, 160, true, 1, 1, 20, 4>(out, n);
  // 102^2: two CTAs per SM (72 registers), yz pass of 13 fields 104.7 -> 84.0 us; 256 threads for few fields (5:
  // 33.5 -> 30.8 us).  Stages of both axes in one pass (z as 2 x 3 x 17): 3 to 9 % slower
  if (ny == 102 && nz == 102) {
    n = add_yz1<102, 102, 448, false, 2>(out, n);
    n = add_yz1<102, 102, 256, false>(out, n);
  }
  // 200^2: yz pass of 7 fields 433 -> 302 us, of 17 882 -> 694 us against clusters that re-lay the plane out.
  // s as 20 in one pass; 2 x 10 (with y) 3 % slower, 224 to 416 threads 2 to 9 %, clusters of ten 0 to 3 %
  if (ny == 200 && nz == 200) n = add_yz<200, 200, 5, 160, true, 1, 1, 20, 3>(out, n);
  return n;
}

}  // namespace pf
