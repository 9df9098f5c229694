// yz-pass instantiations: 128 x 128 planes.  One CTA per plane has its SM to
// itself (136 KB); clusters of two (70 KB, three CTAs per SM) let the passes of
// several planes overlap: yz pass of 17 fields 144.7 -> 137.9 us, 56 fields 428
// -> 422 us, but 4 % slower at 2 fields and equal at 9, where the planes of one
// wave leave nothing to overlap.  The run-creation autotuner chooses.
#include "pf_internal.h"

namespace pf {

int yz_variants_128(int ny, int nz, YZKernels* out, int n) {
  if (ny == 128 && nz == 128) {
    n = add_yz1<128, 128, 512, true>(out, n);
    n = add_yz<128, 128, 2, 256, true, 1, 1, 16, 3>(out, n);
  }
  return n;
}

}  // namespace pf
