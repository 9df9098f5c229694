// yz-pass instantiations: 256 x 256 planes, clusters of 8 CTAs that exchange
// the plane's layouts in place (70 KB of shared memory per CTA, two CTAs per
// SM).  Yz pass of 33 fields 3334 us; clusters of 4 x 512 threads (140 KB, one
// CTA per SM) were 1 % slower, 8 x 512 7 %, 16 x 128 6 %.
#include "pf_internal.h"

namespace pf {

int yz_variants_256(int ny, int nz, YZKernels* out, int n) {
  if (ny == 256 && nz == 256) n = add_yz<256, 256, 8, 256>(out, n);
  return n;
}

}  // namespace pf
