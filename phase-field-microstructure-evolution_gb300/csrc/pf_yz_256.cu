// yz-pass instantiations: 256 x 256 planes, clusters of 4 CTAs that exchange
// the plane's layouts in place (140 KB of shared memory per CTA).
#include "pf_internal.h"

namespace pf {

int yz_variants_256(int ny, int nz, YZKernels* out, int n) {
  if (ny == 256 && nz == 256) n = add_yz<256, 256, 4, 512>(out, n);
  return n;
}

}  // namespace pf
