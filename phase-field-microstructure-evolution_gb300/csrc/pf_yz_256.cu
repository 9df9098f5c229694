// yz-pass instantiations: 256 x 256 planes, clusters of 8 CTAs (70 KB of shared
// memory each, three per SM), z = t + 8 s with one t per CTA.  Yz pass of 33
// fields 3334 -> 2584 us against clusters that re-lay the plane out.  s in one
// pass of 2 (with y) and one of 16; runs of 16 (2 x 8, two t per CTA) were 4 %
// slower, clusters of 16 x 128 threads 3 %, 128 threads 3 %, two CTAs per SM 3 %.
#include "pf_internal.h"

namespace pf {

int yz_variants_256(int ny, int nz, YZKernels* out, int n) {
  if (ny == 256 && nz == 256) n = add_yz<256, 256, 8, 256, true, 1, 2, 16, 3>(out, n);
  return n;
}

}  // namespace pf
