// yz-pass instantiations: 128 x 128 planes, one CTA per plane (136 KB of
// shared memory, no re-layout).
#include "pf_internal.h"

namespace pf {

int yz_variants_128(int ny, int nz, YZKernels* out, int n) {
  if (ny == 128 && nz == 128) n = add_yz1<128, 128, 512, true>(out, n);
  return n;
}

}  // namespace pf
