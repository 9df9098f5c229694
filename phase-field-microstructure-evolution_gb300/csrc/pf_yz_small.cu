// yz-pass instantiations: planes up to 96 x 96, one CTA per plane.
#include "pf_internal.h"

namespace pf {

int yz_variants_small(int ny, int nz, YZKernels* out, int n) {
  if (ny == 16 && nz == 16) n = add_yz1<16, 16, 128, false>(out, n);
  if (ny == 32 && nz == 32) n = add_yz1<32, 32, 128, false>(out, n);
  if (ny == 16 && nz == 32) n = add_yz1<16, 32, 256, false>(out, n);
  if (ny == 32 && nz == 16) n = add_yz1<32, 16, 256, false>(out, n);
  if (ny == 32 && nz == 64) n = add_yz1<32, 64, 256, false>(out, n);
  if (ny == 64 && nz == 32) n = add_yz1<64, 32, 256, false>(out, n);
  if (ny == 64 && nz == 64) n = add_yz1<64, 64, 256, true>(out, n);
  if (ny == 96 && nz == 96) {  // the reference's own grid (inputs/config.yaml, inputs/input.txt)
    n = add_yz1<96, 96, 384, true, 2>(out, n);
    n = add_yz1<96, 96, 256, true, 2>(out, n);
  }
  return n;
}

}  // namespace pf
