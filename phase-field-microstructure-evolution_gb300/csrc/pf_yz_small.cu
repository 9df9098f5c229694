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
  // 64^2, 96^2: stages of both axes in one pass.  Against one stage a pass: 64 runs of 64^3 x 8 509 -> 446 us
  // (128 threads, five CTAs per SM; 503 with 256 threads), a 64^3 x 4 step 20.0 -> 18.5 us (256 threads; 19.8
  // with 128), 96^3 x 55 207 -> 198 us.  At 32^2 both take the same time.
  if (ny == 64 && nz == 64) {
    n = add_yz<64, 64, 1, 256, true, 2, 4>(out, n);
    n = add_yz<64, 64, 1, 128, true, 4, 2, 1, 5>(out, n);
  }
  if (ny == 96 && nz == 96) n = add_yz<96, 96, 1, 256, true, 3, 4, 1, 2>(out, n);  // the reference's own grid
  return n;
}

}  // namespace pf
