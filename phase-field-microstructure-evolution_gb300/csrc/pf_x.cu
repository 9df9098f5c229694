// Instantiations of the x pass (fused bulk kernel and x-direction transforms)
// for the supported Nx: a few (rows per CTA, threads per CTA, CTAs per SM)
// variants per size, each the fastest for some number of fields; the first
// one that fits is the default, the autotuner picks among them.
#include "pf_internal.h"

namespace pf {

int x_variants_a(int nx, XKernels* out, int n) {
  switch (nx) {
    case 16: n = add_x<16, 16, 256>(out, n); break;
    case 32: n = add_x<32, 4, 128>(out, n); n = add_x<32, 8, 256>(out, n); break;
    case 64:
      n = add_x<64, 16, 256, 3>(out, n, ",3/SM");
      n = add_x<64, 8, 256>(out, n);
      n = add_x<64, 16, 256, 4>(out, n, ",4/SM");
      n = add_x<64, 4, 128>(out, n);
      break;
    case 96:
      n = add_x<96, 8, 256>(out, n);
      n = add_x<96, 16, 256>(out, n);
      n = add_x<96, 8, 512>(out, n);
      n = add_x<96, 4, 256>(out, n);
      break;
    case 128:
      n = add_x<128, 8, 256, 0>(out, n);
      n = add_x<128, 8, 256, 3>(out, n, ",3/SM");
      n = add_x<128, 32, 256>(out, n);
      n = add_x<128, 4, 256, 0, true>(out, n, ",async");
      break;
    case 256:
      // as many rows as fit: a warp's access covers WY x 8 bytes of each field and kx (256^3, x pass,
      // 3 fields: 419 us at 4 rows, 278 at 8; 15 fields: 1058 and 907)
      n = add_x<256, 8, 256>(out, n);
      n = add_x<256, 16, 512>(out, n);
      n = add_x<256, 8, 512>(out, n);
      n = add_x<256, 4, 512, 0, true>(out, n, ",async");
      n = add_x<256, 2, 256, 0, true>(out, n, ",async");
      n = add_x<256, 1, 256>(out, n);  // one row per tile: up to 196 fields
      break;
    default: break;
  }
  return n;
}

}  // namespace pf
