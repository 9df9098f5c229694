// Host-side declarations shared by the kernel translation units and the API.
#pragma once
#include <cuda_runtime.h>

#include <string>

#include "pf_kernels.cuh"

namespace pf {

typedef void (*KernelFn)(const RunParams*, const Shape);

// One compiled variant of the x pass (all modes) ...
struct XKernels {
  KernelFn bulk, xj, imp, exp, fields;
  int wy;           // y rows per CTA
  int threads;      // threads per CTA
  const char* tag;  // how the tile is loaded and walked and the CTAs per SM asked for, for reports
};

// ... and of the yz pass (all three modes).
struct YZKernels {
  KernelFn main, c2, imp;  // modes YZ_MAIN, YZ_C2, YZ_IMPORT
  int cluster;   // CTAs per plane
  int threads;   // threads per CTA
  size_t smem;   // dynamic shared memory per CTA
};

// Variant lists: each translation unit appends the variants it compiled for a
// shape to `out` (room for kMaxVariants entries) and returns the new count.  The first variant of a shape is its
// default; the run-creation autotuner times the others.
constexpr int kMaxVariants = 8;
int x_variants_a(int nx, XKernels* out, int n);
int x_variants_r5(int nx, XKernels* out, int n);
int yz_variants_small(int ny, int nz, YZKernels* out, int n);
int yz_variants_128(int ny, int nz, YZKernels* out, int n);
int yz_variants_256(int ny, int nz, YZKernels* out, int n);
int yz_variants_r5(int ny, int nz, YZKernels* out, int n);

// An x-pass variant: WY rows and T threads per CTA, at least MINB CTAs per SM
// (0: as many registers as the compiler likes).  ASYNC: the tile's spectra
// copied in by cp.async and transformed in place.
template <int NX, int WY, int T, int MINB = 0, bool ASYNC = false>
static int add_x(XKernels* out, int n, const char* tag = "") {
  if (n >= kMaxVariants) return n;
  XKernels& k = out[n];
  k.bulk = x_pass_kernel<NX, WY, T, MODE_BULK, ASYNC, MINB>;
  k.xj = x_pass_kernel<NX, WY, T, MODE_XJ, ASYNC>;
  k.imp = x_pass_kernel<NX, WY, T, MODE_IMPORT>;
  k.exp = x_pass_kernel<NX, WY, T, MODE_EXPORT, ASYNC>;
  k.fields = x_pass_kernel<NX, WY, T, MODE_FIELDS, ASYNC>;
  k.wy = WY;
  k.threads = T;
  k.tag = tag;
  return n + 1;
}

// A yz-pass variant with one CTA of T threads per plane (RAWP: unpadded row
// pitch), at least MINB CTAs per SM, k-space values read UC at a time.
template <int NY, int NZ, int T, bool RAWP, int MINB = 0, int UC = Line<NZ>::N1>
static int add_yz1(YZKernels* out, int n) {
  if (n >= kMaxVariants) return n;
  YZKernels& k = out[n];
  k.main = yz1_kernel<NY, NZ, T, YZ_MAIN, RAWP, MINB, UC>;
  k.c2 = yz1_kernel<NY, NZ, T, YZ_C2, RAWP, MINB, UC>;
  k.imp = yz1_kernel<NY, NZ, T, YZ_IMPORT, RAWP, MINB, UC>;
  k.cluster = 1;
  k.threads = T;
  k.smem = YZ1<NY, NZ, RAWP>::SMEM;
  return n + 1;
}

// ... and with C CTAs per plane, ZA, ZB and ZP points of z in the first three passes.
template <int NY, int NZ, int C, int T, bool RAWP, int ZA, int ZB, int ZP = 1, int MINB = 0, int UC = 0>
static int add_yz(YZKernels* out, int n) {
  if (n >= kMaxVariants) return n;
  YZKernels& k = out[n];
  k.main = yz_kernel<NY, NZ, C, T, YZ_MAIN, RAWP, ZA, ZB, ZP, MINB, UC>;
  k.c2 = yz_kernel<NY, NZ, C, T, YZ_C2, RAWP, ZA, ZB, ZP, MINB, UC>;
  k.imp = yz_kernel<NY, NZ, C, T, YZ_IMPORT, RAWP, ZA, ZB, ZP, MINB, UC>;
  k.cluster = C;
  k.threads = T;
  k.smem = YZ<NY, NZ, C, RAWP, ZA, ZB, ZP>::SMEM;
  return n + 1;
}

inline int get_x_variants(int nx, XKernels* out) { return x_variants_r5(nx, out, x_variants_a(nx, out, 0)); }
inline int get_yz_variants(int ny, int nz, YZKernels* out) {
  int n = 0;
  n = yz_variants_small(ny, nz, out, n);
  n = yz_variants_128(ny, nz, out, n);
  n = yz_variants_256(ny, nz, out, n);
  n = yz_variants_r5(ny, nz, out, n);
  return n;
}
// default (first) variant of a shape; `out` receives one entry
inline bool get_x_kernels(int nx, XKernels* out) {
  XKernels v[kMaxVariants];
  if (get_x_variants(nx, v) == 0) return false;
  *out = v[0];
  return true;
}
inline bool get_yz_kernels(int ny, int nz, YZKernels* out) {
  YZKernels v[kMaxVariants];
  if (get_yz_variants(ny, nz, v) == 0) return false;
  *out = v[0];
  return true;
}

void set_error(const std::string& msg);
// ... of a call that failed in CUDA: the runtime's last error has been reported
// with it and is not to be taken for the next call's.
void set_cuda_error(const std::string& msg);

// Let kernel `fn` use `bytes` of dynamic shared memory on the current device;
// false if it cannot.  The limit is the process's, so it is only ever raised.
bool raise_smem(const void* fn, size_t bytes);

}  // namespace pf
