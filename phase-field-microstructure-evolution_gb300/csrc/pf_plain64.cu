// FP64 GPU path and the Fortran-signature shims f_trans_, inv_trans_, k_space_.
//
// The step of src/var_diff.f90:561-1050 in FP64 over global memory, with cuFFT
// for the transforms.  FP64 arithmetic is what bounds it (a GB300 SM retires
// about two FP64 operations a clock, and a transform of 100 x 100 x 90 cells
// needs 45 M of them), so it runs 2 var + 3 transforms a step (2 more with
// variable mobility) where the reference takes 7 var + 9:
//   * the gradient energy (:561-678) by Parseval from the spectra that the
//     update writes anyway, kept as partial sums for the next step's record,
//     instead of 4 transforms per field;
//   * phase 14 is linear, so phi - L dt dF/dphi is formed in real space and
//     transformed once (:1003-1024 transform phi and dF/dphi);
//   * the mobility correction is skipped where mob - D_mean is zero.
// The bulk terms use the two values of gamma (sigma_1, sigma_2) and are linear
// in var.  100 x 100 x 90, 6 order parameters, variable mobility:
// a pass of three steps takes 6.9 ms, 23.8 with the reference's transforms.
#include <cuda_runtime.h>
#include <cufft.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

#include "pf_internal.h"
#include "pf_plain64.h"

namespace pf {

static int fail64(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  if (code == PF_ECUDA || code == PF_ENOMEM) set_cuda_error(buf);
  else set_error(buf);
  return code;
}

#define P64_CUDA(call)                                                                                   \
  do {                                                                                                   \
    cudaError_t e_ = (call);                                                                             \
    if (e_ != cudaSuccess) return fail64(PF_ECUDA, "%s: %s (%s:%d)", #call, cudaGetErrorString(e_),      \
                                         __FILE__, __LINE__);                                            \
  } while (0)
#define P64_FFT(call)                                                                           \
  do {                                                                                          \
    cufftResult r_ = (call);                                                                    \
    if (r_ != CUFFT_SUCCESS) return fail64(PF_ECUDA, "%s: cufft error %d", #call, (int)r_);      \
  } while (0)

static const int NB = 608;  // blocks of the grid-stride reduction kernels: four for each of 152 SMs
static const int NT = 256;
static const int NREC = 256;  // steps whose records stay on the device
// Fields are transformed together as long as their spectra stay within this
// (half of the L2 cache: transform, update and inverse then hit L2); a larger
// grid goes field by field.
static const size_t kChunkBytes = (size_t)64 << 20;

enum P64Acc { PA_FINT = 0, PA_FETA, PA_FCH, PA_MASS, PA_CMIN, PA_CMAX, PA_PHIMIN, PA_PHIPMAX, PA_BAD, PA_COUNT };

struct Axes64 {
  const double* qx; const double* qy; const double* qz;     // q (for kf_sq, kf_4)
  const double* nx; const double* ny; const double* nz;     // Nyquist-zeroed q (kf / i)
  int Nx, Ny, Nz, Kx;
};

struct Plain64 {
  pf_config c;
  int device = 0;
  int Nx, Ny, Nz, Kx, V;
  int B = 1;                 // fields per batched transform
  bool var_mob = false;      // mob - D_mean can be non-zero
  bool have_fint = false;    // fint[cur] holds the gradient energy of the present fields
  int cur = 0;
  size_t ncell, nspec;
  char* mem = nullptr;       // all of the following, and one work area for all plans: they run in turn
  double* phi = nullptr;     // [V][ncell]
  double* con = nullptr;
  double* psi = nullptr;     // [V][ncell]: phi - L dt dF/dphi
  double* dfdc = nullptr;
  double* mob = nullptr;     // mobility (variable mobility only)
  double* work = nullptr;    // real flux (variable mobility only)
  cufftDoubleComplex* spec = nullptr;   // c_hat, mu_hat (, J_hat)
  cufftDoubleComplex* chunk = nullptr;  // B spectra; with set / get also the fields' transfer buffer
  double* dstage = nullptr;  // = chunk
  double* axes = nullptr;
  double* part = nullptr;    // [PA_COUNT][NB] of the bulk kernel
  double* fint = nullptr;    // [2][V + 1][NB]: gradient energy partials of this and the next fields
  double* rec = nullptr;     // [NREC][PA_COUNT]
  Axes64 ax;
  cufftHandle fwd = 0, inv = 0, fwdB = 0, invB = 0;  // one field, B fields
  cudaStream_t stream = nullptr;
  int steps = 0;
};

// k-space index of element i (at most 2^29 of them: 32-bit division)
__device__ __forceinline__ void kidx(size_t i, const Axes64& a, int& kx, int& ky, int& kz) {
  const unsigned j = (unsigned)i, r = j / (unsigned)a.Kx;
  kx = (int)(j - r * (unsigned)a.Kx);
  kz = (int)(r / (unsigned)a.Ny);
  ky = (int)(r - (unsigned)kz * (unsigned)a.Ny);
}

__device__ __forceinline__ double block_sum64(double v, double* sh) {
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int o = NT / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  const double r = sh[0];
  __syncthreads();
  return r;
}

// Weight times |kf|^2 of a k-point (src/var_diff.f90:561-678 by Parseval): the
// planes 0 < kx < Nx/2 stand for their conjugates too.
__device__ __forceinline__ double grad_weight(const Axes64& a, int kx, int ky, int kz) {
  const double gx = a.nx[kx], gy = a.ny[ky], gz = a.nz[kz];
  return (gx * gx + gy * gy + gz * gz) * ((kx == 0 || 2 * kx == a.Nx) ? 1.0 : 2.0);
}

// Gradient energy partials of one spectrum (unnormalised): coef sum w |kf|^2 |s|^2
__global__ void p64_fint(const cufftDoubleComplex* __restrict__ sp, Axes64 a, double coef, size_t n,
                         double* __restrict__ out) {
  __shared__ double sh[NT];
  double s = 0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    int kx, ky, kz;
    kidx(i, a, kx, ky, kz);
    const cufftDoubleComplex v = sp[i];
    s += grad_weight(a, kx, ky, kz) * (v.x * v.x + v.y * v.y);
  }
  s = block_sum64(s, sh);
  if (threadIdx.x == 0) out[blockIdx.x] = coef * s;
}

// phases 5-9 and the mobility of phase 10 (src/var_diff.f90:685-898);
// statistics and mass of the same fields.  psi_i = phi_i - L dt dF/dphi_i.
// With a_i = phi_i^2, S = sum over the matrix variants, Gamma_i = sigma_1
// (S - a_i) + sigma_2 a_P (matrix), sigma_2 S (precipitate).
__global__ void p64_bulk(const double* __restrict__ phi, const double* __restrict__ con, double* __restrict__ psi,
                         double* __restrict__ dfdc, double* __restrict__ mob, int V, size_t n, pf_config c, int c1mc,
                         double* __restrict__ part) {
  __shared__ double sh[NT];
  double feta = 0, fch = 0, mass = 0;
  double cmin = 1.0, cmax = 0.0, pmin = 1.0, ppmax = 0.0, bad = 0;
  const int P = V - 1;
  const double Ldt = c.mob_phi * c.t_step;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    double S = 0, num = 0, pairs = 0;
    for (int iv = 0; iv < P; ++iv) {
      const double f = phi[iv * n + i], a = f * f;
      pairs += a * S;
      S += a;
      num += a * a;
    }
    const double fP = phi[P * n + i], aP = fP * fP, cc = con[i];
    const double ssq = S + aP, den = num + aP * aP;
    // phase 5
    feta += -0.5 * ssq + 0.25 * den + c.sigma_1 * pairs + c.sigma_2 * S * aP;
    // phase 6
    const double rden = 1.0 / den;
    const double pm = num * rden, pp = 1.0 - pm;
    const double dm = cc - c.con_0_mat, dp = cc - c.con_0_ppt;
    const double fmat = c.am * dm * dm, fppt = c.ap * dp * dp;
    fch += pm * fmat + pp * fppt;
    dfdc[i] = 2.0 * (pm * c.am * dm + pp * c.ap * dp);
    // phases 7-9: dF = phi (phi^2 - 1 + 2 Gamma) + term4, its factors as ratios to
    // sum phi^4, whose square leaves the range of a double at |phi| = 1e-39
    const double t4 = 4.0 * (aP * aP * rden) * rden * (fmat - fppt);
    const double g0 = 2.0 * c.sigma_2 * aP - 1.0;
    for (int iv = 0; iv < P; ++iv) {
      const double f = phi[iv * n + i], a = f * f;
      const double d = f * (g0 + a * (1.0 + t4) + 2.0 * c.sigma_1 * (S - a));
      if (!isfinite(d)) bad += 1;
      psi[iv * n + i] = f - Ldt * d;
    }
    {
      const double d = fP * (aP - 1.0 + 2.0 * c.sigma_2 * S + 4.0 * (aP * rden) * pm * (fppt - fmat));
      if (!isfinite(d)) bad += 1;
      psi[P * n + i] = fP - Ldt * d;
    }
    if (mob) mob[i] = c1mc ? c.D_L * (1.0 + cc * (1.0 - cc)) : c.D_L + 2.0 * (1.0 - ssq) * c.D_gb;
    // statistics of these fields (src/var_diff.f90:1082-1096)
    mass += cc;
    cmin = fmin(cmin, cc);
    cmax = fmax(cmax, cc);
    pmin = fmin(pmin, ssq);
    ppmax = fmax(ppmax, fP);
  }
  const double q[4] = {feta, fch, mass, bad};
  const int at[4] = {PA_FETA, PA_FCH, PA_MASS, PA_BAD};
  for (int k = 0; k < 4; ++k) {
    const double v = block_sum64(q[k], sh);
    if (threadIdx.x == 0) part[at[k] * NB + blockIdx.x] = v;
  }
  __shared__ double sm[4][NT];
  sm[0][threadIdx.x] = cmin; sm[1][threadIdx.x] = cmax; sm[2][threadIdx.x] = pmin; sm[3][threadIdx.x] = ppmax;
  __syncthreads();
  for (int o = NT / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      sm[0][threadIdx.x] = fmin(sm[0][threadIdx.x], sm[0][threadIdx.x + o]);
      sm[1][threadIdx.x] = fmax(sm[1][threadIdx.x], sm[1][threadIdx.x + o]);
      sm[2][threadIdx.x] = fmin(sm[2][threadIdx.x], sm[2][threadIdx.x + o]);
      sm[3][threadIdx.x] = fmax(sm[3][threadIdx.x], sm[3][threadIdx.x + o]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[PA_CMIN * NB + blockIdx.x] = sm[0][0];
    part[PA_CMAX * NB + blockIdx.x] = sm[1][0];
    part[PA_PHIMIN * NB + blockIdx.x] = sm[2][0];
    part[PA_PHIPMAX * NB + blockIdx.x] = sm[3][0];
  }
}

// phase 11: J_hat = G mu_hat - kappa_c c_hat K3   (spectra unnormalised on input)
__global__ void p64_flux(const cufftDoubleComplex* __restrict__ ch, const cufftDoubleComplex* __restrict__ mu,
                         cufftDoubleComplex* __restrict__ out, Axes64 a, double kc, double scale, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    int kx, ky, kz;
    kidx(i, a, kx, ky, kz);
    const double g = a.nx[kx] + a.ny[ky] + a.nz[kz];
    const double k3 = -(a.nx[kx] * a.qx[kx] * a.qx[kx] + a.ny[ky] * a.qy[ky] * a.qy[ky] + a.nz[kz] * a.qz[kz] * a.qz[kz]);
    // i*g*mu - kc * c * i*k3 = i (g mu - kc k3 c)
    const double re = (g * mu[i].x - kc * k3 * ch[i].x) * scale;
    const double im = (g * mu[i].y - kc * k3 * ch[i].y) * scale;
    out[i] = make_cuDoubleComplex(-im, re);
  }
}

// phase 12 (real space): J *= (mob - D_mean)
__global__ void p64_jmob(double* __restrict__ J, const double* __restrict__ mob, double dmean, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    J[i] = J[i] * (mob[i] - dmean);
}

// phase 13: c_hat = (c_hat + J'_hat dt G + D K2 dt mu_hat) / (1 + D dt kappa_c K4),
// and the gradient energy partials of the new field (jp: null without the
// mobility correction)
__global__ void p64_ch(cufftDoubleComplex* __restrict__ ch, const cufftDoubleComplex* __restrict__ jp,
                       const cufftDoubleComplex* __restrict__ mu, Axes64 a, double dt, double dm, double kc,
                       double scale, double coef, size_t n, double* __restrict__ fint) {
  __shared__ double sh[NT];
  double s = 0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    int kx, ky, kz;
    kidx(i, a, kx, ky, kz);
    const double qx2 = a.qx[kx] * a.qx[kx], qy2 = a.qy[ky] * a.qy[ky], qz2 = a.qz[kz] * a.qz[kz];
    const double k2 = -(qx2 + qy2 + qz2);
    const double k4 = qx2 * qx2 + qy2 * qy2 + qz2 * qz2;
    const double r = scale / (1.0 + dm * dt * kc * k4);
    const double t33 = dm * k2 * dt;
    double re = ch[i].x + t33 * mu[i].x, im = ch[i].y + t33 * mu[i].y;
    if (jp) {  // J'_hat * dt * (i g)
      const double g = dt * (a.nx[kx] + a.ny[ky] + a.nz[kz]);
      re -= jp[i].y * g;
      im += jp[i].x * g;
    }
    re *= r;
    im *= r;
    ch[i] = make_cuDoubleComplex(re, im);
    s += grad_weight(a, kx, ky, kz) * (re * re + im * im);
  }
  s = block_sum64(s, sh);
  if (threadIdx.x == 0) fint[blockIdx.x] = coef * s;
}

// phase 14 of `nb` fields: phi_hat = psi_hat / (1 - L kappa dt K2), and the
// gradient energy partials of the new fields.  A thread takes one k-point of
// all of them: one division per point.
__global__ void p64_ac(cufftDoubleComplex* __restrict__ sp, Axes64 a, double Lkdt, double scale, double coef, size_t n,
                       int nb, double* __restrict__ fint) {
  __shared__ double sh[NT];
  double s = 0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    int kx, ky, kz;
    kidx(i, a, kx, ky, kz);
    const double q2 = a.qx[kx] * a.qx[kx] + a.qy[ky] * a.qy[ky] + a.qz[kz] * a.qz[kz];
    const double r = scale / (1.0 + Lkdt * q2);
    double e = 0;
    for (int b = 0; b < nb; ++b) {
      cufftDoubleComplex* p = sp + (size_t)b * n + i;
      const double re = p->x * r, im = p->y * r;
      *p = make_cuDoubleComplex(re, im);
      e += re * re + im * im;
    }
    s += grad_weight(a, kx, ky, kz) * e;
  }
  s = block_sum64(s, sh);
  if (threadIdx.x == 0) fint[blockIdx.x] = coef * s;
}

// The step's record: one block per quantity, sums in a fixed order.
__global__ void p64_finish(const double* __restrict__ part, const double* __restrict__ fint, int nfint,
                           double* __restrict__ out) {
  __shared__ double sh[NT];
  const int q = blockIdx.x;
  const bool mn = q == PA_CMIN || q == PA_PHIMIN, mx = q == PA_CMAX || q == PA_PHIPMAX;
  const double* src = q == PA_FINT ? fint : part + q * NB;
  const int n = q == PA_FINT ? nfint : NB;
  double v = mn ? 1.0 : 0.0;
  for (int b = threadIdx.x; b < n; b += NT) {
    const double x = src[b];
    v = mn ? fmin(v, x) : (mx ? fmax(v, x) : v + x);
  }
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int o = NT / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      const double x = sh[threadIdx.x + o], y = sh[threadIdx.x];
      sh[threadIdx.x] = mn ? fmin(y, x) : (mx ? fmax(y, x) : y + x);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) out[q] = sh[0];
}

__global__ void p64_aos_to_soa(const double* __restrict__ aos, double* __restrict__ soa, int V, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    for (int f = 0; f < V; ++f) soa[f * n + i] = aos[i * V + f];
}
__global__ void p64_soa_to_aos(const double* __restrict__ soa, double* __restrict__ aos, int V, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    for (int f = 0; f < V; ++f) aos[i * V + f] = soa[f * n + i];
}

static void host_axis(int n, int count, double* q, double* qn) {
  const double pi = std::atan(1.0) * 4.0;
  const double unit = 2.0 * pi / (double)n;
  for (int m = 0; m < count; ++m) {
    const int mp = (m <= n / 2) ? m : m - n;
    q[m] = (double)mp * unit;
    qn[m] = (2 * m == n) ? 0.0 : q[m];
  }
}

int plain64_validate(const pf_config* c) {
  if (!c) return fail64(PF_EINVAL, "null config");
  if (c->nx < 2 || c->ny < 1 || c->nz < 1 || c->nx % 2) return fail64(PF_EINVAL, "bad grid for the FP64 path");
  if ((double)c->nx * c->ny * c->nz > (double)(1u << 30)) return fail64(PF_EINVAL, "grid too large for the FP64 path");
  if (c->var < 1 || c->var > 256) return fail64(PF_EINVAL, "var=%d outside [1, 256]", c->var);
  return PF_OK;
}

void plain64_destroy(Plain64* p) {
  if (!p) return;
  cudaSetDevice(p->device);
  for (cufftHandle h : {p->fwd, p->inv, p->fwdB, p->invB})
    if (h) cufftDestroy(h);
  if (p->stream) cudaStreamDestroy(p->stream);
  cudaFree(p->mem);
  delete p;
}

int plain64_create(const pf_config* c, Plain64** out) {
  int rc = plain64_validate(c);
  if (rc) return rc;
  Plain64* p = new Plain64();
  p->c = *c;
  p->device = c->device;
  p->Nx = c->nx; p->Ny = c->ny; p->Nz = c->nz; p->Kx = c->nx / 2 + 1; p->V = c->var;
  p->ncell = (size_t)p->Nx * p->Ny * p->Nz;
  p->nspec = (size_t)p->Kx * p->Ny * p->Nz;
  auto bail = [&](int r) { plain64_destroy(p); return r; };
#define TRY(call) do { cudaError_t e_ = (call); if (e_ != cudaSuccess) \
    return bail(fail64(PF_ENOMEM, "%s: %s", #call, cudaGetErrorString(e_))); } while (0)
  TRY(cudaSetDevice(p->device));
  p->var_mob = c->mobility == PF_MOB_C1MC || c->D_gb != 0.0;
  {
    // chunks of (nearly) equal size
    const size_t fit = std::max<size_t>(1, kChunkBytes / (p->nspec * sizeof(cufftDoubleComplex)));
    const int chunks = (int)((p->V + fit - 1) / fit);
    p->B = (p->V + chunks - 1) / chunks;
  }
  TRY(cudaStreamCreateWithFlags(&p->stream, cudaStreamNonBlocking));
  // plans of one field and of B fields, sharing one work area
  size_t need = 0;
  auto plan = [&](cufftHandle* h, cufftType type, int batch) {
    int dims[3] = {p->Nz, p->Ny, p->Nx};
    size_t ws = 0;
    if (cufftCreate(h) != CUFFT_SUCCESS || cufftSetAutoAllocation(*h, 0) != CUFFT_SUCCESS ||
        cufftMakePlanMany(*h, 3, dims, nullptr, 1, 0, nullptr, 1, 0, type, batch, &ws) != CUFFT_SUCCESS)
      return false;
    need = std::max(need, ws);
    return true;
  };
  if (!plan(&p->fwd, CUFFT_D2Z, 1) || !plan(&p->inv, CUFFT_Z2D, 1) ||
      (p->B > 1 && (!plan(&p->fwdB, CUFFT_D2Z, p->B) || !plan(&p->invB, CUFFT_Z2D, p->B))))
    return bail(fail64(PF_ECUDA, "cufftMakePlanMany failed"));
  // All memory in one piece.  A run of one step pays for its memory and plans as
  // much as for the step: made, stepped once and closed, 100 x 100 x 90 with 6
  // order parameters takes 6.7 ms, 7.3 with 13 allocations (10.9 before the
  // transforms were batched).  The two batched plans cost 0.7 to 1.2 ms there
  // and back; they gain 0.06 ms a step at 2 fields, 0.3 at 6.
  const size_t field = p->ncell * sizeof(double), spectrum = p->nspec * sizeof(cufftDoubleComplex);
  size_t bytes = 0;
  const auto take = [&](size_t b) {
    const size_t at = bytes;
    bytes += (b + 255) & ~(size_t)255;
    return at;
  };
  const size_t at_fft = take(need), at_spec = take(3 * spectrum), at_chunk = take(std::max(p->B * spectrum, p->V * field));
  const size_t at_phi = take(p->V * field), at_psi = take(p->V * field), at_con = take(field), at_dfdc = take(field);
  const size_t at_mob = take(p->var_mob ? field : 0), at_work = take(p->var_mob ? field : 0);
  const size_t at_axes = take(2 * (size_t)(p->Kx + p->Ny + p->Nz) * sizeof(double));
  const size_t at_part = take(PA_COUNT * NB * sizeof(double)), at_rec = take(NREC * PA_COUNT * sizeof(double));
  const size_t fint_bytes = 2 * (size_t)(p->V + 1) * NB * sizeof(double), at_fint = take(fint_bytes);
  TRY(cudaMalloc(&p->mem, bytes));
  const auto real = [&](size_t at) { return reinterpret_cast<double*>(p->mem + at); };
  p->phi = real(at_phi);
  p->psi = real(at_psi);
  p->con = real(at_con);
  p->dfdc = real(at_dfdc);
  p->mob = p->var_mob ? real(at_mob) : nullptr;
  p->work = p->var_mob ? real(at_work) : nullptr;
  p->spec = reinterpret_cast<cufftDoubleComplex*>(p->mem + at_spec);
  p->chunk = reinterpret_cast<cufftDoubleComplex*>(p->mem + at_chunk);
  p->dstage = real(at_chunk);
  p->axes = real(at_axes);
  p->part = real(at_part);
  p->rec = real(at_rec);
  p->fint = real(at_fint);
  TRY(cudaMemset(p->fint, 0, fint_bytes));
  void* fftwork = need ? p->mem + at_fft : nullptr;  // a plan that needs none takes none
  for (cufftHandle h : {p->fwd, p->inv, p->fwdB, p->invB})
    if (h && (cufftSetWorkArea(h, fftwork) != CUFFT_SUCCESS || cufftSetStream(h, p->stream) != CUFFT_SUCCESS))
      return bail(fail64(PF_ECUDA, "cufftSetWorkArea failed"));
#undef TRY
  std::vector<double> ax(2 * (size_t)(p->Kx + p->Ny + p->Nz));
  double* hq = ax.data();
  double* hn = ax.data() + (p->Kx + p->Ny + p->Nz);
  host_axis(p->Nx, p->Kx, hq, hn);
  host_axis(p->Ny, p->Ny, hq + p->Kx, hn + p->Kx);
  host_axis(p->Nz, p->Nz, hq + p->Kx + p->Ny, hn + p->Kx + p->Ny);
  cudaError_t e = cudaMemcpy(p->axes, ax.data(), ax.size() * sizeof(double), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return bail(fail64(PF_ECUDA, "table upload: %s", cudaGetErrorString(e)));
  const double* dq = p->axes;
  const double* dn = p->axes + (p->Kx + p->Ny + p->Nz);
  p->ax.qx = dq; p->ax.qy = dq + p->Kx; p->ax.qz = dq + p->Kx + p->Ny;
  p->ax.nx = dn; p->ax.ny = dn + p->Kx; p->ax.nz = dn + p->Kx + p->Ny;
  p->ax.Nx = p->Nx; p->ax.Ny = p->Ny; p->ax.Nz = p->Nz; p->ax.Kx = p->Kx;
  *out = p;
  return PF_OK;
}

int plain64_set_fields(Plain64* p, const double* phi, const double* con) {
  if (!p || !phi || !con) return fail64(PF_EINVAL, "bad arguments to set_fields");
  P64_CUDA(cudaSetDevice(p->device));
  Drain drain{p->stream};
  P64_CUDA(cudaMemcpyAsync(p->dstage, phi, p->V * p->ncell * sizeof(double), cudaMemcpyHostToDevice, p->stream));
  p64_aos_to_soa<<<NB, NT, 0, p->stream>>>(p->dstage, p->phi, p->V, p->ncell);
  P64_CUDA(cudaMemcpyAsync(p->con, con, p->ncell * sizeof(double), cudaMemcpyHostToDevice, p->stream));
  P64_CUDA(cudaStreamSynchronize(p->stream));
  drain.armed = false;
  p->steps = 0;
  p->have_fint = false;
  return PF_OK;
}

int plain64_get_fields(Plain64* p, double* phi, double* con) {
  if (!p || !phi || !con) return fail64(PF_EINVAL, "bad arguments to get_fields");
  P64_CUDA(cudaSetDevice(p->device));
  Drain drain{p->stream};
  p64_soa_to_aos<<<NB, NT, 0, p->stream>>>(p->phi, p->dstage, p->V, p->ncell);
  P64_CUDA(cudaMemcpyAsync(phi, p->dstage, p->V * p->ncell * sizeof(double), cudaMemcpyDeviceToHost, p->stream));
  P64_CUDA(cudaMemcpyAsync(con, p->con, p->ncell * sizeof(double), cudaMemcpyDeviceToHost, p->stream));
  P64_CUDA(cudaStreamSynchronize(p->stream));
  drain.armed = false;
  return PF_OK;
}

int plain64_device_fields(Plain64* p, DeviceFields* out) {
  if (!p || !out) return fail64(PF_EINVAL, "bad arguments to device_fields");
  P64_CUDA(cudaSetDevice(p->device));
  out->phi = p->phi;
  out->con = p->con;
  out->is_double = 1;
  out->fstride = p->ncell;
  out->cstride = 1;
  out->nx = p->Nx; out->ny = p->Ny; out->nz = p->Nz; out->var = p->V; out->device = p->device;
  out->stream = p->stream;
  return PF_OK;
}

// nb fields (B, or 1) forward into the chunk buffer, or back from it.
static int fft_chunk(Plain64* p, bool forward, double* real, int nb) {
  cufftHandle h = nb > 1 ? (forward ? p->fwdB : p->invB) : (forward ? p->fwd : p->inv);
  if (forward) P64_FFT(cufftExecD2Z(h, real, p->chunk));
  else P64_FFT(cufftExecZ2D(h, p->chunk, real));
  return PF_OK;
}

static int one_step(Plain64* p, double* rec) {
  const size_t n = p->ncell, ns = p->nspec;
  const double scale = 1.0 / (double)n;  // f_trans normalisation (src/f_trans.f90:12)
  cudaStream_t s = p->stream;
  cufftDoubleComplex *W0 = p->spec, *W1 = p->spec + ns, *W2 = p->spec + 2 * ns;
  const pf_config& c = p->c;
  const double ecoef = 0.5 * (double)n;  // 0.5 kappa N^3 sum w |kf|^2 |u_hat|^2
  const size_t nfint = (size_t)(p->V + 1) * NB;
  double *now = p->fint + p->cur * nfint, *next = p->fint + (1 - p->cur) * nfint;
  auto chunk_at = [&](int f) { return f + p->B <= p->V ? p->B : 1; };
  int rc;
  if (!p->have_fint) {  // the first step after set_fields: phases 1-4 from the fields' own spectra
    for (int f = 0; f <= p->V; ++f) {
      P64_FFT(cufftExecD2Z(p->fwd, f < p->V ? p->phi + (size_t)f * n : p->con, W0));
      p64_fint<<<NB, NT, 0, s>>>(W0, p->ax, ecoef * (f < p->V ? c.grad_coeff_phi : c.grad_coeff_c) * scale * scale, ns,
                                 now + (size_t)f * NB);
    }
    p->have_fint = true;
  }
  // phases 5-10 (bulk), statistics of the same fields
  p64_bulk<<<NB, NT, 0, s>>>(p->phi, p->con, p->psi, p->dfdc, p->mob, p->V, n, c, c.mobility == PF_MOB_C1MC, p->part);
  P64_FFT(cufftExecD2Z(p->fwd, p->con, W0));   // dft_con
  P64_FFT(cufftExecD2Z(p->fwd, p->dfdc, W1));  // dft_df_dc
  if (p->var_mob) {  // phases 11-12: variable-mobility flux
    p64_flux<<<NB, NT, 0, s>>>(W0, W1, W2, p->ax, c.grad_coeff_c, scale, ns);
    P64_FFT(cufftExecZ2D(p->inv, W2, p->work));
    p64_jmob<<<NB, NT, 0, s>>>(p->work, p->mob, c.D_L, n);
    P64_FFT(cufftExecD2Z(p->fwd, p->work, W2));
  }
  // phase 13
  p64_ch<<<NB, NT, 0, s>>>(W0, p->var_mob ? W2 : nullptr, W1, p->ax, c.t_step, c.D_L, c.grad_coeff_c, scale,
                           ecoef * c.grad_coeff_c, ns, next + (size_t)p->V * NB);
  P64_FFT(cufftExecZ2D(p->inv, W0, p->con));
  // phase 14; a chunk's partials go to its first field's slot, the others stay zero
  for (int f = 0; f < p->V;) {
    const int nb = chunk_at(f);
    if ((rc = fft_chunk(p, true, p->psi + (size_t)f * n, nb))) return rc;
    p64_ac<<<NB, NT, 0, s>>>(p->chunk, p->ax, c.mob_phi * c.grad_coeff_phi * c.t_step, scale, ecoef * c.grad_coeff_phi,
                             ns, nb, next + (size_t)f * NB);
    if ((rc = fft_chunk(p, false, p->phi + (size_t)f * n, nb))) return rc;
    f += nb;
  }
  p64_finish<<<PA_COUNT, NT, 0, s>>>(p->part, now, (int)nfint, rec);
  if (p->B > 1)  // the start's per-field partials must not stay in the slots that chunks leave alone
    P64_CUDA(cudaMemsetAsync(now, 0, nfint * sizeof(double), s));
  p->cur = 1 - p->cur;
  P64_CUDA(cudaGetLastError());
  return PF_OK;
}

int plain64_step(Plain64* p, int nsteps, pf_diag* diag) {
  if (!p || nsteps < 0) return fail64(PF_EINVAL, "bad arguments to step");
  P64_CUDA(cudaSetDevice(p->device));
  int bad = 0;
  std::vector<double> acc((size_t)std::max(nsteps, 1) * PA_COUNT);
  for (int st = 0; st < nsteps; st += NREC) {
    const int m = std::min(NREC, nsteps - st);
    for (int k = 0; k < m; ++k) {
      int rc = one_step(p, p->rec + (size_t)k * PA_COUNT);
      if (rc) return rc;
    }
    P64_CUDA(cudaMemcpyAsync(acc.data() + (size_t)st * PA_COUNT, p->rec, (size_t)m * PA_COUNT * sizeof(double),
                             cudaMemcpyDeviceToHost, p->stream));
    P64_CUDA(cudaStreamSynchronize(p->stream));
  }
  for (int st = 0; st < nsteps; ++st) {
    const double* a = acc.data() + (size_t)st * PA_COUNT;
    if (a[PA_BAD] != 0) bad = 1;
    if (diag) {
      pf_diag& d = diag[st];
      d.step = p->steps + st + 1;
      d.nonfinite = (int)a[PA_BAD];
      d.f_int = a[PA_FINT];
      d.f_eta = a[PA_FETA];
      d.f_ch = a[PA_FCH];
      d.e_tot = a[PA_FINT] + a[PA_FCH] + a[PA_FETA];
      d.c_max = a[PA_CMAX];
      d.c_min = a[PA_CMIN];
      d.phi_min = a[PA_PHIMIN];
      d.phi_P_max = a[PA_PHIPMAX];
      d.mass = a[PA_MASS];
    }
  }
  p->steps += nsteps;
  if (bad) return fail64(PF_ENONFINITE, "a step produced non-finite values");
  return PF_OK;
}

// ---------------------------------------------------------------------------
// Fortran shims
// ---------------------------------------------------------------------------
// out[b][y][a] = scale in[a][y][b]: between cuFFT's [z][y][kx] and P3DFFT's
// transposed order [kx][y][z], 32 x 32 tiles through shared memory so that both
// sides move in 512-byte pieces; `in` may be the caller's own memory.
constexpr int kTile = 32, kTileRows = 8;
__global__ void __launch_bounds__(kTile* kTileRows) p64_transpose(const cufftDoubleComplex* __restrict__ in,
                                                                  cufftDoubleComplex* __restrict__ out, int nA, int Ny,
                                                                  int nB, double scale) {
  __shared__ cufftDoubleComplex tile[kTile][kTile + 1];
  const int y = blockIdx.z, b0 = blockIdx.x * kTile, a0 = blockIdx.y * kTile;
  for (int r = threadIdx.y; r < kTile; r += kTileRows) {
    const int a = a0 + r, b = b0 + threadIdx.x;
    if (a < nA && b < nB) tile[r][threadIdx.x] = in[((size_t)a * Ny + y) * nB + b];
  }
  __syncthreads();
  for (int r = threadIdx.y; r < kTile; r += kTileRows) {
    const int b = b0 + r, a = a0 + threadIdx.x;
    if (a < nA && b < nB) {
      const cufftDoubleComplex v = tile[threadIdx.x][r];
      out[((size_t)b * Ny + y) * nA + a] = make_cuDoubleComplex(v.x * scale, v.y * scale);
    }
  }
}
static int transpose(const cufftDoubleComplex* in, cufftDoubleComplex* out, int nA, int Ny, int nB, double scale) {
  for (int y0 = 0; y0 < Ny; y0 += 65535) {  // the grid's z extent
    const dim3 grid((nB + kTile - 1) / kTile, (nA + kTile - 1) / kTile, std::min(Ny - y0, 65535));
    p64_transpose<<<grid, dim3(kTile, kTileRows)>>>(in + (size_t)y0 * nB, out + (size_t)y0 * nA, nA, Ny, nB, scale);
  }
  P64_CUDA(cudaGetLastError());
  return PF_OK;
}

// Whether the shims' kernels may read the caller's array where it is: host
// memory, aligned as the transforms want it, on a GPU that walks the host's
// page tables.  The first kernel then takes the place of a copy and runs while
// the data arrives.
static bool reads_host(const void* p, int device) {
  int coherent = 0;
  cudaPointerAttributes a;
  if ((uintptr_t)p % 16 != 0 ||
      cudaDeviceGetAttribute(&coherent, cudaDevAttrPageableMemoryAccessUsesHostPageTables, device) != cudaSuccess ||
      !coherent || cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeHost || a.type == cudaMemoryTypeUnregistered;
}

struct ShimCtx {
  std::mutex mu;
  int device = 0;
  struct Plans {
    cufftHandle f = 0, i = 0;
    double* real = nullptr;
    cufftDoubleComplex* a = nullptr;
    cufftDoubleComplex* b = nullptr;
  };
  std::map<std::tuple<int, int, int, int>, Plans> plans;  // plans and memory belong to a device
};
static ShimCtx& shim() {
  static ShimCtx* s = new ShimCtx();
  return *s;
}

static int make_shim_plans(int Nx, int Ny, int Nz, ShimCtx::Plans& pl) {
  const size_t n = (size_t)Nx * Ny * Nz, ns = (size_t)(Nx / 2 + 1) * Ny * Nz;
  P64_CUDA(cudaMalloc(&pl.real, n * sizeof(double)));
  P64_CUDA(cudaMalloc(&pl.a, ns * sizeof(cufftDoubleComplex)));
  P64_CUDA(cudaMalloc(&pl.b, ns * sizeof(cufftDoubleComplex)));
  P64_FFT(cufftPlan3d(&pl.f, Nz, Ny, Nx, CUFFT_D2Z));
  P64_FFT(cufftPlan3d(&pl.i, Nz, Ny, Nx, CUFFT_Z2D));
  return PF_OK;
}

static int shim_plans(int Nx, int Ny, int Nz, ShimCtx::Plans** out) {
  ShimCtx& S = shim();
  auto key = std::make_tuple(S.device, Nx, Ny, Nz);
  auto it = S.plans.find(key);
  if (it != S.plans.end()) { *out = &it->second; return PF_OK; }
  ShimCtx::Plans pl;
  const int rc = make_shim_plans(Nx, Ny, Nz, pl);
  if (rc) {
    for (cufftHandle h : {pl.f, pl.i})
      if (h) cufftDestroy(h);
    cudaFree(pl.real);
    cudaFree(pl.a);
    cudaFree(pl.b);
    return rc;
  }
  S.plans[key] = pl;
  *out = &S.plans[key];
  return PF_OK;
}

static bool single_rank(const int* ist, const int* fst) {
  return ist[0] == 1 && ist[1] == 1 && ist[2] == 1 && fst[0] == 1 && fst[1] == 1 && fst[2] == 1;
}

static void shim_report(int rc, const char* who) {
  if (rc) fprintf(stderr, "%s: %s\n", who, pf_last_error());
}

}  // namespace pf

using namespace pf;

extern "C" {

int pf_shim_device(int device) {
  ShimCtx& S = shim();
  std::lock_guard<std::mutex> lk(S.mu);
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || device < 0 || device >= n)
    return fail64(PF_EINVAL, "no CUDA device %d", device);
  S.device = device;
  return PF_OK;
}

static int f_trans_impl(const double* in, double* out, int Nx, int Ny, int Nz, const int* ist, const int* ien,
                        const int* fst, const int* fen) {
  if (!single_rank(ist, fst) || ien[0] != Nx || ien[1] != Ny || ien[2] != Nz || fen[0] != Nz || fen[1] != Ny ||
      fen[2] != Nx / 2 + 1)
    return fail64(PF_EINVAL, "f_trans_: only the single-rank layout ist=fst=1, ien=(Nx,Ny,Nz), fen=(Nz,Ny,Nx/2+1)");
  ShimCtx& S = shim();
  std::lock_guard<std::mutex> lk(S.mu);
  P64_CUDA(cudaSetDevice(S.device));
  ShimCtx::Plans* pl;
  int rc = shim_plans(Nx, Ny, Nz, &pl);
  if (rc) return rc;
  const size_t n = (size_t)Nx * Ny * Nz, ns = (size_t)(Nx / 2 + 1) * Ny * Nz;
  Drain drain{nullptr};
  double* real = const_cast<double*>(in);  // a real-to-complex transform out of place leaves its input alone
  if (!reads_host(in, S.device)) {
    real = pl->real;
    P64_CUDA(cudaMemcpy(real, in, n * sizeof(double), cudaMemcpyHostToDevice));
  }
  P64_FFT(cufftExecD2Z(pl->f, real, pl->a));
  if ((rc = transpose(pl->a, pl->b, Nz, Ny, Nx / 2 + 1, 1.0 / (double)n))) return rc;
  P64_CUDA(cudaMemcpy(out, pl->b, ns * sizeof(cufftDoubleComplex), cudaMemcpyDeviceToHost));
  drain.armed = false;
  return PF_OK;
}

void f_trans_(const double* in, double* out, const int* Nx, const int* Ny, const int* Nz, const int* ist,
              const int* ien, const int* fst, const int* fen) {
  shim_report(f_trans_impl(in, out, *Nx, *Ny, *Nz, ist, ien, fst, fen), "f_trans_");
}

static int inv_trans_impl(const double* in, double* out, const int* ist, const int* ien, const int* fst,
                          const int* fen) {
  const int Nx = ien[0] - ist[0] + 1, Ny = ien[1] - ist[1] + 1, Nz = ien[2] - ist[2] + 1;
  if (!single_rank(ist, fst) || fen[0] != Nz || fen[1] != Ny || fen[2] != Nx / 2 + 1)
    return fail64(PF_EINVAL, "inv_trans_: only the single-rank layout is supported");
  ShimCtx& S = shim();
  std::lock_guard<std::mutex> lk(S.mu);
  P64_CUDA(cudaSetDevice(S.device));
  ShimCtx::Plans* pl;
  int rc = shim_plans(Nx, Ny, Nz, &pl);
  if (rc) return rc;
  const size_t n = (size_t)Nx * Ny * Nz, ns = (size_t)(Nx / 2 + 1) * Ny * Nz;
  Drain drain{nullptr};
  const cufftDoubleComplex* spec = reinterpret_cast<const cufftDoubleComplex*>(in);
  if (!reads_host(in, S.device)) {
    spec = pl->b;
    P64_CUDA(cudaMemcpy(pl->b, in, ns * sizeof(cufftDoubleComplex), cudaMemcpyHostToDevice));
  }
  if ((rc = transpose(spec, pl->a, Nx / 2 + 1, Ny, Nz, 1.0))) return rc;
  P64_FFT(cufftExecZ2D(pl->i, pl->a, pl->real));
  P64_CUDA(cudaMemcpy(out, pl->real, n * sizeof(double), cudaMemcpyDeviceToHost));
  drain.armed = false;
  return PF_OK;
}

void inv_trans_(const double* in, double* out, const int* ist, const int* ien, const int* fst, const int* fen) {
  shim_report(inv_trans_impl(in, out, ist, ien, fst, fen), "inv_trans_");
}

// src/k_space.f90:13-59 on the caller's (possibly partial) spectral pencil:
// kf(3, fst(1):fen(1), fst(2):fen(2), fst(3):fen(3)) complex, dim 1 = z, dim 3 = kx.
void k_space_(const int* Nx, const int* Ny, const int* Nz, const int* fst, const int* fen, double* kf, double* kf_sq,
              double* kf_4) {
  const double pi = std::atan(1.0) * 4.0;
  const double u1 = 2.0 * pi / (double)*Nx, u2 = 2.0 * pi / (double)*Ny, u3 = 2.0 * pi / (double)*Nz;
  const int n1 = fen[0] - fst[0] + 1, n2 = fen[1] - fst[1] + 1;
  for (int i = fst[2]; i <= fen[2]; ++i) {
    const int ii = i - 1;
    const double l1 = (ii <= *Nx / 2 ? ii : ii - *Nx) * u1;
    for (int j = fst[1]; j <= fen[1]; ++j) {
      const int jj = j - 1;
      const double l2 = (jj <= *Ny / 2 ? jj : jj - *Ny) * u2;
      for (int k = fst[0]; k <= fen[0]; ++k) {
        const int kk = k - 1;
        const double l3 = (kk <= *Nz / 2 ? kk : kk - *Nz) * u3;
        const size_t cell = ((size_t)(i - fst[2]) * n2 + (j - fst[1])) * n1 + (k - fst[0]);
        double* a = kf + cell * 6;
        double* b = kf_sq + cell * 6;
        double* c = kf_4 + cell * 6;
        const double l[3] = {l1, l2, l3};
        const bool nyq[3] = {2 * ii == *Nx, 2 * jj == *Ny, 2 * kk == *Nz};
        for (int d = 0; d < 3; ++d) {
          a[2 * d] = 0.0;
          a[2 * d + 1] = nyq[d] ? 0.0 : l[d];
          b[2 * d] = -l[d] * l[d];
          b[2 * d + 1] = 0.0;
          c[2 * d] = l[d] * l[d] * l[d] * l[d];
          c[2 * d + 1] = 0.0;
        }
      }
    }
  }
}

}  // extern "C"
