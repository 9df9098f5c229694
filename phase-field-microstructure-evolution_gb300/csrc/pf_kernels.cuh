// Fused FP32 kernels of the semi-implicit spectral step (sm_103a).
//
// State of one run, for every field f (the var order parameters, then the
// concentration c):
//   Sk[f][kx][kz][ypos]    u_hat in k-space (normalised like f_trans,
//                          src/f_trans.f90:12), y in digit-transposed order;
//   Sm[f][kx][z][y]        (large runs: [f][z][kx][y]) the same field in "mixed" space: its x half
//                          spectrum (1/Nx) sum_x u e^{-2 pi i kx x/Nx} with y, z
//                          in real space (what the x pass needs).
// The reference keeps phi/con in real space and takes a full 3-D R2C per
// field and use (src/f_trans.f90:11-12, 7*var+9 transforms per step); here one
// step is two passes over the fields:
//
//   x pass  (x_pass_kernel, one CTA per WY y-rows at one z, all fields):
//       Sm --C2R_x--> phi, c --bulk terms (src/var_diff.f90:685-898)-->
//       dF/dphi_i, dF/dc (, mobility) --R2C_x/Nx--> D
//   yz pass (yz1_kernel, yz_kernel: one CTA or cluster per (field, kx) plane):
//       D --DFT_yz--> D_hat;  u_hat += m1 u_hat + m2 D_hat  (pointwise);
//       u_hat --IDFT_yz--> Sm
//
// In exact arithmetic the pointwise update is the reference's
//   u_hat_new = (u_hat - L dt D_hat) / (1 - L kappa dt K2)                (AC, :1020-1024)
//   c_hat_new = (c_hat + D_mean K2 dt mu_hat) / (1 + D_mean dt kappa_c K4)  (CH, :976-983)
// written as an increment so that the state never takes an FP32 round trip
// through an FFT.  The variable-mobility term dt G J'_hat / (...) of :976-983 is
// added by a second x/yz pass pair (xj pass + the yz kernel in C2 mode).
#pragma once
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "pf_fft.cuh"

namespace cg = cooperative_groups;

namespace pf {

// Per-block diagnostic partials of the x pass (floats; the sums as
// compensated hi + lo pairs): part_x[(par * XQ_COUNT + q) * nblk_x + block],
// par = Shape::par, the step's parity: the record of one step reads its
// partials while the next step's x pass writes the other set.
enum XDiag {
  XQ_FETA_H = 0, XQ_FETA_L, XQ_FCH_H, XQ_FCH_L, XQ_MASS_H, XQ_MASS_L,
  XQ_CMIN, XQ_CMAX, XQ_PHIMIN, XQ_PHIPMAX, XQ_BAD, XQ_COUNT
};
// room reserved per (z, y) row for the x partials of both parities (doubles'
// worth, any variant)
constexpr int XD_COUNT = 12;
static_assert(2 * XQ_COUNT * 4 <= XD_COUNT * 8, "x partials must fit the reserved room");
// Per-step diagnostic record layout (doubles)
enum DiagRec {
  DR_STEP = 0, DR_FINT, DR_FETA, DR_FCH, DR_CMIN, DR_CMAX, DR_PHIMIN, DR_PHIPMAX, DR_MASS, DR_NONFINITE, DR_COUNT
};

enum Mobility { MOB_CONST = 0, MOB_REF_VAR = 1, MOB_C1MC = 2 };

// Device-side description of one run (all runs of a launch share one shape)
struct RunParams {
  float2* Sk;      // [nF][Kx] planes [kz][y position] of the k-space state
  float2* Sm;      // [nF] x Kx, Nz, Ny (strides ks, zs, 1): state in mixed space (x spectrum, real-space y, z)
  float2* D;       // as Sm: x-spectra of dF/dphi_i and dF/dc
  float* mob;      // [Nz][Ny][Nx] mobility minus D_mean (variable mobility only)
  float2* J;       // one field as Sm: CH flux scratch (variable mobility only)
  float* part_x;   // [2][XQ_COUNT][nblk_x]: per step parity
  float* part_yz;  // [2][2][nblk_yz]: per step parity, hi and lo of each yz CTA's weighted f_int sum
  double* diag;    // [ring][DR_COUNT]
  double* hdiag;   // the same in pinned host memory (few runs), else null
  int* counter;    // step counter (device)
  float L, kappa_phi, kappa_c, dt, D_L, D_gb, sigma1, sigma2, am, ap, c0m, c0p;
  int mobility;
  int V;           // number of order parameters
  int ring;        // diag ring length
  int pad;
};

// Per-shape tables (FP64-derived, stored as float)
struct Shape {
  int Nx, Ny, Nz, Kx;
  const float2* twM;  // W_{Nx/2}^j, j < Nx/2
  const float2* twN;  // W_{Nx}^j,   j < Nx
  const float2* twY;  // W_{Ny}^j
  const float2* twZ;  // W_{Nz}^j
  const float* qx2; const float* qy2; const float* qz2;  // q_d^2 (kf_sq)
  const float* qx4; const float* qy4; const float* qz4;  // q_d^4 (kf_4)
  const float* qnx; const float* qny; const float* qnz;  // Nyquist-zeroed q_d (kf / i)
  int nblk_x;   // blocks of the x pass per run
  int nblk_yz;  // blocks of the yz pass per run
  int plane0;   // first (field, kx) plane of a yz-pass launch (a launch may cover a subset)
  int ks, zs;   // strides of kx and z in Sm, D and J (y contiguous; see mixed_strides)
  // fields of one run for the import and export modes: the caller's layout,
  // phi(var, x, y, z) and con(x, y, z), and float [nF][Nz][Ny][Nx] (MODE_FIELDS)
  double *io_phi, *io_con;
  float* fin;
  int par;  // parity of the step: which set of diagnostic partials its passes write and its record reads
};

// ---------------------------------------------------------------------------
// Compensated sums for the mass of c (src/var_diff.f90:1076-1102).  A thread
// keeps its running sum as an unevaluated FP32 pair hi + lo updated with
// Knuth's error-free TwoSum (s + e == a + b exactly), warps combine the pairs
// the same way, and from there on the sum is FP64 with Neumaier's
// compensation (KSum) across warps, blocks and the final record.  FP64
// arithmetic is scarce on this part, so only the per-warp and later stages
// use it.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}
struct FF {
  float hi, lo;
  __device__ __forceinline__ void add(float v) {
    float s, e;
    two_sum(hi, v, s, e);
    hi = s;
    lo = __fadd_rn(lo, e);
  }
  __device__ __forceinline__ void add(const FF& o) {
    float s, e;
    two_sum(hi, o.hi, s, e);
    hi = s;
    lo = __fadd_rn(__fadd_rn(lo, o.lo), e);
  }
  __device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
};
__device__ __forceinline__ FF ff(float hi, float lo = 0.f) {
  FF x;
  x.hi = hi;
  x.lo = lo;
  return x;
}
// sum of the pairs of a warp (every lane gets a sum of all 32)
__device__ __forceinline__ FF warp_sum_ff(FF x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x.add(ff(__shfl_xor_sync(0xffffffffu, x.hi, o), __shfl_xor_sync(0xffffffffu, x.lo, o)));
  return x;
}
// compensated FP64 sum (Kahan-Babuska-Neumaier, the error of each addition
// taken exactly by TwoSum): value() = s + c
struct KSum {
  double s = 0.0, c = 0.0;
  __device__ __forceinline__ void add(double v) {
    const double t = __dadd_rn(s, v);
    const double bb = __dsub_rn(t, s);
    c = __dadd_rn(c, __dadd_rn(__dsub_rn(s, __dsub_rn(t, bb)), __dsub_rn(v, bb)));
    s = t;
  }
  __device__ __forceinline__ void add(const KSum& o) {
    add(o.s);
    c = __dadd_rn(c, o.c);
  }
  __device__ __forceinline__ double value() const { return __dadd_rn(s, c); }
};

__device__ __forceinline__ float warp_min(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// ---------------------------------------------------------------------------
// x-direction half spectrum <-> interleaved real line (M = Nx/2 complex).
// With z[m] = x[2m] + i x[2m+1] and Z = DFT_M(z):
//   X[k] = (Z[k] + conj Z[M-k])/2 - (i/2) W_N^k (Z[k] - conj Z[M-k]),
//   X[0] = Re Z0 + Im Z0,  X[M] = Re Z0 - Im Z0;
// the inverse builds Z'[k] = (X[k] + conj X[M-k]) + i conj(W_N^k) (X[k] - conj X[M-k])
// so that IDFT_M(Z') = N z.  Frequencies k and M-k always sit in mirrored
// runs of the four-step layout, so one thread owns both halves of every pair.
// ---------------------------------------------------------------------------
// Since W_N^(M-k) = -conj(W_N^k), the two halves of a pair share one product:
// inverse pre-processing of the pair (k, M-k), 0 < k < M, with
// s = x_k + conj(x_m), d = x_k - conj(x_m), e = i d conj(w_k):
//   z_k = s + e,   z_m = conj(s - e)
// (one twiddle and 9 instructions a pair; two products took two and 12).
__device__ __forceinline__ void pre_pair(float2 xk, float2 xm, float2 wk, float2& zk, float2& zm) {
  const float2 s = __ffma2_rn(xm, make_float2(1.f, -1.f), xk);
  const float2 d = __ffma2_rn(xm, make_float2(-1.f, 1.f), xk);
  const float2 e = make_float2(fmaf(d.x, wk.y, -d.y * wk.x), fmaf(d.x, wk.x, d.y * wk.y));  // i d conj(wk)
  zk = __fadd2_rn(s, e);
  zm = make_float2(s.x - e.x, e.y - s.y);
}
// forward post-processing of the pair (k, M-k), 0 < k < M: twice the spectrum,
// with s = z_k + conj(z_m), d = z_k - conj(z_m), e = -i d w_k:
//   2 x_k = s + e,   2 x_m = conj(s - e).
__device__ __forceinline__ void post_pair(float2 zk, float2 zm, float2 wk, float2& xk, float2& xm) {
  const float2 s = __ffma2_rn(zm, make_float2(1.f, -1.f), zk);
  const float2 d = __ffma2_rn(zm, make_float2(-1.f, 1.f), zk);
  const float2 e = make_float2(fmaf(d.x, wk.y, d.y * wk.x), fmaf(-d.x, wk.x, d.y * wk.y));  // -i d wk
  xk = __fadd2_rn(s, e);
  xm = make_float2(s.x - e.x, e.y - s.y);
}

// Factorization of the x pass's lines (M = Nx/2 complex points): the plan's,
// except M = 128 as 8 x 16.  With runs of 8 the largest per-thread state of
// the x pass is one DFT_16 instead of a pair of them: 80 registers a thread
// at Nx = 256 instead of 128 with spills (the same speed at 33 fields).
template <int M>
struct XPlan {
  static constexpr int N1 = Plan<M>::N1, N2 = Plan<M>::N2;
};
template <>
struct XPlan<128> {
  static constexpr int N1 = 8, N2 = 16;
};
// A line of the x pass in shared memory: the runs follow one another without
// pad slots, and an odd pitch of at least M + 1 (slot M takes kx = M while the
// spectrum is in place).  The transforms' lanes go from line to line, so the
// odd pitch alone keeps them free of bank conflicts; the bulk terms' lanes go
// along a line, where a pad after each run put two of 16 slots in one bank
// pair (a quarter of the pass's shared wavefronts at Nx = 128).
template <int M>
struct XLine {
  static constexpr int N1 = XPlan<M>::N1, N2 = XPlan<M>::N2;
  static constexpr int PITCH = M % 2 == 0 ? M + 1 : M + 2;
};

// A twiddle of the x pass: from a copy of the table in shared memory (TWS),
// else from the global table through the read-only path.
template <bool TWS>
__device__ __forceinline__ float2 ldtw(const float2* p) {
  if constexpr (TWS) return *p;
  else return __ldg(p);
}

// One pass-A item: the N2 elements of column n1 of the line at p (column
// included), twiddles w(k2) = W_L^(n1 k2).
template <int N1, int N2, int STRIDE, bool INV, class Tw>
__device__ __forceinline__ void passA_item(float2* p, const Tw& w) {
  float2 v[N2];
  if (!INV) {
#pragma unroll
    for (int n2 = 0; n2 < N2; ++n2) v[n2] = p[n2 * STRIDE];
    Dft<N2>::fwd(v);
#pragma unroll
    for (int k2 = 1; k2 < N2; ++k2) v[k2] = cmul(v[k2], w(k2));
  } else {
    v[0] = p[0];
#pragma unroll
    for (int k2 = 1; k2 < N2; ++k2) v[k2] = cmulc(p[k2 * STRIDE], w(k2));
    dft_inv<N2>(v);
  }
#pragma unroll
  for (int k = 0; k < N2; ++k) p[k * STRIDE] = v[k];
}

// pass A over a runtime number of lines (pitch P, T threads).  A warp takes 32
// consecutive lines at one column n1: with an odd pitch those 32 accesses hit
// distinct bank pairs.  Where the CTA's warps are a multiple of N1 or divide
// it, a warp loads a column's twiddles once for all its lines; the lines beyond the last
// whole 32 are spread over (line, column), so that they cost rem N1 / 32
// warp items instead of N1 (17 fields x 8 rows: 136 lines, 34 items, not 40).
template <int L, int P, int T, bool INV, bool TWS = false>
__device__ __forceinline__ void passA_rt(float2* buf, int NL, const float2* __restrict__ tw) {
  constexpr int N1 = XLine<L>::N1, N2 = XLine<L>::N2, NW = T / 32;
  if constexpr (NW % N1 == 0 || N1 % NW == 0) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int full = NL & ~31;
    for (int n1 = w % N1; n1 < N1; n1 += NW) {
      float2 wt[N2];
#pragma unroll
      for (int k2 = 1; k2 < N2; ++k2) wt[k2] = ldtw<TWS>(tw + n1 * k2);
      for (int l = (w / N1) * 32 + lane; l < full; l += 32 * (NW > N1 ? NW / N1 : 1))
        passA_item<N1, N2, N1, INV>(buf + l * P + n1, [&](int k2) { return wt[k2]; });
    }
    const int rem = NL - full;
    for (int it = threadIdx.x; it < rem * N1; it += T) {
      const int m1 = it / rem, l = full + it - m1 * rem;
      passA_item<N1, N2, N1, INV>(buf + l * P + m1, [&](int k2) { return ldtw<TWS>(tw + m1 * k2); });
    }
  } else {
    const int nlb = (NL + 31) >> 5;  // groups of 32 lines
    const int items = nlb * 32 * N1;
    for (int it = threadIdx.x; it < items; it += T) {
      const int lo = it & 31, rest = it >> 5;
      const int n1 = rest % N1, l = (rest / N1) * 32 + lo;
      if (l >= NL) continue;
      passA_item<N1, N2, N1, INV>(buf + l * P + n1, [&](int k2) { return ldtw<TWS>(tw + n1 * k2); });
    }
  }
}

// Division of small counts by a count n fixed for the kernel: a multiply
// (exact for x n < 2^32) instead of about 20 instructions.
struct FastDiv {
  unsigned n, magic;
  __device__ __forceinline__ explicit FastDiv(int n_) : n(n_), magic(0xffffffffu / (unsigned)n_ + 1u) {}
  __device__ __forceinline__ int operator()(int x) const { return n == 1 ? x : (int)__umulhi((unsigned)x, magic); }
};

// Where element kx of a line's half spectrum is read from:
//   SPEC_GLOBAL  src + kx * stride in read-only global memory;
//   SPEC_INPLACE the line itself, kx at run kx % N2, element kx / N2 of the
//                run (x_spec_slot), and kx = M in slot M.
// In place, the inputs of a run pair are exactly the slots its outputs go
// to, so every item reads its inputs into registers and overwrites them.
enum SpecSrc { SPEC_GLOBAL = 0, SPEC_INPLACE = 1 };

template <int M>
__device__ __forceinline__ int x_spec_slot(int kx) {
  constexpr int N1 = XLine<M>::N1, N2 = XLine<M>::N2;
  return kx == M ? M : N1 * (kx % N2) + kx / N2;
}

// Element k1 of run r: kx = r + N2 k1, step = N2 strides of kx.
template <int SRC, int M>
__device__ __forceinline__ float2 ld_spec(const float2* src, int step, int r, int k1) {
  if constexpr (SRC == SPEC_INPLACE) return src[XLine<M>::N1 * r + k1];
  else return __ldg(src + (ptrdiff_t)k1 * step);
}

// Run pair of item group q of a line (x_inv_runs / x_fwd_runs), q < N2/2 + 1:
// the pairs (pr, N2 - pr), 0 < pr < N2/2, first, then the single runs 0 and
// (N2 even) N2/2.  A pair item costs two DFT_N1, a single one, so with the
// pairs handed out first the last round of items holds only single runs
// (132 lines at N2 = 8 and 512 threads: 3 rounds of DFT_N1 instead of 4).
template <int M>
__device__ __forceinline__ int x_run_pair(int q) {
  constexpr int N2 = XLine<M>::N2, NPR = (N2 - 1) / 2;
  return q < NPR ? q + 1 : (q == NPR ? 0 : N2 / 2);
}

// Inverse x transform, first half: read the half spectrum of line (f, yy)
// for the run pair `pr` (from where SRC says), pre-process, inverse DFT_N1 of
// each run, store the runs (pass B' output) into the line.
template <int M, int SRC = SPEC_GLOBAL, bool TWS = false>
__device__ __forceinline__ void x_inv_runs(const float2* src, int ks, float2* line, int pr,
                                           const float2* __restrict__ twN) {  // src may be line (in place)
  constexpr int N1 = XLine<M>::N1, N2 = XLine<M>::N2;
  const int step = N2 * ks;
  const auto run = [&](int r) { return SRC == SPEC_INPLACE ? src : src + r * ks; };
  if (pr > 0 && 2 * pr < N2) {
    const int ra = pr, rb = N2 - pr;
    const float2 *sa = run(ra), *sb = run(rb);
    float2 a[N1], b[N1];
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1) {
      a[k1] = ld_spec<SRC, M>(sa, step, ra, k1);
      b[k1] = ld_spec<SRC, M>(sb, step, rb, k1);
    }
    float2 za[N1], zb[N1];
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1) {
      const int k = ra + N2 * k1;
      pre_pair(a[k1], b[N1 - 1 - k1], ldtw<TWS>(twN + k), za[k1], zb[N1 - 1 - k1]);
    }
    dft_inv<N1>(za);
    dft_inv<N1>(zb);
#pragma unroll
    for (int n1 = 0; n1 < N1; ++n1) {
      line[n1 + N1 * ra] = za[n1];
      line[n1 + N1 * rb] = zb[n1];
    }
  } else if (pr == 0) {
    float2 a[N1];
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1) a[k1] = ld_spec<SRC, M>(src, step, 0, k1);
    const float2 xM = SRC == SPEC_INPLACE ? src[M] : ld_spec<SRC, M>(src, step, 0, N1);
    float2 z[N1];
    z[0] = make_float2(a[0].x + xM.x, a[0].x - xM.x);
#pragma unroll
    for (int k1 = 1; k1 <= N1 / 2; ++k1) {
      const int k = N2 * k1;
      float2 zk, zm;
      pre_pair(a[k1], a[N1 - k1], ldtw<TWS>(twN + k), zk, zm);
      z[k1] = zk;
      if (k1 != N1 - k1) z[N1 - k1] = zm;
    }
    dft_inv<N1>(z);
#pragma unroll
    for (int n1 = 0; n1 < N1; ++n1) line[n1] = z[n1];
  } else {  // pr == N2/2: the run pairs with itself, element k1 with N1-1-k1
    const int ra = N2 / 2;
    const float2* sa = run(ra);
    float2 a[N1];
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1) a[k1] = ld_spec<SRC, M>(sa, step, ra, k1);
    float2 z[N1];
#pragma unroll
    for (int k1 = 0; k1 < N1 / 2; ++k1) {
      const int k = ra + N2 * k1;
      pre_pair(a[k1], a[N1 - 1 - k1], ldtw<TWS>(twN + k), z[k1], z[N1 - 1 - k1]);
    }
    dft_inv<N1>(z);
#pragma unroll
    for (int n1 = 0; n1 < N1; ++n1) line[n1 + N1 * ra] = z[n1];
  }
}

// Forward x transform, last half: forward DFT_N1 of the run pair `pr` (pass
// B), post-process, store the half spectrum to global: as it comes, 2 Nx times
// the normalised one, which the yz pass takes into its coefficients, or
// (SCALED) normalised.
template <int M, bool SCALED, bool TWS = false>
__device__ __forceinline__ void x_fwd_runs(float2* __restrict__ dst, int ks, const float2* line, int pr,
                                           const float2* __restrict__ twN) {
  constexpr int N1 = XLine<M>::N1, N2 = XLine<M>::N2;
  const int step = N2 * ks;
  const auto out = [](float2 x) {
    constexpr float h = 0.25f / (float)M;  // 1 / (2 Nx)
    return SCALED ? __fmul2_rn(x, make_float2(h, h)) : x;
  };
  if (pr > 0 && 2 * pr < N2) {
    const int ra = pr, rb = N2 - pr;
    float2 za[N1], zb[N1];
#pragma unroll
    for (int n1 = 0; n1 < N1; ++n1) {
      za[n1] = line[n1 + N1 * ra];
      zb[n1] = line[n1 + N1 * rb];
    }
    Dft<N1>::fwd(za);
    Dft<N1>::fwd(zb);
    float2 *da = dst + ra * ks, *db = dst + rb * ks;
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1) {
      const int k = ra + N2 * k1;
      float2 xk, xm;
      post_pair(za[k1], zb[N1 - 1 - k1], ldtw<TWS>(twN + k), xk, xm);
      da[(ptrdiff_t)k1 * step] = out(xk);
      db[(ptrdiff_t)(N1 - 1 - k1) * step] = out(xm);  // kx = M - k
    }
  } else if (pr == 0) {
    float2 z[N1];
#pragma unroll
    for (int n1 = 0; n1 < N1; ++n1) z[n1] = line[n1];
    Dft<N1>::fwd(z);
    dst[0] = out(make_float2(2.f * (z[0].x + z[0].y), 0.f));
    dst[(ptrdiff_t)N1 * step] = out(make_float2(2.f * (z[0].x - z[0].y), 0.f));  // kx = M
#pragma unroll
    for (int k1 = 1; k1 <= N1 / 2; ++k1) {
      const int k = N2 * k1;
      float2 xk, xm;
      post_pair(z[k1], z[N1 - k1], ldtw<TWS>(twN + k), xk, xm);
      dst[(ptrdiff_t)k1 * step] = out(xk);
      if (k1 != N1 - k1) dst[(ptrdiff_t)(N1 - k1) * step] = out(xm);
    }
  } else {
    const int ra = N2 / 2;
    float2* da = dst + ra * ks;
    float2 z[N1];
#pragma unroll
    for (int n1 = 0; n1 < N1; ++n1) z[n1] = line[n1 + N1 * ra];
    Dft<N1>::fwd(z);
#pragma unroll
    for (int k1 = 0; k1 < N1 / 2; ++k1) {
      const int k = ra + N2 * k1;
      float2 xk, xm;
      post_pair(z[k1], z[N1 - 1 - k1], ldtw<TWS>(twN + k), xk, xm);
      da[(ptrdiff_t)k1 * step] = out(xk);
      da[(ptrdiff_t)(N1 - 1 - k1) * step] = out(xm);
    }
  }
}

// ---------------------------------------------------------------------------
// Bulk terms (src/var_diff.f90:685-898) on the interleaved real lines of all
// fields.
// ---------------------------------------------------------------------------
struct BulkAcc {
  // per-thread partial sums over a few cells, one for each cell of a slot
  // (compensated from the warp level up; the mass, hi + lo, throughout)
  float2 feta, fch, mass_hi, mass_lo;
  float cmin, cmax, phimin, phipmax;
  int nonfinite;
  __device__ __forceinline__ void init() {
    feta = fch = mass_hi = mass_lo = make_float2(0.f, 0.f);
    cmin = 1.0f; cmax = 0.0f; phimin = 1.0f; phipmax = 0.0f;  // reference start values (:1076-1079)
    nonfinite = 0;
  }
  __device__ __forceinline__ void add_mass(float2 c) {  // two_sum of both cells at once
    const float2 t = cadd(mass_hi, c), bb = csub(t, mass_hi);
    mass_lo = cadd(mass_lo, cadd(csub(mass_hi, csub(t, bb)), csub(c, bb)));
    mass_hi = t;
  }
  __device__ __forceinline__ FF mass() const {
    FF a = ff(mass_hi.x, mass_lo.x);
    a.add(ff(mass_hi.y, mass_lo.y));
    return a;
  }
};

// Bulk terms of a slot cell by cell, phi rescaled by 1/max|phi| where FP32
// would lose phi^4 (bulk_slot).
template <int PM, int WY>
__device__ __forceinline__ void bulk_slot_tiny(float2* base, const RunParams& rp, float2 pre2, float2 n4v, float2 prs,
                                               float2& dfdc, float2& mob, BulkAcc& acc) {
  const int V = rp.V;
  const float sg1 = rp.sigma1, sg2 = rp.sigma2;
  constexpr int FS = WY * PM;
  const float pre0 = pre2.x, pre1 = pre2.y, n40 = n4v.x, n41 = n4v.y, pr0 = prs.x, pr1 = prs.y;
  const float2 pP = base[(V - 1) * FS];
  const float2 cc = base[V * FS];
  float2 out_df[2];
  float fch[2], feta[2];
  float t4a[2], t4p[2], invm[2], rP4[2];
  float Smat[2], gP[2];
  // per-cell scalar work (two cells)
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const float pp = q ? pP.y : pP.x;
    const float c = q ? cc.y : cc.x;
    const float pre = q ? pre1 : pre0;
    const float n4 = q ? n41 : n40;
    const float pairs = q ? pr1 : pr0;
    const float pp2 = pp * pp;
    const float S2 = pre + pp2;
    const float S4 = n4 + pp2 * pp2;
    // h = N4/S4 and the term4 ratios (phi^3/S4)(phiP^4/S4).  Below S4 = 1e-30
    // (|phi| < ~1e-8) FP32 would lose them: rescale phi by 1/max|phi|.  All-zero
    // cells give 0/0 in the reference; here h = 0 and term4 = 0.
    float invS4, n4n, sc, im = 1.f;
    float mabs = 0.f;
    if (S4 < 1e-30f) {  // rare: max |phi| of the cell for the rescaled branch
      mabs = fabsf(pp);
      for (int f = 0; f < V - 1; ++f) {
        const float2 p = base[f * FS];
        mabs = fmaxf(mabs, fabsf(q ? p.y : p.x));
      }
    }
    if (S4 >= 1e-30f) {
      invS4 = 1.f / S4;
      n4n = n4 * invS4;
      sc = 4.f;
    } else if (mabs > 0.f) {
      im = 1.f / mabs;
      float s4 = 0.f, nn = 0.f;
      for (int f = 0; f < V - 1; ++f) {
        const float2 p = base[f * FS];
        const float x = (q ? p.y : p.x) * im;
        nn = fmaf(x * x, x * x, nn);
      }
      const float xq = pp * im;
      s4 = nn + (xq * xq) * (xq * xq);
      invS4 = 1.f / s4;
      n4n = nn * invS4;
      sc = 4.f * im;
    } else {
      invS4 = 0.f;
      n4n = 0.f;
      sc = 0.f;
    }
    const float h = n4n;  // phi_mat (:741)
    const float dcm = c - rp.c0m, dcp = c - rp.c0p;
    const float fm = rp.am * dcm * dcm, fp = rp.ap * dcp * dcp;
    const float dfm = fm - fp;
    fch[q] = h * fm + (1.f - h) * fp;
    const float dc = 2.f * h * rp.am * dcm + 2.f * (1.f - h) * rp.ap * dcp;
    feta[q] = -0.5f * S2 + 0.25f * S4 + sg1 * pairs + sg2 * pp2 * pre;
    acc.cmin = fminf(acc.cmin, c);
    acc.cmax = fmaxf(acc.cmax, c);
    acc.phimin = fminf(acc.phimin, S2);
    acc.phipmax = fmaxf(acc.phipmax, pp);
    float mb;
    if (rp.mobility == MOB_REF_VAR) mb = 2.f * (1.f - S2) * rp.D_gb;
    else if (rp.mobility == MOB_C1MC) mb = rp.D_L * c * (1.f - c);
    else mb = 0.f;
    const float qP = pp * im;
    const float qP2 = qP * qP;
    rP4[q] = qP2 * qP2 * invS4;           // phiP^4 / S4
    t4a[q] = sc * invS4 * rP4[q] * dfm;   // term4_i = t4a * q_i^3         (i < V-1)
    t4p[q] = -sc * (qP * qP2 * invS4) * n4n * dfm;  // term4_P                 (:829-835)
    invm[q] = im;
    Smat[q] = pre;
    gP[q] = sg2 * pp2;
    out_df[q] = make_float2(dc, mb);
  }
  dfdc = make_float2(out_df[0].x, out_df[1].x);
  mob = make_float2(out_df[0].y, out_df[1].y);
  acc.fch = cadd(acc.fch, make_float2(fch[0], fch[1]));
  acc.feta = cadd(acc.feta, make_float2(feta[0], feta[1]));
  acc.add_mass(cc);
  float dsum = dfdc.x + dfdc.y;
  {
    for (int f = 0; f < V - 1; ++f) {
      float2 p = base[f * FS];
      const float g0 = fmaf(sg1, Smat[0] - p.x * p.x, gP[0]);
      const float g1 = fmaf(sg1, Smat[1] - p.y * p.y, gP[1]);
      const float q0 = p.x * invm[0], q1 = p.y * invm[1];
      const float d0 = fmaf(p.x, p.x * p.x, -p.x) + 2.f * p.x * g0 + t4a[0] * (q0 * q0 * q0);
      const float d1 = fmaf(p.y, p.y * p.y, -p.y) + 2.f * p.y * g1 + t4a[1] * (q1 * q1 * q1);
      dsum += d0 + d1;
      base[f * FS] = make_float2(d0, d1);
    }
  }
  {
    const float g0 = sg2 * Smat[0], g1 = sg2 * Smat[1];
    const float d0 = fmaf(pP.x, pP.x * pP.x, -pP.x) + 2.f * pP.x * g0 + t4p[0];
    const float d1 = fmaf(pP.y, pP.y * pP.y, -pP.y) + 2.f * pP.y * g1 + t4p[1];
    dsum += d0 + d1;
    base[(V - 1) * FS] = make_float2(d0, d1);
  }
  acc.nonfinite += !isfinite(dsum);  // any NaN/Inf term makes the sum non-finite
}

// Bulk terms of the two cells x = 2m, 2m+1 held in one float2 slot of every
// field line, both at once in packed FP32 pairs.  Pass 1 forms the per-cell
// aggregates, pass 2 overwrites each phi slot with dF/dphi_i; dF/dc and the
// mobility are returned.  Cells with S4 = sum phi^4 below 1e-30 (or a NaN) take
// bulk_slot_tiny instead.
template <int PM, int WY>
__device__ __forceinline__ void bulk_slot(float2* smem, int yy, int slot, const RunParams& rp, float2& dfdc,
                                          float2& mob, BulkAcc& acc) {
  const int V = rp.V;
  const float sg1 = rp.sigma1, sg2 = rp.sigma2;
  float2* base = smem + yy * PM + slot;
  constexpr int FS = WY * PM;  // stride between fields
  const auto both = [](float x) { return make_float2(x, x); };
  // pass 1: pre = sum_{i<V-1} phi^2, n4 = sum_{i<V-1} phi^4, prs = the f_eta pair sum
  float2 pre = both(0.f), n4 = both(0.f), prs = both(0.f);
#pragma unroll 4
  for (int f = 0; f < V - 1; ++f) {
    const float2 p = base[f * FS];
    const float2 a = __fmul2_rn(p, p);
    prs = __ffma2_rn(a, pre, prs);
    pre = __fadd2_rn(pre, a);
    n4 = __ffma2_rn(a, a, n4);
  }
  const float2 pP = base[(V - 1) * FS], c = base[V * FS];
  const float2 pp2 = __fmul2_rn(pP, pP), pp4 = __fmul2_rn(pp2, pp2);
  const float2 S2 = __fadd2_rn(pre, pp2), S4 = __fadd2_rn(n4, pp4);
  if (!(S4.x >= 1e-30f && S4.y >= 1e-30f)) {
    bulk_slot_tiny<PM, WY>(base, rp, pre, n4, prs, dfdc, mob, acc);
    return;
  }
  const float2 invS4 = make_float2(1.f / S4.x, 1.f / S4.y);
  const float2 h = __fmul2_rn(n4, invS4), g = csub(both(1.f), h);  // phi_mat (:741) and phi_ppt
  const float2 dcm = __fadd2_rn(c, both(-rp.c0m)), dcp = __fadd2_rn(c, both(-rp.c0p));
  const float2 adm = __fmul2_rn(both(rp.am), dcm), adp = __fmul2_rn(both(rp.ap), dcp);
  const float2 fm = __fmul2_rn(adm, dcm), fp = __fmul2_rn(adp, dcp), dfm = csub(fm, fp);
  acc.fch = __fadd2_rn(acc.fch, __ffma2_rn(h, fm, __fmul2_rn(g, fp)));
  dfdc = __fmul2_rn(both(2.f), __ffma2_rn(h, adm, __fmul2_rn(g, adp)));
  // -0.5 S2 + 0.25 S4 + sigma_1 pairs + sigma_2 phi_P^2 pre
  const float2 eta = __ffma2_rn(both(0.25f), S4, __fmul2_rn(both(-0.5f), S2));
  acc.feta = __fadd2_rn(acc.feta, __ffma2_rn(both(sg2), __fmul2_rn(pp2, pre), __ffma2_rn(both(sg1), prs, eta)));
  acc.add_mass(c);
  acc.cmin = fminf(acc.cmin, fminf(c.x, c.y));
  acc.cmax = fmaxf(acc.cmax, fmaxf(c.x, c.y));
  acc.phimin = fminf(acc.phimin, fminf(S2.x, S2.y));
  acc.phipmax = fmaxf(acc.phipmax, fmaxf(pP.x, pP.y));
  if (rp.mobility == MOB_REF_VAR) mob = __fmul2_rn(both(2.f * rp.D_gb), csub(both(1.f), S2));
  else if (rp.mobility == MOB_C1MC) mob = __fmul2_rn(__fmul2_rn(both(rp.D_L), c), csub(both(1.f), c));
  else mob = both(0.f);
  // term4_i = t4a phi_i^3 (i < V-1), t4p for the precipitate (:829-835), in
  // the ratios phi_P^4 / S4, phi_P^3 / S4 and N4 / S4
  const float2 d4 = __fmul2_rn(both(4.f), dfm);
  const float2 t4a = __fmul2_rn(__fmul2_rn(invS4, __fmul2_rn(pp4, invS4)), d4);
  const float2 t4p = __fmul2_rn(__fmul2_rn(__fmul2_rn(__fmul2_rn(pP, pp2), invS4), h), d4);  // its negative
  // pass 2: dF/dphi_i = phi^3 - phi + 2 phi Gamma_i + term4_i   (:782-857)
  // with Gamma_i = sigma1 (Smat - phi_i^2) + sigma2 phiP^2:
  //   dF = phi (2 sigma1 (Smat - phi^2) + phi^2 (1 + t4a) + 2 sigma2 phiP^2 - 1)
  const float2 two_s1 = both(2.f * sg1), m1 = both(-1.f);
  const float2 opt4 = __fadd2_rn(both(1.f), t4a);
  const float2 cterm = __ffma2_rn(both(2.f * sg2), pp2, m1);
  float2 ds = dfdc;
#pragma unroll 4
  for (int f = 0; f < V - 1; ++f) {
    const float2 p = base[f * FS];
    const float2 p2 = __fmul2_rn(p, p);
    const float2 sd = __ffma2_rn(p2, m1, pre);  // Smat - phi^2
    const float2 q = __ffma2_rn(sd, two_s1, __ffma2_rn(p2, opt4, cterm));
    const float2 d = __fmul2_rn(p, q);
    ds = __fadd2_rn(ds, d);
    base[f * FS] = d;
  }
  // precipitate: phi^3 - phi + 2 sigma2 Smat phi + t4p
  const float2 dP = csub(__fmul2_rn(pP, __ffma2_rn(both(2.f * sg2), pre, __fadd2_rn(pp2, m1))), t4p);
  ds = __fadd2_rn(ds, dP);
  base[(V - 1) * FS] = dP;
  acc.nonfinite += !isfinite(ds.x + ds.y);  // any NaN/Inf term makes the sum non-finite
}

// Block reduction of the x pass's diagnostics into the block's partials
// part_x[(par * XQ_COUNT + q) * nblk_x + blk] (all threads of the block call it).  Sums travel as
// compensated FP32 pairs: FP64 arithmetic is scarce on this part, and a
// serial FP64 chain at the end of every block held its shared memory (and
// the next block) back.
template <int T>
__device__ __forceinline__ void store_block_diag(const BulkAcc& acc, const RunParams& rp, const Shape& sh, int blk) {
  static_assert(T % 32 == 0 && T <= 1024, "whole warps");
  constexpr int NW = T / 32;
  __shared__ float red_s[6][NW];  // hi, lo of f_eta, f_ch, mass per warp
  __shared__ float red_m[4][NW];
  __shared__ int red_i[NW];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const FF s0 = warp_sum_ff(ff(acc.feta.x + acc.feta.y)), s1 = warp_sum_ff(ff(acc.fch.x + acc.fch.y)),
           s2 = warp_sum_ff(acc.mass());
  const float m0 = warp_min(acc.cmin), m1 = warp_max(acc.cmax), m2 = warp_min(acc.phimin), m3 = warp_max(acc.phipmax);
  const int nb = __reduce_add_sync(0xffffffffu, acc.nonfinite);
  if (lane == 0) {
    red_s[0][wid] = s0.hi; red_s[1][wid] = s0.lo; red_s[2][wid] = s1.hi; red_s[3][wid] = s1.lo;
    red_s[4][wid] = s2.hi; red_s[5][wid] = s2.lo;
    red_m[0][wid] = m0; red_m[1][wid] = m1; red_m[2][wid] = m2; red_m[3][wid] = m3;
    red_i[wid] = nb;
  }
  __syncthreads();
  if (wid == 0) {  // the warps' values, one per lane (the reference's start values as identities)
    const bool in = lane < NW;
    const FF a0 = warp_sum_ff(in ? ff(red_s[0][lane], red_s[1][lane]) : ff(0.f));
    const FF a1 = warp_sum_ff(in ? ff(red_s[2][lane], red_s[3][lane]) : ff(0.f));
    const FF a2 = warp_sum_ff(in ? ff(red_s[4][lane], red_s[5][lane]) : ff(0.f));
    const float b0 = warp_min(in ? red_m[0][lane] : 1.f), b1 = warp_max(in ? red_m[1][lane] : 0.f);
    const float b2 = warp_min(in ? red_m[2][lane] : 1.f), b3 = warp_max(in ? red_m[3][lane] : 0.f);
    const int nn = __reduce_add_sync(0xffffffffu, in ? red_i[lane] : 0);
    if (lane == 0) {
      const int nbk = sh.nblk_x;
      float* p = rp.part_x + (size_t)sh.par * XQ_COUNT * nbk + blk;
      p[XQ_FETA_H * nbk] = a0.hi; p[XQ_FETA_L * nbk] = a0.lo;
      p[XQ_FCH_H * nbk] = a1.hi;  p[XQ_FCH_L * nbk] = a1.lo;
      p[XQ_MASS_H * nbk] = a2.hi; p[XQ_MASS_L * nbk] = a2.lo;
      p[XQ_CMIN * nbk] = b0;
      p[XQ_CMAX * nbk] = b1;
      p[XQ_PHIMIN * nbk] = b2;
      p[XQ_PHIPMAX * nbk] = b3;
      p[XQ_BAD * nbk] = (float)nn;
    }
  }
}

// Bulk terms of one tile (WY rows of every field in shared memory), one
// float2 slot (two cells) per item.
template <int NX, int WY, int T>
__device__ __forceinline__ void bulk_tile(float2* smem, const RunParams& rp, const Shape& sh, int z, int y0,
                                          BulkAcc& acc) {
  constexpr int M = NX / 2, PM = XLine<M>::PITCH;
  for (int it = threadIdx.x; it < WY * M; it += T) {
    const int m = it % M, yy = it / M;
    float2 dfdc, mob;
    bulk_slot<PM, WY>(smem, yy, m, rp, dfdc, mob, acc);
    smem[(rp.V * WY + yy) * PM + m] = dfdc;
    if (rp.mobility != MOB_CONST)
      *reinterpret_cast<float2*>(rp.mob + ((size_t)z * sh.Ny + y0 + yy) * NX + 2 * m) = mob;
  }
}

// ---------------------------------------------------------------------------
// x pass.  MODE_BULK: S -> D (+ mob, diagnostics).  MODE_XJ: J~ -> J~' with the
// variable-mobility multiply (:947-965).  MODE_IMPORT: the caller's fields
// (phi(var, x, y, z) and con, REAL*8) -> S.  MODE_EXPORT: S -> the caller's
// fields.  MODE_FIELDS: S -> float fields [f][z][y][x].
// A tile's rows are one contiguous piece of the caller's layout, so import and
// export read and write it in full lines straight from and to shared memory --
// in the host's own memory where the GPU reaches that at the link's full rate
// (NVLink-C2C: kernels move 210 GB/s in and 193 out, as copies do).
// ---------------------------------------------------------------------------
enum XMode { MODE_BULK = 0, MODE_XJ = 1, MODE_IMPORT = 2, MODE_EXPORT = 3, MODE_FIELDS = 4 };

// Walk over the cells of a tile in the caller's layout: op(value in memory,
// its place in the tile's lines) for phi (field fastest), then con.
template <int NX, int WY, int T, class Op>
__device__ __forceinline__ void walk_tile(float2* smem, const Shape& sh, int V, size_t cell0, Op op) {
  using LM = XLine<NX / 2>;
  float* lines = reinterpret_cast<float*>(smem);
  const auto place = [&](int f, int cell) {
    const int yy = cell / NX, x = cell % NX;
    return lines + 2 * ((f * WY + yy) * LM::PITCH + (x >> 1)) + (x & 1);
  };
  const FastDiv by_v(V);
  double* phi = sh.io_phi + cell0 * V;
#pragma unroll 4
  for (int it = threadIdx.x; it < WY * NX * V; it += T) {
    const int cell = by_v(it);
    op(phi + it, place(it - cell * V, cell));
  }
  double* con = sh.io_con + cell0;
  for (int it = threadIdx.x; it < WY * NX; it += T) op(con + it, place(V, it));
}

__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
}
// ASYNC: the tile's half spectra are copied into the line buffer by cp.async
// (all of them in flight at once, no registers held) in the in-place slot
// order, and the inverse transform then runs in place; otherwise each item
// loads its own inputs from global memory.
template <int NX, int WY, int T, int MODE, bool ASYNC = false, int MINB = 0>
__global__ void __launch_bounds__(T, MINB) x_pass_kernel(const RunParams* __restrict__ runs, const Shape sh) {
  constexpr int M = NX / 2;
  using LM = XLine<M>;
  constexpr int PM = LM::PITCH;
  constexpr int NP = LM::N2 / 2 + 1;  // run pairs per line
  // run pairs (pr, N2 - pr) for 0 < pr < N2/2, run 0 alone, and for even N2
  // the run N2/2 paired with itself (x_inv_runs / x_fwd_runs)
  extern __shared__ float2 smem[];
  // The twiddle tables W_NX^j and W_M^j, read by every run and pass-A item:
  // copied to shared memory from Nx = 96 up.  There a CTA's tile of every
  // field leaves room for one or two CTAs per SM, so the extra registers the
  // compiler then spends on early twiddle loads cost no occupancy (x pass
  // 0.129 -> 0.124 ms at 128^3 x 16, 2.67 -> 2.59 ms at 256^3 x 32); the
  // small grids' tiles fit more CTAs than those registers would.
  constexpr bool TWS = NX >= 96;
  __shared__ float2 stwN[TWS ? NX : 1], stwM[TWS ? M : 1];
  if constexpr (TWS) {
    for (int j = threadIdx.x; j < NX; j += T) stwN[j] = __ldg(sh.twN + j);
    for (int j = threadIdx.x; j < M; j += T) stwM[j] = __ldg(sh.twM + j);
    __syncthreads();
  }
  const float2* twN = TWS ? stwN : sh.twN;
  const float2* twM = TWS ? stwM : sh.twM;
  const RunParams& rp = runs[blockIdx.y];
  const int nF = (MODE == MODE_XJ) ? 1 : rp.V + 1;
  const FastDiv by_line(nF * WY);
  const int ny_tiles = sh.Ny / WY;
  const int z = blockIdx.x / ny_tiles;
  const int y0 = (blockIdx.x - z * ny_tiles) * WY;
  const int ks = sh.ks;
  const size_t fstride = (size_t)sh.Kx * sh.Nz * sh.Ny;
  const int row_off = z * sh.zs + y0;
  const float2* __restrict__ src = (MODE == MODE_XJ) ? rp.J : rp.Sm;

  if (MODE == MODE_IMPORT) {
    walk_tile<NX, WY, T>(smem, sh, rp.V, (size_t)(z * sh.Ny + y0) * NX,
                         [](const double* v, float* at) { *at = (float)*v; });
  } else {
    // 1. inverse x transform: global half spectrum -> pre-processing -> pass B'
    // a warp covers consecutive (y row, field) lines at one run pair: the
    // global reads are y-contiguous and the line offsets hit distinct banks
    if constexpr (ASYNC) {
      constexpr int KX = M + 1;
      // consecutive threads copy consecutive rows of one (field, kx): 64-byte
      // runs of global memory, destination lines PM apart (distinct banks)
      for (int it = threadIdx.x; it < nF * KX * WY; it += T) {
        const int yy = it % WY, r = it / WY, kx = r % KX, f = r / KX;
        cp_async8(smem + (f * WY + yy) * PM + x_spec_slot<M>(kx),
                  src + f * fstride + (kx * ks + row_off + yy));
      }
      cp_async_wait_all();
      __syncthreads();
      for (int it = threadIdx.x; it < nF * WY * NP; it += T) {
        const int q = by_line(it), l = it - q * (nF * WY), pr = x_run_pair<M>(q);
        x_inv_runs<M, SPEC_INPLACE, TWS>(smem + l * PM, 0, smem + l * PM, pr, twN);
      }
    } else {
      for (int it = threadIdx.x; it < nF * WY * NP; it += T) {
        const int q = by_line(it), l = it - q * (nF * WY), pr = x_run_pair<M>(q);
        const int f = l / WY, yy = l - f * WY;
        x_inv_runs<M, SPEC_GLOBAL, TWS>(src + f * fstride + row_off + yy, ks, smem + l * PM, pr, twN);
      }
    }
    __syncthreads();
    passA_rt<M, PM, T, true, TWS>(smem, nF * WY, twM);
  }
  __syncthreads();

  if (MODE == MODE_EXPORT) {
    walk_tile<NX, WY, T>(smem, sh, rp.V, (size_t)(z * sh.Ny + y0) * NX,
                         [](double* v, const float* at) { *v = (double)*at; });
    return;
  }
  if (MODE == MODE_FIELDS) {
    for (int it = threadIdx.x; it < nF * WY * M; it += T) {
      const int m = it % M, r = it / M, yy = r % WY, f = r / WY;
      *reinterpret_cast<float2*>(sh.fin + (((size_t)f * sh.Nz + z) * sh.Ny + y0 + yy) * NX + 2 * m) =
          smem[(f * WY + yy) * PM + m];
    }
    return;
  }

  BulkAcc acc;
  acc.init();

  if (MODE == MODE_BULK) {
    // 2. bulk terms, two cells per slot
    bulk_tile<NX, WY, T>(smem, rp, sh, z, y0, acc);
    __syncthreads();
  } else if (MODE == MODE_XJ) {
    for (int it = threadIdx.x; it < WY * M; it += T) {
      const int m = it % M, yy = it / M;
      const int slot = m;
      const float2 mb = *reinterpret_cast<const float2*>(rp.mob + ((size_t)z * sh.Ny + y0 + yy) * NX + 2 * m);
      float2 v = smem[yy * PM + slot];
      v.x *= mb.x;
      v.y *= mb.y;
      smem[yy * PM + slot] = v;
    }
    __syncthreads();
  }

  // 3. forward x transform: pass A, then pass B + post-processing -> global
  passA_rt<M, PM, T, false, TWS>(smem, nF * WY, twM);
  __syncthreads();
  float2* __restrict__ dst = (MODE == MODE_BULK) ? rp.D : (MODE == MODE_XJ ? rp.J : rp.Sm);
  for (int it = threadIdx.x; it < nF * WY * NP; it += T) {
    const int q = by_line(it), l = it - q * (nF * WY), pr = x_run_pair<M>(q);
    const int f = l / WY, yy = l - f * WY;
    x_fwd_runs<M, MODE == MODE_IMPORT, TWS>(dst + f * fstride + row_off + yy, ks, smem + l * PM, pr, twN);
  }

  if (MODE != MODE_BULK) return;

  // 6. diagnostics: block reduction into per-block partials
  store_block_diag<T>(acc, rp, sh, blockIdx.x);
}


// ---------------------------------------------------------------------------
// yz pass.  The state of every field is kept in full k-space,
//     Sk[f][kx][kz][ypos] = u_hat (normalised like f_trans, src/f_trans.f90:12),
// y in the digit-transposed position order of its transform, and is
// updated pointwise there (exact increment, no FFT round trip of the state).
// Per (field, kx) plane the yz pass
//   * transforms D~ (the x pass output, mixed space) forward over y and z,
//   * forms u_hat_new = u_hat + m1 u_hat + m2 D_hat (semi-implicit update),
//   * transforms u_hat_new back over z and y to the mixed-space field the next
//     x pass reads (Sm).
// Two kernels do it: yz1_kernel, one CTA per plane, one transform stage per
// pass over shared memory; and yz_kernel, stages of y and z in one pass and a
// cluster of CTAs where a plane is shared.  All loops have compile-time trip counts.
// ---------------------------------------------------------------------------
enum YZMode { YZ_MAIN = 0, YZ_C2 = 1, YZ_IMPORT = 2 };

// ---------------------------------------------------------------------------
// Pointwise semi-implicit update of one k-point, shared by both yz kernels.
// The reference's forms (var_diff.f90 lines cited at the call sites)
//   AC: u += (-L dt kappa q^2 u - L dt D) / (1 + L dt kappa q^2)
//   CH: c += (-D dt kappa_c K4 c - D dt q^2 mu) / (1 + D dt kappa_c K4)
// are evaluated as u' = u - (t u + b D) / (1 + t), t = a Q, Q = q^2 (AC) or
// K4 (CH), with the 1/(NY NZ) normalisation of the transform folded into b.
// The increment is formed first and added to u, as in the reference: the
// rounding of the (fast, about 2 ulp) reciprocal then scales only the
// increment, so low modes, whose factor is close to 1, do not drift by a
// fixed relative bias per step.  The kz factors come from a shared-memory
// table {qz^2, qz^4, qn_z, qn_z^2} staged once per CTA.
// ---------------------------------------------------------------------------
template <int NZ, int T>
__device__ __forceinline__ void stage_kz(float4* qt, const Shape& sh) {
  for (int k = threadIdx.x; k < NZ; k += T) {
    const float n = __ldg(sh.qnz + k);
    qt[k] = make_float4(__ldg(sh.qz2 + k), __ldg(sh.qz4 + k), n, n * n);
  }
}

// Normalisation of what a yz pass transforms: over y and z, and over x where
// the x pass has left that to it (x_fwd_runs).
template <int MODE>
__device__ __forceinline__ float yz_norm(int nyz, int nx) {
  return 1.0f / ((float)nyz * (MODE == YZ_IMPORT ? 1.0f : 2.0f * (float)nx));
}

struct KPlane {
  float qx2, qx4, qnx;
  float a;    // t = a Q
  float b;    // coefficient of the driving term, normalisation included
  float nrm;  // normalisation of the transforms
  float kc;   // kappa_c
  __device__ __forceinline__ KPlane(const RunParams& rp, const Shape& sh, int kx, int mode, bool is_c, float nrm_) {
    qx2 = sh.qx2[kx];
    qx4 = sh.qx4[kx];
    qnx = sh.qnx[kx];
    nrm = nrm_;
    kc = rp.kappa_c;
    if (mode == YZ_MAIN && !is_c) {
      a = rp.L * rp.dt * rp.kappa_phi;
      b = rp.L * rp.dt * nrm_;
    } else {
      a = rp.D_L * rp.dt * rp.kappa_c;
      b = (mode == YZ_MAIN ? rp.D_L * rp.dt : rp.dt) * nrm_;
    }
  }
};

// the kx + ky parts of the k-point factors of one y position
struct KRow {
  float q2, q4, n2, g, k3;
  __device__ __forceinline__ KRow(const KPlane& P, const Shape& sh, int ky) {
    const float qy2 = __ldg(sh.qy2 + ky), qy4 = __ldg(sh.qy4 + ky), qny = __ldg(sh.qny + ky);
    q2 = P.qx2 + qy2;
    q4 = P.qx4 + qy4;
    n2 = fmaf(P.qnx, P.qnx, qny * qny);
    g = P.qnx + qny;
    k3 = fmaf(P.qnx, P.qx2, qny * qy2);
  }
};

// u: the k-space state (in: old, out: new); d: the unnormalised transform of
// the driving term (MAIN: dF/dphi or mu; C2: J'), on return J_hat where the
// c plane of a variable-mobility run hands it to the inverse transform.
template <int MODE>
__device__ __forceinline__ void kpoint(const KPlane& P, const KRow& R, const float4 z, const bool is_c, const bool var_c,
                                       float2& u, float2& d, float& fint) {
  if (MODE == YZ_IMPORT) {
    u = make_float2(d.x * P.nrm, d.y * P.nrm);
    return;
  }
  const float2 uu = u;
  const float q2 = R.q2 + z.x;
  if (MODE == YZ_MAIN) {
    // f_int by Parseval: |kf|^2 |u_hat|^2
    fint = fmaf(R.n2 + z.w, fmaf(uu.x, uu.x, uu.y * uu.y), fint);
    if (!is_c) {
      // AC (:1015-1024)
      const float t = P.a * q2;
      const float inv = __fdividef(1.0f, 1.0f + t);
      const float ix = fmaf(t, uu.x, P.b * d.x), iy = fmaf(t, uu.y, P.b * d.y);
      u = make_float2(fmaf(-ix, inv, uu.x), fmaf(-iy, inv, uu.y));
    } else {
      // CH (:976-983), K2 = -q^2
      const float t = P.a * (R.q4 + z.y);
      const float inv = __fdividef(1.0f, 1.0f + t);
      const float bq = P.b * q2;
      const float ix = fmaf(t, uu.x, bq * d.x), iy = fmaf(t, uu.y, bq * d.y);
      u = make_float2(fmaf(-ix, inv, uu.x), fmaf(-iy, inv, uu.y));
      if (var_c) {
        // J_hat = G mu_hat - kappa_c c_hat K3 (:932-935), G = i g, K3 = -i (qn . q^2)
        const float gn = (R.g + z.z) * P.nrm;
        const float kk = P.kc * fmaf(z.z, z.x, R.k3);
        d = cmul_pi(make_float2(fmaf(gn, d.x, kk * uu.x), fmaf(gn, d.y, kk * uu.y)));
      }
    }
  } else {
    // C2: c += dt G J'_hat / (1 + D dt kappa_c K4)  (:976)
    const float sg = __fdividef(P.b * (R.g + z.z), fmaf(P.a, R.q4 + z.y, 1.0f));
    u = cadd(uu, cmul_pi(make_float2(d.x * sg, d.y * sg)));
  }
}

// One run of N1 positions of a z line: last forward pass, update, first inverse
// pass.  d: the run of the driving term (in), of the new field or J (out);
// gk: its k-space state, element k1 at gk[k1 * SK1], read UC at a time.
template <int N1, int N2, int MODE, int UC>
__device__ __forceinline__ void update_run(float2 (&d)[N1], float2* __restrict__ gk, size_t SK1, const KPlane& P,
                                           const KRow& R, const float4* qz, const bool is_c, const bool var_c,
                                           float& fint) {
  float2 u[UC];
  if (MODE != YZ_IMPORT) {
#pragma unroll
    for (int j = 0; j < UC; ++j) u[j] = gk[j * SK1];
  }
  Dft<N1>::fwd(d);
#pragma unroll
  for (int k0 = 0; k0 < N1; k0 += UC) {
    if (MODE != YZ_IMPORT && k0 > 0) {
#pragma unroll
      for (int j = 0; j < UC; ++j)
        if (k0 + j < N1) u[j] = gk[(k0 + j) * SK1];
    }
#pragma unroll
    for (int j = 0; j < UC; ++j) {
      const int k1 = k0 + j;
      if (k1 < N1) {
        kpoint<MODE>(P, R, qz[N2 * k1], is_c, var_c, u[j], d[k1], fint);
        gk[k1 * SK1] = u[j];
        if (!var_c) d[k1] = u[j];
      }
    }
  }
  if (MODE != YZ_IMPORT) dft_inv<N1>(d);
}

// ---------------------------------------------------------------------------
// The step's record (src/var_diff.f90:1058-1118): one CTA per run reduces the
// x-pass partials and the yz pass's f_int partials in a fixed order (the same
// bits whichever other runs share the launch), writes the record into the
// ring and advances the step counter.  Sums are compensated FP32 pairs up to
// the warp totals; the mass is then summed over the warps in FP64 with
// compensation (KSum).  A separate launch, not the last CTA of the yz pass:
// the fence a CTA needs before announcing its partial holds that CTA (and the
// SM's next one) until all of its stores have drained.
// ---------------------------------------------------------------------------
template <int T>
__global__ void __launch_bounds__(T) record_kernel(const RunParams* __restrict__ runs, const Shape sh) {
  static_assert(T % 32 == 0 && T <= 1024, "whole warps");
  constexpr int NW = T / 32;
  __shared__ float sd[10][NW];  // hi, lo of f_eta, f_ch, mass, f_int (order parameters), f_int (c)
  __shared__ float sf[4][NW];
  __shared__ int si[NW];
  const RunParams& rp = runs[blockIdx.x];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int nb = sh.nblk_x;
  const float* __restrict__ px = rp.part_x + (size_t)sh.par * XQ_COUNT * sh.nblk_x;
  FF eta = ff(0.f), ch = ff(0.f), mass = ff(0.f), fphi = ff(0.f), fc = ff(0.f);
  float cmin = 1.f, cmax = 0.f, pmin = 1.f, ppmax = 0.f;  // reference start values (:1076-1079)
  int bad = 0;
  for (int i = t; i < nb; i += T) {
    eta.add(ff(__ldcg(px + XQ_FETA_H * nb + i), __ldcg(px + XQ_FETA_L * nb + i)));
    ch.add(ff(__ldcg(px + XQ_FCH_H * nb + i), __ldcg(px + XQ_FCH_L * nb + i)));
    mass.add(ff(__ldcg(px + XQ_MASS_H * nb + i), __ldcg(px + XQ_MASS_L * nb + i)));
    cmin = fminf(cmin, __ldcg(px + XQ_CMIN * nb + i));
    cmax = fmaxf(cmax, __ldcg(px + XQ_CMAX * nb + i));
    pmin = fminf(pmin, __ldcg(px + XQ_PHIMIN * nb + i));
    ppmax = fmaxf(ppmax, __ldcg(px + XQ_PHIPMAX * nb + i));
    bad += (int)__ldcg(px + XQ_BAD * nb + i);
  }
  // f_int partials: the last nblk_yz / nF slots belong to the c planes
  const int nyz = sh.nblk_yz, cstart = nyz - nyz / (rp.V + 1);
  const float* __restrict__ pyz = rp.part_yz + (size_t)sh.par * 2 * nyz;
  for (int i = t; i < nyz; i += T) {
    const FF v = ff(__ldcg(pyz + i), __ldcg(pyz + nyz + i));
    if (i < cstart) fphi.add(v);
    else fc.add(v);
  }
  eta = warp_sum_ff(eta); ch = warp_sum_ff(ch); mass = warp_sum_ff(mass);
  fphi = warp_sum_ff(fphi); fc = warp_sum_ff(fc);
  cmin = warp_min(cmin); cmax = warp_max(cmax); pmin = warp_min(pmin); ppmax = warp_max(ppmax);
  bad = __reduce_add_sync(0xffffffffu, bad);
  if (lane == 0) {
    sd[0][w] = eta.hi; sd[1][w] = eta.lo; sd[2][w] = ch.hi; sd[3][w] = ch.lo; sd[4][w] = mass.hi; sd[5][w] = mass.lo;
    sd[6][w] = fphi.hi; sd[7][w] = fphi.lo; sd[8][w] = fc.hi; sd[9][w] = fc.lo;
    sf[0][w] = cmin; sf[1][w] = cmax; sf[2][w] = pmin; sf[3][w] = ppmax;
    si[w] = bad;
  }
  __syncthreads();
  if (w == 0) {
    const bool in = lane < NW;
    const FF e = warp_sum_ff(in ? ff(sd[0][lane], sd[1][lane]) : ff(0.f));
    const FF c = warp_sum_ff(in ? ff(sd[2][lane], sd[3][lane]) : ff(0.f));
    const FF a = warp_sum_ff(in ? ff(sd[6][lane], sd[7][lane]) : ff(0.f));
    const FF b = warp_sum_ff(in ? ff(sd[8][lane], sd[9][lane]) : ff(0.f));
    // mass: the warps' compensated sums in FP64, combined with compensation
    KSum m;
    if (in) m.add(ff(sd[4][lane], sd[5][lane]).value());
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      KSum other;
      other.s = __shfl_xor_sync(0xffffffffu, m.s, o);
      other.c = __shfl_xor_sync(0xffffffffu, m.c, o);
      m.add(other);
    }
    const float m0 = warp_min(in ? sf[0][lane] : 1.f), m1 = warp_max(in ? sf[1][lane] : 0.f);
    const float m2 = warp_min(in ? sf[2][lane] : 1.f), m3 = warp_max(in ? sf[3][lane] : 0.f);
    const int nbad = __reduce_add_sync(0xffffffffu, in ? si[lane] : 0);
    if (lane == 0) {
      const int step = *rp.counter;
      const double n3 = (double)sh.Nx * sh.Ny * sh.Nz;
      const double fint = 0.5 * n3 * ((double)rp.kappa_phi * a.value() + (double)rp.kappa_c * b.value());
      const double mass = m.value();
      // to the host as well where it keeps a ring: pf_step then needs no copy
      for (double* ring : {rp.diag, rp.hdiag}) {
        if (!ring) break;
        double* d = ring + (size_t)(step % rp.ring) * DR_COUNT;
        d[DR_STEP] = step + 1;
        d[DR_FINT] = fint;
        d[DR_FETA] = e.value();
        d[DR_FCH] = c.value();
        d[DR_CMIN] = m0;
        d[DR_CMAX] = m1;
        d[DR_PHIMIN] = m2;
        d[DR_PHIPMAX] = m3;
        d[DR_MASS] = mass;
        d[DR_NONFINITE] = nbad;
      }
      *rp.counter = step + 1;
    }
  }
}

// Store this CTA's f_int partial -- w times the sum of the per-thread FP32
// sums of |kf|^2 |u_hat|^2 (w = 2 for the kx planes that stand for their
// conjugates, else 1) -- as a compensated pair in slot `slot`.
template <int T>
__device__ __forceinline__ void yz_finish(const RunParams& rp, const Shape& sh, float fint, float w, size_t slot) {
  constexpr int NW = T / 32;
  __shared__ float red[2][NW];
  const FF v = warp_sum_ff(ff(fint * w));
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) {
    red[0][wid] = v.hi;
    red[1][wid] = v.lo;
  }
  __syncthreads();
  if (wid == 0) {
    const FF s = warp_sum_ff(lane < NW ? ff(red[0][lane], red[1][lane]) : ff(0.f));
    if (lane == 0) {
      float* pyz = rp.part_yz + (size_t)sh.par * 2 * sh.nblk_yz;
      pyz[slot] = s.hi;
      pyz[sh.nblk_yz + slot] = s.lo;
    }
  }
}

__device__ __forceinline__ void cluster_barrier() { cg::this_cluster().sync(); }

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t map_rank(uint32_t a, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ float2 ld_peer(uint32_t a) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
  return v;
}

__device__ __forceinline__ void st_peer(uint32_t a, float2 v) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}

// run pass (forward or inverse) over NL lines of length L, pitch P, T threads
template <int L, int NL, int P, int T, bool INV>
__device__ __forceinline__ void passB(float2* buf) {
  constexpr int N1 = Line<L>::N1, N2 = Line<L>::N2;
  constexpr int ITEMS = NL * N2, ITER = (ITEMS + T - 1) / T;
#pragma unroll
  for (int j = 0; j < ITER; ++j) {
    const int it = threadIdx.x + j * T;
    if (ITEMS % T != 0 && it >= ITEMS) break;
    const int l = it / N2, k2 = it - l * N2;  // k2 is fixed per thread when N2 divides T
    float2* p = buf + l * P + k2 * (N1 + 1);
    float2 u[N1];
#pragma unroll
    for (int n1 = 0; n1 < N1; ++n1) u[n1] = p[n1];
    if (INV) dft_inv<N1>(u); else Dft<N1>::fwd(u);
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1) p[k1] = u[k1];
  }
}

// ---------------------------------------------------------------------------
// Single-CTA yz pass for planes that fit one CTA's shared memory: the plane
// stays in one buffer U[z][phys_y(y)] (row pitch PY, odd); y transforms run
// along rows, z transforms down columns (consecutive threads take consecutive
// y positions, so column accesses are conflict-free).  No re-layout, no
// cluster.  Same k-space position order as yz_kernel.
// ---------------------------------------------------------------------------
// Row pitch: the odd line pitch, or (RAWP) the unpadded run layout
// N2 (N1 + 1).  yz1 reads columns with lanes along y, so only its row passes
// see the pitch: a warp covers two rows (first/last y pass) or 32/N2 rows of
// N2 runs (pass B); with N2 (N1 + 1) = 8 (mod 16) float2 the rows of a half
// warp fall in disjoint bank pairs (128 x 128: no conflicts, against one
// extra wavefront in four at the odd pitch).
template <int NY, int NZ, bool RAWP = false>
struct YZ1 {
  static constexpr int PY = RAWP ? Line<NY>::RAW : Line<NY>::PITCH;
  static constexpr size_t SMEM = (size_t)NZ * PY * sizeof(float2);
};

// column pass A (forward or inverse) over the NY y positions.  Where the CTA's
// warps are a multiple of N1 a warp keeps one column n1 and loads its twiddles
// once (as broadcast loads of every item they were 7 of 23 shared wavefronts).
template <int NY, int NZ, int T, bool INV, bool RAWP, bool TWS = false>
__device__ __forceinline__ void colA(float2* U, const float2* __restrict__ tw) {
  constexpr int N1 = Line<NZ>::N1, N2 = Line<NZ>::N2, PY = YZ1<NY, NZ, RAWP>::PY, NW = T / 32;
  if constexpr (NW % N1 == 0) {
    const int w = threadIdx.x >> 5, n1 = w % N1;
    float2 wt[N2];
#pragma unroll
    for (int k2 = 1; k2 < N2; ++k2) wt[k2] = ldtw<TWS>(tw + n1 * k2);
#pragma unroll 1
    for (int yp = (w / N1) * 32 + (threadIdx.x & 31); yp < NY; yp += 32 * (NW / N1))
      passA_item<N1, N2, N1 * PY, INV>(U + n1 * PY + Line<NY>::phys(yp), [&](int k2) { return wt[k2]; });
  } else {
    constexpr int ITEMS = NY * N1, ITER = (ITEMS + T - 1) / T;
#pragma unroll 1
    for (int j = 0; j < ITER; ++j) {
      const int it = threadIdx.x + j * T;
      if (ITEMS % T != 0 && it >= ITEMS) break;
      const int yp = it % NY, n1 = it / NY;
      passA_item<N1, N2, N1 * PY, INV>(U + n1 * PY + Line<NY>::phys(yp), [&](int k2) { return ldtw<TWS>(tw + n1 * k2); });
    }
  }
}

template <int NY, int NZ, int T, int MODE, bool RAWP = false, int MINB = 0, int UC = Line<NZ>::N1>
__global__ void __launch_bounds__(T, MINB) yz1_kernel(const RunParams* __restrict__ runs, const Shape sh) {
  using LY = Line<NY>;
  using LZ = Line<NZ>;
  constexpr int N1y = LY::N1, N2y = LY::N2, N1z = LZ::N1, N2z = LZ::N2;
  constexpr int PY = YZ1<NY, NZ, RAWP>::PY;
  static_assert(T % 32 == 0, "whole warps");
  extern __shared__ float2 U[];
  __shared__ float4 qzt[NZ];  // kz factors of the k-space update
  stage_kz<NZ, T>(qzt, sh);   // read after the barriers of the forward passes
  // the z twiddles of the column passes in shared memory from 128 x 128 planes
  // up (one CTA per SM there: the registers of early loads cost no occupancy)
  constexpr bool TWS = NY >= 128;
  __shared__ float2 stwZ[TWS ? NZ : 1];
  if constexpr (TWS)
    for (int j = threadIdx.x; j < NZ; j += T) stwZ[j] = __ldg(sh.twZ + j);  // read after the first barrier
  const float2* twZ = TWS ? stwZ : sh.twZ;
  const RunParams& rp = runs[blockIdx.y];
  const int p = sh.plane0 + (int)blockIdx.x;
  const int Kx = sh.Kx;
  const int f = (MODE == YZ_C2) ? rp.V : p / Kx;
  const int kx = p - (p / Kx) * Kx;
  const size_t plane_elems = (size_t)NZ * NY;
  const size_t poff = ((size_t)f * Kx + kx) * plane_elems;          // k-space state
  const size_t moff = (size_t)f * Kx * plane_elems + kx * sh.ks;  // mixed space
  const bool is_c = (f == rp.V);
  const bool var_c = (MODE == YZ_MAIN) && is_c && rp.mobility != MOB_CONST;

  // 1. forward y transform of all NZ rows, first pass straight from global
  {
    const float2* src = (MODE == YZ_MAIN) ? rp.D + moff : (MODE == YZ_C2 ? rp.J + kx * sh.ks : rp.Sm + moff);
    // twiddles: preloaded when every iteration of a thread has the same n1
    constexpr bool FIXED = (T % N1y) == 0;
    float2 wt[N2y];
    if constexpr (FIXED) {
#pragma unroll
      for (int k2 = 1; k2 < N2y; ++k2) wt[k2] = __ldg(sh.twY + (threadIdx.x % N1y) * k2);
    }
    constexpr int ITEMS = NZ * N1y, ITER = (ITEMS + T - 1) / T;
#pragma unroll 4
    for (int j = 0; j < ITER; ++j) {
      const int it = threadIdx.x + j * T;
      if (ITEMS % T != 0 && it >= ITEMS) break;
      const int z = it / N1y, n1 = it - z * N1y;
      const float2* s = src + z * sh.zs + n1;
      float2 v[N2y];
#pragma unroll
      for (int n2 = 0; n2 < N2y; ++n2) v[n2] = __ldg(s + n2 * N1y);
      Dft<N2y>::fwd(v);
      float2* d = U + z * PY + n1;
      d[0] = v[0];
#pragma unroll
      for (int k2 = 1; k2 < N2y; ++k2) d[k2 * (N1y + 1)] = cmul(v[k2], FIXED ? wt[k2] : __ldg(sh.twY + n1 * k2));
    }
  }
  __syncthreads();
  passB<NY, NZ, PY, T, false>(U);
  __syncthreads();
  colA<NY, NZ, T, false, RAWP, TWS>(U, twZ);
  __syncthreads();
  // 2. last forward z pass, pointwise k-space update, first inverse z pass
  const KPlane P(rp, sh, kx, MODE, is_c, yz_norm<MODE>(NY * NZ, sh.Nx));
  const float wkx = (kx == 0 || 2 * kx == sh.Nx) ? 1.0f : 2.0f;
  float fint = 0.f;
  {
    constexpr int ITEMS = NY * N2z, ITER = (ITEMS + T - 1) / T;
#pragma unroll 1
    for (int j = 0; j < ITER; ++j) {
      const int it = threadIdx.x + j * T;
      if (ITEMS % T != 0 && it >= ITEMS) break;
      const int yp = it % NY, k2 = it / NY;
      const KRow R(P, sh, LY::freq_of_pos(yp));
      float2* pc = U + (k2 * N1z) * PY + LY::phys(yp);
      // k-space state of this plane in [k1][k2][y position] order: for every
      // k1 a warp reads and writes 32 consecutive y positions (coalesced)
      float2* gk = rp.Sk + poff + it;  // it == k2 NY + yp
      constexpr size_t SK1 = (size_t)N2z * NY;  // stride of k1
      float2 d[N1z];
#pragma unroll
      for (int k1 = 0; k1 < N1z; ++k1) d[k1] = pc[k1 * PY];
      update_run<N1z, N2z, MODE, UC>(d, gk, SK1, P, R, qzt + k2, is_c, var_c, fint);
      if (MODE != YZ_IMPORT) {
#pragma unroll
        for (int k1 = 0; k1 < N1z; ++k1) pc[k1 * PY] = d[k1];
      }
    }
  }
  if (MODE == YZ_IMPORT) return;
  __syncthreads();
  colA<NY, NZ, T, true, RAWP, TWS>(U, twZ);
  __syncthreads();
  passB<NY, NZ, PY, T, true>(U);
  __syncthreads();

  // 3. last inverse y pass straight to the mixed-space output
  {
    const bool real_plane = (kx == 0) || (2 * kx == sh.Nx);  // the x-DFT of real data is real there
    float2* dst = var_c ? rp.J + kx * sh.ks : rp.Sm + moff;
    constexpr bool FIXED = (T % N1y) == 0;
    float2 wt[N2y];
    if constexpr (FIXED) {
#pragma unroll
      for (int k2 = 1; k2 < N2y; ++k2) wt[k2] = __ldg(sh.twY + (threadIdx.x % N1y) * k2);
    }
    constexpr int ITEMS = NZ * N1y, ITER = (ITEMS + T - 1) / T;
#pragma unroll 4
    for (int j = 0; j < ITER; ++j) {
      const int it = threadIdx.x + j * T;
      if (ITEMS % T != 0 && it >= ITEMS) break;
      const int z = it / N1y, n1 = it - z * N1y;
      const float2* sp = U + z * PY + n1;
      float2 v[N2y];
      v[0] = sp[0];
#pragma unroll
      for (int k2 = 1; k2 < N2y; ++k2) v[k2] = cmulc(sp[k2 * (N1y + 1)], FIXED ? wt[k2] : __ldg(sh.twY + n1 * k2));
      dft_inv<N2y>(v);
      float2* o = dst + z * sh.zs + n1;
#pragma unroll
      for (int n2 = 0; n2 < N2y; ++n2) {
        float2 x = v[n2];
        if (real_plane && !var_c) x.y = 0.f;
        o[n2 * N1y] = x;
      }
    }
  }

  if (MODE == YZ_MAIN) {
    yz_finish<T>(rp, sh, fint, wkx, (size_t)p);
  }
}

// ---------------------------------------------------------------------------
// Yz pass whose register passes take stages of both axes, with C CTAs (a
// cluster) per plane.  z = t + N1 s: a run is the N1 points t of one frequency
// of s, the s transform has Q = ZA ZB ZP points.  CTA r holds the z rows
// z = r (mod C), whole rows of y, so every stage but the last is its own:
//   P1  N2y points of y (stride N1y) x ZA of z, straight from global memory,
//   P2  a run of N1y points of y x ZB of z,
//   P3  ZP points of z (left out where ZP = 1),
//   P4  a run: last forward stage, update, first inverse.
// and P3, P2, P1 again for the inverse.  A run's points t lie t mod C over the
// cluster, ZL = N1/C in each CTA: P4 reads them from there, and puts them back
// there.  Every stage works in place: s frequency kb + ZA ka + ZA ZB kp is found
// at rows ZL (kp + ZP (ka + ZB kb)) on.  The k-space order is yz1_kernel's.
//
// Against re-laying the plane out over the cluster before and after the z
// transform (each way a pass and two cluster barriers of its own): two cluster
// barriers instead of five, 12 crossings of shared memory instead of 16, and a
// P4 that hides the peers' latency behind the state's loads.  Yz pass of 33
// fields of 256^3 3340 -> 2584 us, of 7 of 200^3 433 -> 302 us, and 160^2 planes
// (200 KB: one CTA per SM) by clusters of four 385 -> 350 us for 21 fields.
// C = 1: passes that join two axes save 2 of 6 crossings and barriers.  What
// bounds several CTAs per SM is the shared-memory data pipe, so it gains at
// 64^2 (64 runs of 64^3 x 8: 509 -> 446 us, 5.6 TB/s), 96^2 (96^3 x 55: 207 ->
// 198 us) and 80^2 (80^3 x 50: 97 -> 90 us).
// What bounds it: the load/store pipe (53 to 60 %) and barriers; DRAM at 42 to 82 % of its rate.
// One item of P1 at a time: 32 values in flight (unroll 2 to 4) cost 1 to 2 %.
// ---------------------------------------------------------------------------
template <int NY, int NZ, int C, bool RAWP, int ZA, int ZB, int ZP>
struct YZ {
  static constexpr int Q = ZA * ZB * ZP, N1 = NZ / Q, R = NZ / C, ZL = N1 / C;  // z points a CTA holds: R, ZL of each run
  static constexpr int PY = RAWP ? Line<NY>::RAW : Line<NY>::PITCH;
  static constexpr size_t SMEM = (size_t)R * PY * sizeof(float2);
  static_assert(Q * N1 == NZ && ZL * C == N1 && Q % C == 0, "whole factors");
};

// P3 (forward or inverse): ZP points (stride S rows) of the H S columns of every y position
template <int NY, int H, int ZP, int S, int PY, int C, int T, bool INV>
__device__ __forceinline__ void colP(float2* U, const float2* twZ, int r) {
#pragma unroll 2
  for (int it = threadIdx.x; it < NY * S * H; it += T) {
    const int g = it / NY, yp = it - g * NY, h = g / S, j = g - h * S;
    const int t = (r + C * j) * H;
    passA_item<S, ZP, S * PY, INV>(U + (j + S * ZP * h) * PY + Line<NY>::phys(yp), [&](int k) { return twZ[t * k]; });
  }
}

template <int NY, int NZ, int C, int T, int MODE, bool RAWP, int ZA, int ZB, int ZP, int MINB, int UCT>
__global__ void __launch_bounds__(T, MINB) yz_kernel(const RunParams* __restrict__ runs, const Shape sh) {
  using LY = Line<NY>;
  using G = YZ<NY, NZ, C, RAWP, ZA, ZB, ZP>;
  constexpr int N1y = LY::N1, N2y = LY::N2, N1z = G::N1, Q = G::Q, ZL = G::ZL, PY = G::PY;
  constexpr int S3 = ZL, S2 = S3 * ZP, S1 = S2 * ZB;  // row strides of the stages ZP, ZB, ZA
  constexpr int UC = UCT ? UCT : N1z;
  static_assert(T % 32 == 0, "whole warps");
  extern __shared__ float2 U[];
  constexpr int QC = Q / C;           // runs a CTA updates
  __shared__ float4 qzt[QC * N1z];    // their kz factors, in the runs' order
  __shared__ float2 twZ[NZ];
  const int r = C == 1 ? 0 : (int)(blockIdx.x % C);
  const auto freq = [](int rr) { return rr / (ZP * ZB) + ZA * (rr / ZP % ZB) + ZA * ZB * (rr % ZP); };
  for (int j = threadIdx.x; j < QC * N1z; j += T) {
    const int k = freq(r * QC + j / N1z) + Q * (j % N1z);
    const float n = __ldg(sh.qnz + k);
    qzt[j] = make_float4(__ldg(sh.qz2 + k), __ldg(sh.qz4 + k), n, n * n);
  }
  for (int j = threadIdx.x; j < NZ; j += T) twZ[j] = __ldg(sh.twZ + j);
  const RunParams& rp = runs[blockIdx.y];
  const int p = sh.plane0 + (int)(blockIdx.x / C);
  const int Kx = sh.Kx;
  const int f = (MODE == YZ_C2) ? rp.V : p / Kx;
  const int kx = p - (p / Kx) * Kx;
  const size_t plane_elems = (size_t)NZ * NY;
  const size_t poff = ((size_t)f * Kx + kx) * plane_elems;        // k-space state
  const size_t moff = (size_t)f * Kx * plane_elems + kx * sh.ks;  // mixed space
  const bool is_c = (f == rp.V);
  const bool var_c = (MODE == YZ_MAIN) && is_c && rp.mobility != MOB_CONST;

  // y twiddles of a column n1y: preloaded when every item of a thread has the same one
  constexpr bool FIXED = T % N1y == 0;
  const auto load_wy = [&](float2* wy, int n1y) {
#pragma unroll
    for (int k2 = 1; k2 < N2y; ++k2) wy[k2] = __ldg(sh.twY + n1y * k2);
  };
  constexpr int I1 = N1y * S1, I2 = N2y * S2 * ZA;  // items of P1 and P2
  __syncthreads();  // the tables

  // P1 forward
  {
    const float2* src = (MODE == YZ_MAIN) ? rp.D + moff : (MODE == YZ_C2 ? rp.J + kx * sh.ks : rp.Sm + moff);
    float2 wy[N2y];
    if constexpr (FIXED) load_wy(wy, threadIdx.x % N1y);
#pragma unroll 1
    for (int it = threadIdx.x; it < I1; it += T) {
      const int m = it / N1y, n1y = it - m * N1y;
      float2 v[ZA][N2y];
#pragma unroll
      for (int b = 0; b < ZA; ++b) {
        const float2* s = src + (r + C * (m + S1 * b)) * sh.zs + n1y;
#pragma unroll
        for (int n2 = 0; n2 < N2y; ++n2) v[b][n2] = __ldg(s + n2 * N1y);
      }
      if constexpr (!FIXED) load_wy(wy, n1y);
      float2* d = U + m * PY + n1y;
#pragma unroll
      for (int b = 0; b < ZA; ++b) {
        Dft<N2y>::fwd(v[b]);
#pragma unroll
        for (int k2 = 1; k2 < N2y; ++k2) v[b][k2] = cmul(v[b][k2], wy[k2]);
      }
      float2 wz[ZA];
#pragma unroll
      for (int kb = 1; kb < ZA; ++kb) wz[kb] = twZ[(r + C * m) * kb];
#pragma unroll
      for (int k2 = 0; k2 < N2y; ++k2) {
        float2 c[ZA];
#pragma unroll
        for (int b = 0; b < ZA; ++b) c[b] = v[b][k2];
        Dft<ZA>::fwd(c);
#pragma unroll
        for (int kb = 0; kb < ZA; ++kb)
          d[S1 * kb * PY + k2 * (N1y + 1)] = kb == 0 ? c[0] : cmul(c[kb], wz[kb]);
      }
    }
  }
  __syncthreads();
  // P2 forward
#pragma unroll 1
  for (int it = threadIdx.x; it < I2; it += T) {
    const int g = it / N2y, k2y = it - g * N2y, kb = g / S2, m = g - kb * S2;
    float2* q = U + (m + S1 * kb) * PY + k2y * (N1y + 1);
    float2 v[ZB][N1y];
#pragma unroll
    for (int a = 0; a < ZB; ++a) {
#pragma unroll
      for (int j = 0; j < N1y; ++j) v[a][j] = q[S2 * a * PY + j];
    }
#pragma unroll
    for (int a = 0; a < ZB; ++a) Dft<N1y>::fwd(v[a]);
    float2 wz[ZB];
#pragma unroll
    for (int ka = 1; ka < ZB; ++ka) wz[ka] = twZ[(r + C * m) * ZA * ka];
#pragma unroll
    for (int j = 0; j < N1y; ++j) {
      float2 c[ZB];
#pragma unroll
      for (int a = 0; a < ZB; ++a) c[a] = v[a][j];
      Dft<ZB>::fwd(c);
#pragma unroll
      for (int ka = 0; ka < ZB; ++ka) q[S2 * ka * PY + j] = ka == 0 ? c[0] : cmul(c[ka], wz[ka]);
    }
  }
  if (C == 1 || ZP > 1) __syncthreads();
  // P3 forward: z points ZP of a column
  if constexpr (ZP > 1) {
    colP<NY, ZA * ZB, ZP, S3, PY, C, T, false>(U, twZ, r);
    if (C == 1) __syncthreads();
  }
  if (C > 1) cluster_barrier();
  // P4: last forward z stage, pointwise k-space update, first inverse z stage
  const KPlane P(rp, sh, kx, MODE, is_c, yz_norm<MODE>(NY * NZ, sh.Nx));
  const float wkx = (kx == 0 || 2 * kx == sh.Nx) ? 1.0f : 2.0f;
  float fint = 0.f;
#pragma unroll 1
  for (int it = threadIdx.x; it < NY * QC; it += T) {
    const int yp = it % NY, rl = it / NY, rr = r * QC + rl;
    const KRow R(P, sh, LY::freq_of_pos(yp));
    float2* pc = U + rr * ZL * PY + LY::phys(yp);
    // k-space state of this plane in [k1][k2][y position] order: for every
    // k1 a warp reads and writes 32 consecutive y positions (coalesced)
    float2* gk = rp.Sk + poff + freq(rr) * NY + yp;
    constexpr size_t SK1 = (size_t)Q * NY;  // stride of k1
    const uint32_t a = smem_addr(pc);
    float2 d[N1z];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const uint32_t ac = C > 1 ? map_rank(a, c) : 0;
#pragma unroll
      for (int j = 0; j < ZL; ++j) d[c + C * j] = C > 1 ? ld_peer(ac + (uint32_t)(j * PY * 8)) : pc[j * PY];
    }
    update_run<N1z, 1, MODE, UC>(d, gk, SK1, P, R, qzt + rl * N1z, is_c, var_c, fint);
    if (MODE != YZ_IMPORT) {
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const uint32_t ac = C > 1 ? map_rank(a, c) : 0;
#pragma unroll
        for (int j = 0; j < ZL; ++j) {
          if (C > 1) st_peer(ac + (uint32_t)(j * PY * 8), d[c + C * j]);
          else pc[j * PY] = d[j];
        }
      }
    }
  }
  if (C > 1) cluster_barrier();  // also: nothing reads a CTA that has left
  if (MODE == YZ_IMPORT) return;
  if (C == 1) __syncthreads();
  // P3 inverse: z points ZP of a column
  if constexpr (ZP > 1) {
    colP<NY, ZA * ZB, ZP, S3, PY, C, T, true>(U, twZ, r);
    __syncthreads();
  }
  // P2 inverse
#pragma unroll 1
  for (int it = threadIdx.x; it < I2; it += T) {
    const int g = it / N2y, k2y = it - g * N2y, kb = g / S2, m = g - kb * S2;
    float2* q = U + (m + S1 * kb) * PY + k2y * (N1y + 1);
    float2 wz[ZB];
#pragma unroll
    for (int ka = 1; ka < ZB; ++ka) wz[ka] = twZ[(r + C * m) * ZA * ka];
    float2 v[ZB][N1y];
#pragma unroll
    for (int j = 0; j < N1y; ++j) {
      float2 c[ZB];
#pragma unroll
      for (int ka = 0; ka < ZB; ++ka) {
        const float2 x = q[S2 * ka * PY + j];
        c[ka] = ka == 0 ? x : cmulc(x, wz[ka]);
      }
      dft_inv<ZB>(c);
#pragma unroll
      for (int a = 0; a < ZB; ++a) v[a][j] = c[a];
    }
#pragma unroll
    for (int a = 0; a < ZB; ++a) {
      dft_inv<N1y>(v[a]);
#pragma unroll
      for (int j = 0; j < N1y; ++j) q[S2 * a * PY + j] = v[a][j];
    }
  }
  __syncthreads();
  // P1 inverse, straight to the mixed-space output
  {
    const bool real_plane = (kx == 0) || (2 * kx == sh.Nx);  // the x-DFT of real data is real there
    const bool real_out = real_plane && !var_c;
    float2* dst = var_c ? rp.J + kx * sh.ks : rp.Sm + moff;
    float2 wy[N2y];
    if constexpr (FIXED) load_wy(wy, threadIdx.x % N1y);
#pragma unroll 1
    for (int it = threadIdx.x; it < I1; it += T) {
      const int m = it / N1y, n1y = it - m * N1y;
      const float2* q = U + m * PY + n1y;
      float2 wz[ZA];
#pragma unroll
      for (int kb = 1; kb < ZA; ++kb) wz[kb] = twZ[(r + C * m) * kb];
      float2 v[ZA][N2y];
#pragma unroll
      for (int k2 = 0; k2 < N2y; ++k2) {
        float2 c[ZA];
#pragma unroll
        for (int kb = 0; kb < ZA; ++kb) {
          const float2 x = q[S1 * kb * PY + k2 * (N1y + 1)];
          c[kb] = kb == 0 ? x : cmulc(x, wz[kb]);
        }
        dft_inv<ZA>(c);
#pragma unroll
        for (int b = 0; b < ZA; ++b) v[b][k2] = c[b];
      }
      if constexpr (!FIXED) load_wy(wy, n1y);
#pragma unroll
      for (int b = 0; b < ZA; ++b) {
#pragma unroll
        for (int k2 = 1; k2 < N2y; ++k2) v[b][k2] = cmulc(v[b][k2], wy[k2]);
        dft_inv<N2y>(v[b]);
        float2* o = dst + (r + C * (m + S1 * b)) * sh.zs + n1y;
#pragma unroll
        for (int n2 = 0; n2 < N2y; ++n2) {
          float2 x = v[b][n2];
          if (real_out) x.y = 0.f;
          o[n2 * N1y] = x;
        }
      }
    }
  }

  if (MODE == YZ_MAIN) {
    yz_finish<T>(rp, sh, fint, wkx, (size_t)sh.plane0 * C + blockIdx.x);
  }
}

}  // namespace pf
