// Voxel analysis of the post-processor paraview.x (src/paraview.f90) on the GPU.
//
// Per voxel (src/paraview.f90:189-244), in FP64 with the reference's order
// of operations (no contraction into FMA, so results are bit-identical to a
// plain loop):
//   phi_sq   = sum_{i=1..var} phi_i^2
//   var_num  = the last i with phi_i > 0.8 (0 if none)
//   phi_3    = phi_3 (the index 3 is fixed in the reference, whatever var is)
//   boundary = 1 if more than one phi_i > threshold, else 0
// and two counts: boundary voxels, and boundary voxels with phi_var > threshold.
// |grad phi_3| (src/paraview.f90:380-429): central differences / 2 on the
// interior cells 2..N-1 of every axis, 0 on the outer layer.
//
// One pass over the fields (the classification reads var values and writes up
// to four per voxel; the gradient reads the phi_3 that it wrote, with its six
// neighbours through L1 and L2), grid-stride loops, counts reduced per block
// and added once per block (integers: the result does not depend on the
// order).  Fields in host memory, phi(var, x, y, z), are what the
// post-processor has: the kernel reads them where they are, over NVLink-C2C, a
// warp 32 whole cells at a time through shared memory.  That reading is the
// bound (96^3 x 55: 389 MB, 2.0 ms at the link's 200 GB/s); copying them to
// the device first cost an allocation of their size and a second pass.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <string>

#include "../../include/pfgpu.h"
#include "pf_internal.h"
#include "pf_plain64.h"

namespace pf {
namespace {

constexpr int kThreads = 256;

// Source fields: value of field f at cell i is base[f * fstride + i * cstride].
template <typename T>
struct Src {
  const T* phi;
  const T* con;
  size_t fstride, cstride;
  __device__ __forceinline__ double at(int f, size_t i) const { return (double)phi[f * fstride + i * cstride]; }
};

// Device outputs of one analysis; any may be null.
struct Outs {
  double *phi_sq, *phi_3, *grad, *boundary, *con;
  int* var_num;
};

// One cell, at(f) = phi_f: writes its outputs, returns (boundary, boundary with phi_var above).
template <class At>
__device__ __forceinline__ uint2 classify_cell(const At& at, int V, size_t i, double thr, const Outs& o) {
  double sq = 0.0;
  int vmax = 0, above = 0;
  for (int f = 0; f < V; ++f) {
    const double p = at(f);
    sq = __dadd_rn(sq, __dmul_rn(p, p));
    if (p > 0.8) vmax = f + 1;
    above += p > thr;
  }
  const bool b = above > 1;
  if (o.phi_sq) o.phi_sq[i] = sq;
  if (o.var_num) o.var_num[i] = vmax;
  if (o.phi_3) o.phi_3[i] = at(2);
  if (o.boundary) o.boundary[i] = b ? 1.0 : 0.0;
  return make_uint2(b, b && at(V - 1) > thr);
}

__device__ __forceinline__ void add_counts(uint2 n, unsigned long long* counts) {
  n.x = __reduce_add_sync(0xffffffffu, n.x);
  n.y = __reduce_add_sync(0xffffffffu, n.y);
  __shared__ unsigned sb[kThreads / 32], sp[kThreads / 32];
  if ((threadIdx.x & 31) == 0) {
    sb[threadIdx.x >> 5] = n.x;
    sp[threadIdx.x >> 5] = n.y;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long tb = 0, tp = 0;
    for (unsigned w = 0; w < blockDim.x / 32; ++w) {
      tb += sb[w];
      tp += sp[w];
    }
    if (tb) atomicAdd(&counts[0], tb);
    if (tp) atomicAdd(&counts[1], tp);
  }
}

template <typename T>
__global__ void __launch_bounds__(kThreads) classify_kernel(Src<T> s, int V, size_t n, double thr, Outs o,
                                                            unsigned long long* counts) {
  uint2 c = make_uint2(0, 0);
  for (size_t i = blockIdx.x * (size_t)kThreads + threadIdx.x; i < n; i += (size_t)gridDim.x * kThreads) {
    const uint2 d = classify_cell([&](int f) { return s.at(f, i); }, V, i, thr, o);
    c.x += d.x;
    c.y += d.y;
    if (o.con) o.con[i] = (double)s.con[i];  // c is contiguous in both layouts
  }
  add_counts(c, counts);
}

// Fields of a cell next to each other (cstride = V): a warp copies 32 cells,
// one contiguous piece, into its part of shared memory (odd pitch).
__global__ void __launch_bounds__(kThreads) classify_cells_kernel(Src<double> s, int V, size_t n, double thr, Outs o,
                                                                  unsigned long long* counts) {
  extern __shared__ double cells[];
  const int pitch = V | 1, lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double* mine = cells + (size_t)w * 32 * pitch;
  uint2 c = make_uint2(0, 0);
  for (size_t i0 = ((size_t)blockIdx.x * nw + w) * 32; i0 < n; i0 += (size_t)gridDim.x * nw * 32) {
    const int m = (int)(n - i0 < 32 ? n - i0 : 32);
    const double* src = s.phi + i0 * V;
    __syncwarp();
    int cell = lane / V, f = lane - cell * V;  // of value it = lane, lane + 32, ...
    const int dc = 32 / V, df = 32 - dc * V;
#pragma unroll 4
    for (int it = lane; it < m * V; it += 32) {
      mine[cell * pitch + f] = src[it];
      cell += dc;
      f += df;
      if (f >= V) {
        f -= V;
        ++cell;
      }
    }
    __syncwarp();
    if (lane < m) {
      const size_t i = i0 + lane;
      const double* p = mine + lane * pitch;
      const uint2 d = classify_cell([&](int k) { return p[k]; }, V, i, thr, o);
      c.x += d.x;
      c.y += d.y;
      if (o.con) o.con[i] = s.con[i];
    }
  }
  add_counts(c, counts);
}

__global__ void __launch_bounds__(kThreads) grad3_kernel(const double* __restrict__ p, int Nx, int Ny, int Nz,
                                                         double* __restrict__ grad) {
  const size_t n = (size_t)Nx * Ny * Nz;
  const size_t sx = 1, sy = (size_t)Nx, sz = (size_t)Nx * Ny;
  for (size_t i = blockIdx.x * (size_t)kThreads + threadIdx.x; i < n; i += (size_t)gridDim.x * kThreads) {
    const int x = (int)(i % Nx), y = (int)((i / Nx) % Ny), z = (int)(i / sz);
    double g = 0.0;
    if (x > 0 && x < Nx - 1 && y > 0 && y < Ny - 1 && z > 0 && z < Nz - 1) {
      const double gx = __ddiv_rn(__dsub_rn(p[i + sx], p[i - sx]), 2.0);
      const double gy = __ddiv_rn(__dsub_rn(p[i + sy], p[i - sy]), 2.0);
      const double gz = __ddiv_rn(__dsub_rn(p[i + sz], p[i - sz]), 2.0);
      g = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(gx, gx), __dmul_rn(gy, gy)), __dmul_rn(gz, gz)));
    }
    grad[i] = g;
  }
}

// Blocks for n items, `per_block` at a time, at most `per_sm` of them an SM.
unsigned grid_for(size_t n, size_t per_block = kThreads, int per_sm = 8) {
  int dev = 0, sms = 152;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return (unsigned)std::min<size_t>((n + per_block - 1) / per_block, (size_t)sms * per_sm);
}

#define AN_CUDA(call)                                                                  \
  do {                                                                                 \
    cudaError_t e_ = (call);                                                           \
    if (e_ != cudaSuccess) {                                                           \
      set_cuda_error(std::string("analysis: ") + #call + ": " + cudaGetErrorString(e_)); \
      rc = PF_ECUDA;                                                                   \
      goto done;                                                                       \
    }                                                                                  \
  } while (0)

template <typename T>
cudaError_t launch_classify(const Src<T>& s, int V, size_t n, double thr, cudaStream_t st, const Outs& o,
                            unsigned long long* counts) {
  if constexpr (sizeof(T) == sizeof(double)) {
    if (s.cstride == (size_t)V && V > 1) {
      // as many warps as share 48 KB, at least one (V = 255: 65 KB); beyond V = 799, 200 KB, the general way
      const size_t per_warp = (size_t)32 * (V | 1) * sizeof(double);
      const int warps = (int)std::max<size_t>(1, std::min<size_t>(kThreads / 32, (48u << 10) / per_warp));
      const size_t smem = warps * per_warp;
      if (smem <= (200u << 10) && (smem <= (48u << 10) || raise_smem((const void*)classify_cells_kernel, smem))) {
        classify_cells_kernel<<<grid_for(n, 32 * warps, 4), warps * 32, smem, st>>>(s, V, n, thr, o, counts);
        return cudaGetLastError();
      }
    }
  }
  classify_kernel<T><<<grid_for(n), kThreads, 0, st>>>(s, V, n, thr, o, counts);
  return cudaGetLastError();
}

template <typename T>
int analyze(const Src<T>& src, int Nx, int Ny, int Nz, int V, double thr, cudaStream_t st, const pf_analysis_out* ho,
            pf_voxel_counts* counts) {
  const size_t n = (size_t)Nx * Ny * Nz;
  int rc = PF_OK;
  Outs d{};
  unsigned long long hc[2] = {0, 0};
  // one allocation: the counts, then the arrays asked for (the gradient needs phi_3 on the device)
  const bool grad = ho && ho->grad_phi_3;
  char* mem = nullptr;
  size_t bytes = 256;
  const auto take = [&](bool want, size_t b) {
    const size_t at = bytes;
    if (want) bytes += (b + 255) & ~(size_t)255;
    return want ? at : 0;
  };
  const size_t at_sq = take(ho && ho->phi_sq, n * sizeof(double)), at_num = take(ho && ho->var_num, n * sizeof(int));
  const size_t at_3 = take((ho && ho->phi_3) || grad, n * sizeof(double)), at_grad = take(grad, n * sizeof(double));
  const size_t at_bnd = take(ho && ho->boundary, n * sizeof(double)), at_con = take(ho && ho->con, n * sizeof(double));
  AN_CUDA(cudaMalloc(&mem, bytes));
  {
    const auto at = [&](size_t off) { return off ? (void*)(mem + off) : nullptr; };
    d.phi_sq = (double*)at(at_sq);
    d.var_num = (int*)at(at_num);
    d.phi_3 = (double*)at(at_3);
    d.grad = (double*)at(at_grad);
    d.boundary = (double*)at(at_bnd);
    d.con = (double*)at(at_con);
  }
  AN_CUDA(cudaMemsetAsync(mem, 0, sizeof hc, st));
  AN_CUDA(launch_classify(src, V, n, thr, st, d, (unsigned long long*)mem));
  if (grad) {
    grad3_kernel<<<grid_for(n), kThreads, 0, st>>>(d.phi_3, Nx, Ny, Nz, d.grad);
    AN_CUDA(cudaGetLastError());
  }
  AN_CUDA(cudaMemcpyAsync(hc, mem, sizeof hc, cudaMemcpyDeviceToHost, st));
  if (ho && ho->phi_sq) AN_CUDA(cudaMemcpyAsync(ho->phi_sq, d.phi_sq, n * sizeof(double), cudaMemcpyDeviceToHost, st));
  if (ho && ho->var_num) AN_CUDA(cudaMemcpyAsync(ho->var_num, d.var_num, n * sizeof(int), cudaMemcpyDeviceToHost, st));
  if (ho && ho->phi_3) AN_CUDA(cudaMemcpyAsync(ho->phi_3, d.phi_3, n * sizeof(double), cudaMemcpyDeviceToHost, st));
  if (grad) AN_CUDA(cudaMemcpyAsync(ho->grad_phi_3, d.grad, n * sizeof(double), cudaMemcpyDeviceToHost, st));
  if (ho && ho->boundary)
    AN_CUDA(cudaMemcpyAsync(ho->boundary, d.boundary, n * sizeof(double), cudaMemcpyDeviceToHost, st));
  if (ho && ho->con) AN_CUDA(cudaMemcpyAsync(ho->con, d.con, n * sizeof(double), cudaMemcpyDeviceToHost, st));
  AN_CUDA(cudaStreamSynchronize(st));
  counts->boundary_voxels = (long long)hc[0];
  counts->precipitate_voxels = (long long)hc[1];
  counts->precipitate_fraction = hc[0] ? (double)hc[1] / (double)hc[0] : 0.0;
done:
  if (rc) cudaStreamSynchronize(st);  // copies into the caller's arrays may be in flight
  cudaFree(mem);
  return rc;
}

int check_args(const pf_config* c, pf_voxel_counts* counts) {
  if (!c || !counts) {
    set_error("analysis: null argument");
    return PF_EINVAL;
  }
  if (c->nx < 1 || c->ny < 1 || c->nz < 1 || c->var < 3) {
    set_error("analysis: needs a grid and var >= 3 (phi_3 is analysed)");
    return PF_EINVAL;
  }
  return PF_OK;
}

}  // namespace
}  // namespace pf

extern "C" int pf_analyze_fields(const pf_config* cfg, const double* phi_aos, const double* con, double threshold,
                                 const pf_analysis_out* out, pf_voxel_counts* counts) {
  using namespace pf;
  int rc = check_args(cfg, counts);
  if (rc) return rc;
  if (!phi_aos || !con) {
    set_error("analysis: null field");
    return PF_EINVAL;
  }
  const size_t n = (size_t)cfg->nx * cfg->ny * cfg->nz;
  const int V = cfg->var;
  double* dev = nullptr;  // copies, where the GPU does not reach the caller's memory
  cudaStream_t st = nullptr;
  Src<double> s{phi_aos, con, 1, (size_t)V};
  {
    int coherent = 0;
    cudaError_t e = cudaSetDevice(cfg->device);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e == cudaSuccess)
      e = cudaDeviceGetAttribute(&coherent, cudaDevAttrPageableMemoryAccessUsesHostPageTables, cfg->device);
    const auto host = [&](const void* p) {
      cudaPointerAttributes a;
      if ((uintptr_t)p % sizeof(double) != 0 || cudaPointerGetAttributes(&a, p) != cudaSuccess) return false;
      return a.type == cudaMemoryTypeHost || a.type == cudaMemoryTypeUnregistered;
    };
    if (e == cudaSuccess && !(coherent && host(phi_aos) && host(con))) {
      cudaGetLastError();
      e = cudaMalloc(&dev, n * (V + 1) * sizeof(double));
      if (e == cudaSuccess) e = cudaMemcpyAsync(dev, phi_aos, n * V * sizeof(double), cudaMemcpyHostToDevice, st);
      if (e == cudaSuccess) e = cudaMemcpyAsync(dev + n * V, con, n * sizeof(double), cudaMemcpyHostToDevice, st);
      s.phi = dev;
      s.con = dev + n * V;
    }
    if (e != cudaSuccess) {
      set_cuda_error(std::string("analysis: ") + cudaGetErrorString(e));
      rc = e == cudaErrorMemoryAllocation ? PF_ENOMEM : PF_ECUDA;
    }
  }
  if (!rc) rc = analyze(s, cfg->nx, cfg->ny, cfg->nz, V, threshold, st, out, counts);
  cudaFree(dev);
  if (st) cudaStreamDestroy(st);
  return rc;
}

// In-situ analysis of a run's resident fields (no host copy of the fields).
extern "C" int pf_analyze_run(pf_run* run, double threshold, const pf_analysis_out* out, pf_voxel_counts* counts) {
  using namespace pf;
  DeviceFields f{};
  int rc = run_device_fields(run, &f);
  if (rc) return rc;
  pf_config c{};
  c.nx = f.nx; c.ny = f.ny; c.nz = f.nz; c.var = f.var; c.device = f.device;
  rc = check_args(&c, counts);
  if (rc) return rc;
  if (f.is_double) {
    Src<double> s{(const double*)f.phi, (const double*)f.con, f.fstride, f.cstride};
    return analyze(s, f.nx, f.ny, f.nz, f.var, threshold, (cudaStream_t)f.stream, out, counts);
  }
  Src<float> s{(const float*)f.phi, (const float*)f.con, f.fstride, f.cstride};
  return analyze(s, f.nx, f.ny, f.nz, f.var, threshold, (cudaStream_t)f.stream, out, counts);
}
