// FP64 GPU path: cuFFT D2Z/Z2D and plain kernels for the phases of the
// reference loop body, 2 var + 3 transforms per step (2 more with variable
// mobility).  It is the comparator for the fused FP32 path, an FP64 GPU
// cross-check of the CPU oracle, and what runs grids outside the fused list.
#pragma once
#include <cuda_runtime.h>

#include "../../include/pfgpu.h"

namespace pf {
// A run's real-space fields on its device: field f of cell i is
// phi[f * fstride + i * cstride] (float or double), c contiguous; valid on
// `stream` until the run is stepped or destroyed or its fields are set or got.
struct DeviceFields {
  const void* phi;
  const void* con;
  int is_double;
  size_t fstride, cstride;
  int nx, ny, nz, var, device;
  void* stream;
};
// for either precision path (the fused path first transforms its spectral
// state into its staging buffer)
int run_device_fields(pf_run* run, DeviceFields* out);

// Waits for a stream when the scope ends, unless disarmed by then: a call that
// fails halfway must not leave a kernel or a copy at work on the caller's arrays.
struct Drain {
  cudaStream_t stream;
  bool armed = true;
  ~Drain() {
    if (armed) cudaStreamSynchronize(stream);
  }
};

struct Plain64;
int plain64_device_fields(Plain64* p, DeviceFields* out);
int plain64_validate(const pf_config* c);
int plain64_create(const pf_config* c, Plain64** out);
int plain64_set_fields(Plain64* p, const double* phi_aos, const double* con);
int plain64_step(Plain64* p, int nsteps, pf_diag* diag);
int plain64_get_fields(Plain64* p, double* phi_aos, double* con);
void plain64_destroy(Plain64* p);
}  // namespace pf
