// A CUDA runtime and cuFFT of the host, for tests of the library's host code
// without a GPU: memory is host memory, kernels do nothing, and every call is
// counted and can be made to fail.  Linked with the library's own objects in
// place of the CUDA libraries.
#include <cuda_runtime_api.h>
#include <cufft.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

namespace {
std::mutex mu;
std::map<std::string, int> counts;
std::map<void*, int> device_mem, host_mem;  // device the block belongs to
std::map<const void*, int> smem;            // kernels' shared-memory attribute
std::map<cufftHandle, int> plan_device;
std::string fail_name, order;  // the call that fails, the calls so far
int last = 0, fail_in = 0, fail_code = 0, coherent = 1, lowered = 0, strays = 0, next_plan = 1;
thread_local int dev = 0;

int hit(const char* name) {
  std::lock_guard<std::mutex> lk(mu);
  ++counts[name];
  order += name;
  order += ' ';
  if (fail_name != name || fail_in == 0 || --fail_in > 0) return 0;
  order += "FAILED ";
  return last = fail_code;
}
// a call of device `dev` given memory of another one
void check(const void* p) {
  std::lock_guard<std::mutex> lk(mu);
  auto it = device_mem.upper_bound(const_cast<void*>(p));
  if (it == device_mem.begin()) return;
  --it;
  if (it->first == p && it->second != dev) ++strays;
}
cudaError_t get(const char* name, void** p, size_t n, std::map<void*, int>& m) {
  *p = nullptr;
  if (const int e = hit(name)) return (cudaError_t)e;
  *p = std::calloc(1, n ? n : 1);
  std::lock_guard<std::mutex> lk(mu);
  m[*p] = dev;
  return cudaSuccess;
}
cudaError_t drop(const char* name, void* p, std::map<void*, int>& m) {
  hit(name);
  std::lock_guard<std::mutex> lk(mu);
  m.erase(p);
  std::free(p);
  return cudaSuccess;
}
}  // namespace

#define CALL(name) \
  if (const int e_ = hit(name)) return (cudaError_t)e_; \
  return cudaSuccess

extern "C" {
// the tests' side
void fake_reset() {
  std::lock_guard<std::mutex> lk(mu);
  counts.clear();
  order.clear();
  fail_name.clear();
  last = fail_in = lowered = strays = 0;
  coherent = 1;
}
void fake_fail(const char* name, int nth, int code) { fail_name = name, fail_in = nth, fail_code = code; }
void fake_coherent(int on) { coherent = on; }
int fake_count(const char* name) { return counts[name]; }
const char* fake_order() { return order.c_str(); }
int fake_lowered() { return lowered; }  // kernels whose shared-memory attribute was lowered
int fake_strays() { return strays; }    // plans and memory used on another device than their own
int fake_live() { return (int)(device_mem.size() + host_mem.size() + plan_device.size()); }

cudaError_t cudaMalloc(void** p, size_t n) { return get("cudaMalloc", p, n, device_mem); }
cudaError_t cudaFree(void* p) { return drop("cudaFree", p, device_mem); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return get("cudaHostAlloc", p, n, host_mem); }
cudaError_t cudaMallocHost(void** p, size_t n) { return get("cudaHostAlloc", p, n, host_mem); }
cudaError_t cudaFreeHost(void* p) { return drop("cudaFreeHost", p, host_mem); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  if (const int e = hit("cudaMemcpy")) return (cudaError_t)e;
  check(d), check(s);
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  if (const int e = hit("cudaMemcpyAsync")) return (cudaError_t)e;
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy2D(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind) {
  if (const int e = hit("cudaMemcpy2D")) return (cudaError_t)e;
  for (size_t i = 0; i < h; ++i) std::memcpy((char*)d + i * dp, (const char*)s + i * sp, w);
  return cudaSuccess;
}
cudaError_t cudaMemset(void*, int, size_t) { CALL("cudaMemset"); }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { CALL("cudaMemsetAsync"); }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
  *f = *t = (size_t)1 << 38;
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  std::memset(a, 0, sizeof *a);
  std::lock_guard<std::mutex> lk(mu);
  void* q = const_cast<void*>(p);
  a->type = device_mem.count(q) ? cudaMemoryTypeDevice : (host_mem.count(q) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered);
  return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* n) {
  *n = 2;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = dev;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
  dev = d;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 152 : (a == cudaDevAttrPageableMemoryAccessUsesHostPageTables ? coherent : 0);
  return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* lo, int* hi) {
  *lo = 0, *hi = -5;
  return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "made to fail"; }
cudaError_t cudaGetLastError() {
  const int e = last;
  last = 0;
  return (cudaError_t)e;
}
cudaError_t cudaDeviceSynchronize() { CALL("cudaDeviceSynchronize"); }

cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  if (const int e = hit("cudaFuncSetAttribute")) return (cudaError_t)e;
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
    std::lock_guard<std::mutex> lk(mu);
    int& cur = smem[f];
    lowered += v < cur;
    cur = v;
  }
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) { CALL("cudaLaunchKernelExC"); }
cudaError_t cudaGetSymbolAddress(void** p, const void* s) {
  *p = const_cast<void*>(s);
  return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = nullptr;
  CALL("cudaStreamCreate");
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned, int) {
  *s = nullptr;
  CALL("cudaStreamCreate");
}
cudaError_t cudaStreamDestroy(cudaStream_t) { CALL("cudaStreamDestroy"); }
cudaError_t cudaStreamSynchronize(cudaStream_t) { CALL("cudaStreamSynchronize"); }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
  *s = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = nullptr;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
  *x = nullptr;
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { CALL("cudaGraphLaunch"); }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = nullptr;
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.f;
  return cudaSuccess;
}

// what nvcc's launch stubs call
void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
  *k = (cudaKernel_t)f;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) { CALL("launch"); }

static cufftResult new_plan(cufftHandle* h) {
  if (hit("cufftPlan")) return CUFFT_ALLOC_FAILED;
  std::lock_guard<std::mutex> lk(mu);
  *h = next_plan++;
  plan_device[*h] = dev;
  return CUFFT_SUCCESS;
}
static cufftResult exec(cufftHandle h) {
  if (hit("cufftExec")) return CUFFT_EXEC_FAILED;
  std::lock_guard<std::mutex> lk(mu);
  strays += plan_device[h] != dev;
  return CUFFT_SUCCESS;
}
cufftResult cufftCreate(cufftHandle* h) { return new_plan(h); }
cufftResult cufftPlan3d(cufftHandle* h, int, int, int, cufftType) { return new_plan(h); }
cufftResult cufftMakePlanMany(cufftHandle, int, int*, int*, int, int, int*, int, int, cufftType, int, size_t* ws) {
  *ws = 256;
  return CUFFT_SUCCESS;
}
cufftResult cufftSetAutoAllocation(cufftHandle, int) { return CUFFT_SUCCESS; }
cufftResult cufftSetWorkArea(cufftHandle, void*) { return CUFFT_SUCCESS; }
cufftResult cufftSetStream(cufftHandle, cudaStream_t) { return CUFFT_SUCCESS; }
cufftResult cufftDestroy(cufftHandle h) {
  std::lock_guard<std::mutex> lk(mu);
  plan_device.erase(h);
  return CUFFT_SUCCESS;
}
cufftResult cufftExecD2Z(cufftHandle h, cufftDoubleReal*, cufftDoubleComplex*) { return exec(h); }
cufftResult cufftExecZ2D(cufftHandle h, cufftDoubleComplex*, cufftDoubleReal*) { return exec(h); }
}
