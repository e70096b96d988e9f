// A CUDA runtime of two devices without GPUs, loaded before libgisapr_gb300.so: memory comes from malloc, kernels do
// not run. The dynamic shared memory a kernel may take is kept per device, as the runtime keeps it; a launch that asks
// for more fails, and a limit that is lowered is counted.
#include <cuda_runtime_api.h>
#include <cufft.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <utility>

namespace {
thread_local int current = 0;
std::mutex guard;
std::map<std::pair<int, const void*>, size_t> limits;
int launched = 0, refused = 0, lowered = 0;
int recorded = 0, waited = 0;  // events
unsigned long long stream_id = 1;
size_t held = 0, plan_held = 0, plan_bytes = 1024;  // device memory of the callers and of plans; what a plan takes
std::map<void*, size_t> sizes;
std::map<int, size_t> plans;  // handle -> work area of its own
std::map<int, bool> automatic;
int last_plan = 0;

cufftResult plan_made(int h) {
  if (automatic.count(h) && !automatic[h]) return CUFFT_SUCCESS;
  plans[h] = plan_bytes;
  plan_held += plan_bytes;
  return CUFFT_SUCCESS;
}

cudaError_t check(const void* kernel, size_t smem) {
  std::lock_guard<std::mutex> lock(guard);
  auto it = limits.find({current, kernel});
  const size_t allowed = it == limits.end() ? 48 * 1024 : it->second;
  if (smem > allowed) {
    ++refused;
    return cudaErrorInvalidValue;
  }
  ++launched;
  return cudaSuccess;
}
}  // namespace

extern "C" {

int fake_launched() { return launched; }
int fake_refused() { return refused; }
int fake_lowered() { return lowered; }
int fake_recorded() { return recorded; }
int fake_waited() { return waited; }
void fake_new_stream() { ++stream_id; }  // the handles now belong to new streams
long long fake_held() { return (long long)(held + plan_held); }
void fake_plan_bytes(long long n) { plan_bytes = (size_t)n; }

cudaError_t cudaGetDeviceCount(int* n) { *n = 2; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { current = d; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = current; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) { *s = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaStreamGetId(cudaStream_t, unsigned long long* id) { *id = stream_id; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { ++waited; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { ++recorded; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {  // no more than 1 MB of it is there
  *p = calloc(1, n < (1 << 20) ? n : 1 << 20);
  if (*p == nullptr) return cudaErrorMemoryAllocation;
  sizes[*p] = n;
  held += n;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  held -= sizes[p];
  sizes.erase(p);
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void*, int, size_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }

cudaError_t cudaFuncSetAttribute(const void* kernel, cudaFuncAttribute a, int value) {
  if (a != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaSuccess;
  std::lock_guard<std::mutex> lock(guard);
  size_t& limit = limits[{current, kernel}];
  if ((size_t)value < limit) ++lowered;
  limit = (size_t)value;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* handle, const void* kernel) {
  *handle = (cudaKernel_t)kernel;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t kernel, dim3, dim3, void**, size_t smem, cudaStream_t) {
  return check((const void*)kernel, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* kernel, void**) {
  return check(kernel, c->dynamicSmemBytes);
}

cufftResult cufftCreate(cufftHandle* h) { *h = ++last_plan; return CUFFT_SUCCESS; }
cufftResult cufftDestroy(cufftHandle h) { plan_held -= plans[h]; plans.erase(h); return CUFFT_SUCCESS; }
cufftResult cufftSetStream(cufftHandle, cudaStream_t) { return CUFFT_SUCCESS; }
cufftResult cufftSetAutoAllocation(cufftHandle h, int on) { automatic[h] = on != 0; return CUFFT_SUCCESS; }
cufftResult cufftSetWorkArea(cufftHandle, void*) { return CUFFT_SUCCESS; }
cufftResult cufftMakePlanMany(cufftHandle h, int, int*, int*, int, int, int*, int, int, cufftType, int, size_t* n) {
  *n = plan_bytes;
  return plan_made(h);
}
cufftResult cufftPlanMany(cufftHandle* h, int, int*, int*, int, int, int*, int, int, cufftType, int) {
  *h = ++last_plan;
  return plan_made(*h);
}
cufftResult cufftPlan3d(cufftHandle* h, int, int, int, cufftType) { *h = 1; return CUFFT_SUCCESS; }
cufftResult cufftExecR2C(cufftHandle, cufftReal*, cufftComplex*) { return CUFFT_SUCCESS; }
cufftResult cufftExecD2Z(cufftHandle, cufftDoubleReal*, cufftDoubleComplex*) { return CUFFT_SUCCESS; }
cufftResult cufftExecZ2D(cufftHandle, cufftDoubleComplex*, cufftDoubleReal*) { return CUFFT_SUCCESS; }

}  // extern "C"
