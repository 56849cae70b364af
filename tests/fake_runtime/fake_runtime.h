// A CUDA runtime of the host alone, for checks of what libgpb.so launches: it
// is linked into the check, so its definitions come before libcudart's.
// Device memory is host memory, kernels do nothing, and each launch is
// recorded with the device that was current.  As on a GPU, a launch with more
// than 48 KB of dynamic shared memory is refused unless the kernel was given
// that much on that device.
#pragma once
#include <cuda_runtime.h>
#include <stdlib.h>
#include <string.h>

#include <chrono>
#include <map>
#include <mutex>
#include <string>
#include <thread>
#include <utility>
#include <vector>

struct FakeLaunch {
  int device;
  std::string kernel;  // mangled name
  dim3 grid, block;
  size_t smem;
};
struct FakeRuntime {
  std::mutex mu;
  std::map<const void*, std::string> names;
  std::map<std::pair<int, const void*>, int> smem_max;
  std::vector<FakeLaunch> launches;
  int refused = 0;            // launches without the shared memory they need
  bool fail_attributes = false;
  double ctas(const char* part) {  // of the recorded launches whose kernel's name has this part
    double s = 0;
    for (const FakeLaunch& l : launches)
      if (l.kernel.find(part) != std::string::npos) s += (double)l.grid.x * l.grid.y * l.grid.z;
    return s;
  }
};
inline FakeRuntime& fake() {
  static FakeRuntime* f = new FakeRuntime();
  return *f;
}
inline thread_local int fake_device = 0;
struct FakeConfig {
  dim3 g, b;
  size_t smem;
  void* stream;
};
inline thread_local FakeConfig fake_config;

inline cudaError_t fake_launch(const void* fn, dim3 g, dim3 b, size_t smem) {
  FakeRuntime& f = fake();
  std::lock_guard<std::mutex> lk(f.mu);
  if (smem > 48 * 1024) {
    auto it = f.smem_max.find({fake_device, fn});
    if (it == f.smem_max.end() || (size_t)it->second < smem) {
      f.refused++;
      return cudaErrorInvalidValue;
    }
  }
  if (!g.x || !g.y || !g.z || g.x > 0x7fffffffu || g.y > 65535u || g.z > 65535u) return cudaErrorInvalidConfiguration;
  f.launches.push_back({fake_device, f.names[fn], g, b, smem});
  return cudaSuccess;
}

extern "C" {
void** __cudaRegisterFatBinary(void*) { return (void**)malloc(8); }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  fake().names[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, CUstream_st* stream) {
  fake_config = {g, b, smem, stream};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* stream) {
  *g = fake_config.g, *b = fake_config.b, *smem = fake_config.smem, *(void**)stream = fake_config.stream;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* fn) {
  *k = (cudaKernel_t)fn;
  return cudaSuccess;
}
thread_local cudaError_t fake_last = cudaSuccess;
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void**, size_t smem, cudaStream_t) {
  const cudaError_t e = fake_launch((const void*)k, g, b, smem);
  if (e != cudaSuccess) fake_last = e;
  return e;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* fn, void**) {
  const cudaError_t e = fake_launch(fn, c->gridDim, c->blockDim, c->dynamicSmemBytes);
  if (e != cudaSuccess) fake_last = e;
  return e;
}
cudaError_t cudaFuncSetAttribute(const void* fn, cudaFuncAttribute attr, int v) {
  FakeRuntime& f = fake();
  std::this_thread::sleep_for(std::chrono::milliseconds(2));  // other threads get their chance
  std::lock_guard<std::mutex> lk(f.mu);
  if (f.fail_attributes) return cudaErrorInvalidValue;
  if (attr == cudaFuncAttributeMaxDynamicSharedMemorySize) f.smem_max[{fake_device, fn}] = v;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = fake_last;
  fake_last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetDevice(int* d) { return *d = fake_device, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return fake_device = d, cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { return *n = 2, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { return *p = calloc(n + 1, 1), cudaSuccess; }
cudaError_t cudaFree(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { return *p = calloc(n + 1, 1), cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return *p = calloc(n + 1, 1), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  return memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaMemcpyToSymbolAsync(const void*, const void*, size_t, size_t, cudaMemcpyKind, cudaStream_t) {
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) { return memset(p, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return memset(p, v, n), cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = (cudaStream_t)malloc(1), cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return free(s), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
  return *s = cudaStreamCaptureStatusNone, cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = (cudaEvent_t)malloc(1), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = (cudaEvent_t)malloc(1), cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return free(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.f, cudaSuccess; }
}
