// A CUDA runtime without a device, for the library's host side: memory is the
// host's, copies and fills happen at once, kernels do nothing.  Linked with the
// library's object files in place of the CUDA runtime (fake_device.py).  It
// keeps the rule that a launch may take more than 48 KB of dynamic shared
// memory only where the kernel was allowed to on the device it is launched on.
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

namespace {
constexpr int kDevices = 4;
std::mutex mu;
std::map<std::pair<int, const void*>, size_t> allowed;  // dynamic shared memory, by device and kernel
size_t refused, largest, free_bytes = (size_t)1 << 40;
std::map<size_t, std::vector<unsigned char>> replies;  // by size
long launches, fail_at = -1, allocations, no_memory_at = -1;
thread_local int device;
thread_local cudaError_t last = cudaSuccess;
thread_local struct {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
} config;

template <class T>
cudaError_t handle(T* out) {
  *out = (T)malloc(16);
  return cudaSuccess;
}

cudaError_t launch(const void* f, size_t smem) {
  std::lock_guard<std::mutex> lk(mu);
  if (launches++ == fail_at) return last = cudaErrorLaunchOutOfResources;
  const auto it = allowed.find({device, f});
  if (smem <= std::max<size_t>(48 << 10, it == allowed.end() ? 0 : it->second)) return cudaSuccess;
  ++refused;
  return last = cudaErrorInvalidValue;
}

cudaError_t take(void** p, size_t n, bool on_device) {
  std::lock_guard<std::mutex> lk(mu);
  if (allocations++ == no_memory_at) return last = cudaErrorMemoryAllocation;
  if (on_device) largest = std::max(largest, n);
  *p = calloc(1, n + 64);
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
}  // namespace

extern "C" {

// launches refused, and the largest device buffer, since the last reset
size_t fake_refused() { return refused; }
size_t fake_largest() { return largest; }
void fake_reset(size_t free_memory) {
  refused = largest = 0;
  free_bytes = free_memory;
  replies.clear();
  launches = allocations = 0;
  fail_at = no_memory_at = -1;
}
// What the next copy of n bytes to the host brings.
void fake_reply(const void* data, size_t n) {
  const unsigned char* p = (const unsigned char*)data;
  replies[n].assign(p, p + n);
}
// The k-th launch from now (from 0) fails; the launches since the last reset.
void fake_fail_at(long k) { fail_at = launches + k; }
long fake_launches() { return launches; }
// The same of allocations, on the device or pinned.
void fake_no_memory_at(long k) { no_memory_at = allocations + k; }
long fake_allocations() { return allocations; }

void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
  *k = (cudaKernel_t)f;
  return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st* stream) {
  config = {grid, block, smem, stream};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  *grid = config.grid;
  *block = config.block;
  *smem = config.smem;
  *(cudaStream_t*)stream = config.stream;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void**, size_t smem, cudaStream_t) {
  return launch((const void*)k, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  return launch(f, c->dynamicSmemBytes);
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  std::lock_guard<std::mutex> lk(mu);
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) allowed[{device, f}] = (size_t)v;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = 1;
  return cudaSuccess;
}

cudaError_t cudaSetDevice(int d) {
  if (d < 0 || d >= kDevices) return last = cudaErrorInvalidDevice;
  device = d;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = device;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr, int) {
  *v = 152;  // asked for multiprocessors only
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "refused by the test's runtime"; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* r) {
  *f = nullptr;
  if (r) *r = cudaDriverEntryPointSymbolNotFound;
  return cudaErrorNotSupported;
}

cudaError_t cudaMalloc(void** p, size_t n) { return take(p, n, true); }
cudaError_t cudaMallocHost(void** p, size_t n) { return take(p, n, false); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return take(p, n, false); }
cudaError_t cudaFree(void* p) {
  free(p);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
  *f = *t = free_bytes;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind kind, cudaStream_t) {
  const auto it = kind == cudaMemcpyDeviceToHost ? replies.find(n) : replies.end();
  memcpy(d, it == replies.end() ? s : it->second.data(), n);
  if (it != replies.end()) replies.erase(it);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
  memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { return cudaMemsetAsync(d, v, n, nullptr); }
cudaError_t cudaMemcpyToSymbol(const void*, const void*, size_t, size_t, enum cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
  static uint64_t room[64];
  *p = room;
  return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return handle(s); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return cudaFree((void*)s); }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, enum cudaStreamCaptureStatus* s) {
  *s = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, enum cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return handle(g); }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return cudaFree((void*)g); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) { return handle(e); }
cudaError_t cudaGraphExecUpdate(cudaGraphExec_t, cudaGraph_t, cudaGraphExecUpdateResultInfo*) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { return cudaFree((void*)e); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return handle(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return handle(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return cudaFree((void*)e); }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 0;
  return cudaSuccess;
}

}  // extern "C"
