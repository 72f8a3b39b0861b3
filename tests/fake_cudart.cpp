// fake_cudart.cpp -- the CUDA runtime calls that the library's host code makes,
// on the CPU: device memory is host memory, streams are in order, a kernel
// launch calls the program's on_launch() and nothing else.  Linked with the
// library's own object files in place of libcudart, it lets a test drive their
// host code (allocation, error paths, launch settings) without a GPU.
#include "fake_cudart.h"

#include <sys/mman.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <utility>

namespace fake {
std::map<const void*, std::string>& kernels() {
  static std::map<const void*, std::string> k;
  return k;
}
std::map<void*, size_t> allocs;  // live device allocations
size_t allocated = 0;
int device = 0;                  // current
int devices = 1;
int num_regs = 128;
// Per device and kernel, as set.
std::map<std::pair<int, const void*>, int> max_dynamic_smem, carveout;
int attribute(const std::map<std::pair<int, const void*>, int>& of, const void* kernel, int unset) {
  const auto it = of.find({device, kernel});
  return it == of.end() ? unset : it->second;
}
cudaError_t last = cudaSuccess;
struct Config {
  dim3 grid, block;
  size_t smem;
} config;
}  // namespace fake

extern "C" {
void** __cudaRegisterFatBinary(void*) { return reinterpret_cast<void**>(&fake::config); }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
char __cudaInitModule(void**) { return 1; }
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*,
                            int*) {
  fake::kernels()[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, CUstream_st*) {
  fake::config = {grid, block, smem};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  *grid = fake::config.grid;
  *block = fake::config.block;
  *smem = fake::config.smem;
  *static_cast<cudaStream_t*>(stream) = nullptr;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* host) {
  *k = reinterpret_cast<cudaKernel_t>(const_cast<void*>(host));
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3 block, void** args, size_t smem, cudaStream_t) {
  const void* host = reinterpret_cast<const void*>(k);
  // More than 48 KiB of dynamic shared memory need the kernel's opt-in on the
  // current device.
  const size_t limit = (size_t)fake::attribute(fake::max_dynamic_smem, host, 48 << 10);
  const cudaError_t e = smem > limit ? cudaErrorInvalidValue
                                     : on_launch(FakeLaunch{fake::kernels()[host], grid, block, smem,
                                                            fake::attribute(fake::carveout, host, -1), args});
  if (e != cudaSuccess) fake::last = e;
  return e;
}

cudaError_t cudaGetLastError() { return std::exchange(fake::last, cudaSuccess); }
cudaError_t cudaGetDeviceCount(int* n) {
  *n = fake::devices;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = fake::device;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {  // asked for the SM count only
  *v = 152;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
  fake::device = d;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) fake::max_dynamic_smem[{fake::device, f}] = v;
  if (a == cudaFuncAttributePreferredSharedMemoryCarveout) fake::carveout[{fake::device, f}] = v;
  return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
  std::memset(a, 0, sizeof(*a));
  a->numRegs = fake::num_regs;
  return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) {
  void* m = mmap(nullptr, n ? n : 1, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
  if (m == MAP_FAILED) return cudaErrorMemoryAllocation;
  fake::allocs[m] = n;
  fake::allocated += n;
  *p = m;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  const auto it = fake::allocs.find(p);
  if (it == fake::allocs.end()) return p ? cudaErrorInvalidValue : cudaSuccess;
  munmap(p, it->second ? it->second : 1);
  fake::allocated -= it->second;
  fake::allocs.erase(it);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = std::calloc(n ? n : 1, 1);
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFreeHost(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
  return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t) {
  for (size_t y = 0; y < h; ++y) std::memcpy(static_cast<char*>(d) + y * dp, static_cast<const char*>(s) + y * sp, w);
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* symbol) {  // a block larger than any of the library's arrays
  static std::map<std::pair<int, const void*>, void*> at;
  void*& m = at[{fake::device, symbol}];
  if (!m) m = std::calloc(16u << 20, 1);
  *p = m;
  return m ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = nullptr;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = nullptr;
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = nullptr;
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 0.0f;
  return cudaSuccess;
}
}  // extern "C"
