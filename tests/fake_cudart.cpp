// A stand-in for the CUDA runtime on a machine without a GPU: the library's objects linked with it run
// their host code on plain memory, kernels do nothing (a callback sees their name and arguments), and
// an allocation can be made to fail.  For tests of what the host code hands to the kernels and of its
// ways out when a call fails.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

namespace {
std::recursive_mutex mu;
std::map<char*, size_t> live;                // device allocations
struct Kernel { std::string name; int module; };
std::map<const void*, Kernel> kernels;  // by their host stub
int modules = 0;                        // in the order their objects are linked
void* handles[256];
bool used[256];                         // modules whose kernels were launched or asked about
long long fail_in = -1;                      // allocations until one fails (-1: none does)
long long bytes = 0;
cudaError_t last = cudaSuccess;
void (*hook)(const char* kernel, void** args) = nullptr;
struct { dim3 grid, block; size_t smem; void* st; } config;

cudaError_t set(cudaError_t e) { if (e != cudaSuccess) last = e; return e; }
cudaError_t take(void** p, size_t n) {
  std::lock_guard<std::recursive_mutex> l(mu);
  *p = nullptr;
  if (fail_in >= 0 && fail_in-- == 0) return set(cudaErrorMemoryAllocation);
  char* q = static_cast<char*>(calloc(1, n ? n : 1));
  if (!q) return set(cudaErrorMemoryAllocation);
  live[q] = n;
  bytes += (long long)n;
  *p = q;
  return cudaSuccess;
}
cudaError_t give(void* p) {
  std::lock_guard<std::recursive_mutex> l(mu);
  if (!p) return cudaSuccess;
  auto it = live.find(static_cast<char*>(p));
  if (it == live.end()) return set(cudaErrorInvalidValue);
  bytes -= (long long)it->second;
  live.erase(it);
  free(p);
  return cudaSuccess;
}
}  // namespace

extern "C" {

// ---- for the tests
void fake_set_hook(void (*h)(const char*, void**)) { hook = h; }
void fake_fail_in(long long k) { fail_in = k; }
long long fake_fail_left(void) { return fail_in; }
long long fake_live(void) { return (long long)live.size(); }
long long fake_live_bytes(void) { return bytes; }
// bytes from p to the end of the allocation it lies in, -1 outside every one; *base: the allocation
long long fake_room(void* p, void** base) {
  std::lock_guard<std::recursive_mutex> l(mu);
  char* c = static_cast<char*>(p);
  auto it = live.upper_bound(c);
  if (it == live.begin()) return -1;
  --it;
  if (base) *base = it->first;
  return c <= it->first + it->second ? (long long)(it->first + it->second - c) : -1;
}

int fake_module_used(int k) { return k < modules ? used[k] : -1; }

// ---- what nvcc's stubs call
void** __cudaRegisterFatBinary(void*) { return &handles[modules++]; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void** h, const char* stub, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  kernels[stub] = {name, (int)(h - handles)};
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st* st) {
  config = {grid, block, smem, st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* st) {
  *grid = config.grid;
  *block = config.block;
  *smem = config.smem;
  *static_cast<void**>(st) = config.st;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void** args, size_t, cudaStream_t) {
  std::lock_guard<std::recursive_mutex> l(mu);
  used[kernels[f].module] = true;
  if (hook) hook(kernels[f].name.c_str(), args);
  return cudaSuccess;
}

// ---- the runtime
cudaError_t cudaGetLastError(void) { const cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t* p, int) { *p = nullptr; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t, cudaMemPoolAttr, void* v) { memset(v, 0, 8); return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { return take(p, n); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return take(p, n); }
cudaError_t cudaFree(void* p) { return give(p); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return give(p); }
cudaError_t cudaMallocHost(void** p, size_t n) { *p = malloc(n); return *p ? cudaSuccess : set(cudaErrorMemoryAllocation); }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
  if (n < (size_t)1 << 30) memset(d, v, n);  // larger ones would only touch the host's memory
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int) { used[kernels[f].module] = true; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { *p = nullptr; return set(cudaErrorInvalidSymbol); }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* f, int, size_t) {
  used[kernels[f].module] = true;
  *n = 2;
  return cudaSuccess;
}

}  // extern "C"
