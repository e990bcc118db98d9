// The stand-in runtime of host_cuda.h.
#include "host_cuda.h"

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>

namespace {
std::mutex mu;
std::map<const void*, std::string>& names() {
  static std::map<const void*, std::string> m;
  return m;
}
std::map<const void*, size_t> smem_limit;
std::map<const void*, void*> symbols;
std::vector<HostLaunch> launches;
std::function<void(const HostLaunch&)> on_launch;
thread_local dim3 cfg_grid, cfg_block;
thread_local size_t cfg_smem;
thread_local cudaStream_t cfg_stream;
thread_local cudaError_t last = cudaSuccess;
// a B200's limits on a block's shared memory
constexpr size_t kSmemDefault = 48 * 1024, kSmemOptIn = 227 * 1024;

cudaError_t set(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}
cudaError_t host_alloc(void** p, size_t n) {
  *p = std::calloc(n ? n : 1, 1);
  return *p ? cudaSuccess : set(cudaErrorMemoryAllocation);
}
}  // namespace

std::vector<HostLaunch> host_launches() {
  std::lock_guard<std::mutex> l(mu);
  return launches;
}
void host_launches_clear() {
  std::lock_guard<std::mutex> l(mu);
  launches.clear();
}
void host_on_launch(std::function<void(const HostLaunch&)> f) {
  std::lock_guard<std::mutex> l(mu);
  on_launch = std::move(f);
}

extern "C" {

void** __cudaRegisterFatBinary(void*) {
  static void* handle;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*,
                            void*, void*, int*) {
  names()[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t s) {
  cfg_grid = g;
  cfg_block = b;
  cfg_smem = smem;
  cfg_stream = s;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
  *g = cfg_grid;
  *b = cfg_block;
  *smem = cfg_smem;
  *(cudaStream_t*)s = cfg_stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void** args, size_t smem,
                             cudaStream_t) {
  HostLaunch h;
  std::function<void(const HostLaunch&)> call;
  {
    std::lock_guard<std::mutex> l(mu);
    const size_t limit = smem_limit.count(f) ? smem_limit[f] : kSmemDefault;
    if (smem > limit || !g.x || !b.x || b.x > 1024) return set(cudaErrorInvalidValue);
    h = {names()[f], g.x, b.x, smem, args, std::this_thread::get_id()};
    launches.push_back(h);
    call = on_launch;
  }
  if (call) call(h);
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  std::lock_guard<std::mutex> l(mu);
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
    if (v < 0 || (size_t)v > kSmemOptIn) return set(cudaErrorInvalidValue);
    smem_limit[f] = (size_t)v;
  }
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* s) {
  std::lock_guard<std::mutex> l(mu);
  if (!symbols[s]) symbols[s] = std::calloc(1, 64);  // nothing reads or writes it
  *p = symbols[s];
  return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) { return host_alloc(p, n); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return host_alloc(p, n); }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) {
  return host_alloc(p, n);
}
cudaError_t cudaFree(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h,
                              cudaMemcpyKind, cudaStream_t) {
  for (size_t r = 0; r < h; ++r) std::memcpy((char*)d + r * dp, (const char*)s + r * sp, w);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : 1;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t e) {
  return e == cudaErrorInvalidValue ? "invalid argument" : "host stand-in error";
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = (cudaStream_t)std::calloc(1, 8);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  std::free((void*)s);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = (cudaGraph_t)std::calloc(1, 8);
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  *e = (cudaGraphExec_t)std::calloc(1, 8);
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
  std::free((void*)g);
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) {
  std::free((void*)e);
  return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) {
  *p = (cudaMemPool_t)std::calloc(1, 8);
  return cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t p) {
  std::free((void*)p);
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = (cudaEvent_t)std::calloc(1, 8);
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  std::free((void*)e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.f;
  return cudaSuccess;
}

}  // extern "C"
