// A CUDA runtime without a device, for CPU tests of the engine's host side: the
// engine's objects are linked against it (conftest.fake_engine).  Kernels and
// copies do nothing.  What it keeps:
//   memory   addresses that nothing backs, live allocations, bytes in use and
//            their peak, the number of cudaMalloc calls; the n-th can be made to
//            fail; copies and memsets must lie inside an allocation, and only
//            live addresses may be freed
//   launches kernel names, in order; a grid or block past the limits of the
//            hardware fails as cudaErrorInvalidConfiguration
// Device-to-host copies give zeros (so every status word says "done").
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include <cuda_runtime_api.h>

namespace {
std::mutex mu;
std::map<uintptr_t, size_t> live;
uintptr_t top = (uintptr_t)1 << 44;
size_t in_use = 0, peak = 0;
long long mallocs = 0, waits = 0, fail_at = -1;
int misuse = 0;
std::map<const void*, std::string>& names() {
  static std::map<const void*, std::string> m;
  return m;
}
std::vector<std::string> launched;
cudaError_t last = cudaSuccess;
thread_local dim3 cfg_grid, cfg_block;
thread_local size_t cfg_smem;
thread_local void* cfg_stream;

cudaError_t fail(cudaError_t e) {
  last = e;
  return e;
}
bool inside(const void* p, size_t n) {
  const uintptr_t a = (uintptr_t)p;
  auto it = live.upper_bound(a);
  if (it == live.begin()) return false;
  --it;
  return a + n <= it->first + it->second;
}
bool check(const void* p, size_t n) {
  std::lock_guard<std::mutex> l(mu);
  if (n == 0 || inside(p, n)) return true;
  ++misuse;
  return false;
}
cudaError_t copy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
  if (k != cudaMemcpyDeviceToHost && !check(d, n)) return fail(cudaErrorInvalidValue);
  if (k != cudaMemcpyHostToDevice && !check(s, n)) return fail(cudaErrorInvalidValue);
  if (k == cudaMemcpyDeviceToHost) std::memset(d, 0, n);
  return cudaSuccess;
}
cudaError_t launch(const void* f, dim3 g, dim3 b) {
  std::lock_guard<std::mutex> l(mu);
  launched.push_back(names()[f]);
  const bool ok = g.x > 0 && g.y > 0 && g.z > 0 && g.x <= 0x7fffffffu && g.y <= 65535 && g.z <= 65535 &&
                  b.x * b.y * b.z > 0 && b.x * b.y * b.z <= 1024;
  return ok ? cudaSuccess : fail(cudaErrorInvalidConfiguration);
}
int encode(...) { return 0; }
}  // namespace

extern "C" {
// -- what tests read and set ---------------------------------------------------
long long fake_in_use() { return (long long)in_use; }
long long fake_peak() { return (long long)peak; }
long long fake_mallocs() { return mallocs; }
long long fake_waits() { return waits; }
int fake_misuse() { return misuse; }
void fake_reset_peak() { peak = in_use; }
// the n-th cudaMalloc from now on fails (1 = the next; -1: none)
void fake_fail_malloc(long long n) { fail_at = n < 0 ? -1 : mallocs + n; }
// names of the kernels launched since the last call, one per line; their length
int fake_launches(char* buf, int len) {
  std::lock_guard<std::mutex> l(mu);
  std::string s;
  for (const std::string& n : launched) s += n + "\n";
  launched.clear();
  if (buf && len > 0) std::snprintf(buf, (size_t)len, "%s", s.c_str());
  return (int)s.size();
}

// -- registration and launches ---------------------------------------------------
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, void* st) {
  cfg_grid = g, cfg_block = b, cfg_smem = s, cfg_stream = st;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* st) {
  *g = cfg_grid, *b = cfg_block, *s = cfg_smem, *(void**)st = cfg_stream;
  return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) {
  static void* x;
  return &x;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* device, int, void*, void*, void*, void*,
                            int*) {
  names()[host] = device;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void**, size_t, cudaStream_t) { return launch(f, g, b); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  return launch(f, c->gridDim, c->blockDim);
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = 5;
  return cudaSuccess;
}

// -- memory ----------------------------------------------------------------------
cudaError_t cudaMalloc(void** p, size_t n) {
  std::lock_guard<std::mutex> l(mu);
  *p = nullptr;
  if (++mallocs == fail_at) return fail(cudaErrorMemoryAllocation);
  *p = (void*)top;
  live[top] = n;
  top += (n + 511) / 256 * 256;
  in_use += n;
  if (in_use > peak) peak = in_use;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  std::lock_guard<std::mutex> l(mu);
  if (!p) return cudaSuccess;
  auto it = live.find((uintptr_t)p);
  if (it == live.end()) {
    ++misuse;
    return fail(cudaErrorInvalidValue);
  }
  in_use -= it->second;
  live.erase(it);
  return cudaSuccess;
}
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = std::calloc(1, n);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int, size_t n) { return check(p, n) ? cudaSuccess : fail(cudaErrorInvalidValue); }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return cudaMemset(p, v, n); }
cudaError_t cudaMemset2DAsync(void* p, size_t pitch, int v, size_t w, size_t h, cudaStream_t) {
  return h ? cudaMemset(p, v, pitch * (h - 1) + w) : cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) { return copy(d, s, n, k); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
  return copy(d, s, n, k);
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind k,
                              cudaStream_t) {
  for (size_t i = 0; i < h; ++i)
    if (cudaError_t e = copy((char*)d + i * dp, (const char*)s + i * sp, w, k); e != cudaSuccess) return e;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
  static void* block = nullptr;
  if (!block) cudaMalloc(&block, (size_t)64 << 20);
  *p = block;
  return cudaSuccess;
}

// -- device, streams, events, graphs ---------------------------------------------
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* d) {
  *d = 1;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
  *v = 148;  // multiprocessors, the only one asked for
  return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* a, int* b) {
  *a = 0, *b = -5;
  return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char*, void** p, unsigned long long, cudaDriverEntryPointQueryResult* q) {
  *p = (void*)&encode;
  *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "error of the fake runtime"; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
cudaError_t cudaPeekAtLastError() { return last; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = (cudaStream_t)std::malloc(1);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned f, int) { return cudaStreamCreateWithFlags(s, f); }
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  std::free((void*)s);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
  ++waits;
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
// nothing can be captured: steps run uncaptured
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return fail(cudaErrorStreamCaptureUnsupported); }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return fail(cudaErrorStreamCaptureInvalidated); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) {
  return fail(cudaErrorNotSupported);
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return fail(cudaErrorNotSupported); }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = (cudaEvent_t)std::malloc(1);
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  std::free((void*)e);
  return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.0f;
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
}
