// fake_cuda.cpp -- a stand-in for the CUDA runtime, for CPU tests of the
// engine's host code (tests only; linked with the engine's object files).
//
// Device memory is host memory, copies and clears are done at once, and a
// kernel launch does nothing.  What the tests look at: on which stream every
// operation was queued and whether the host waited for it (fake_op), and what
// the engine does when one of these calls (fake_fail) or a host allocation of
// its own (fake_fail_new) fails.
#include <cuda_runtime_api.h>

#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <string>
#include <vector>

namespace {

struct Op {
  std::string what;
  uintptr_t stream;
  int waits;  // 1: complete when the call returns
  const void *at;  // the memory that an allocation gave or a clear wrote ...
  size_t bytes;    // ... and its size
};
std::mutex g_mu;
std::vector<Op> g_ops;
std::map<std::string, int> g_fail;  // call -> the n-th one from now fails (0: the next)
std::map<std::string, cudaError_t> g_fail_code;
thread_local cudaError_t g_last = cudaSuccess;
uintptr_t g_next = 0x1000;
std::atomic<long> g_fail_new{-1};  // the n-th operator new from now fails (0: the next)
thread_local bool t_own = false;   // the log's own allocations do not count

// Logs the call; its error when a test asked for one.
cudaError_t op(const char *what, cudaStream_t s = nullptr, int waits = 0, const void *at = nullptr, size_t bytes = 0) {
  std::lock_guard<std::mutex> lock(g_mu);
  t_own = true;
  cudaError_t e = cudaSuccess;
  auto it = g_fail.find(what);
  if (it != g_fail.end() && it->second-- == 0) {
    g_fail.erase(it);
    e = g_last = g_fail_code[what];
  } else {
    g_ops.push_back(Op{what, (uintptr_t)s, waits, at, bytes});
  }
  t_own = false;
  return e;
}
template <class T>
cudaError_t handle(const char *what, T *out) {
  cudaError_t e = op(what);
  if (e == cudaSuccess) *out = (T)(g_next += 16);
  return e;
}
std::map<void *, size_t> g_device;  // live device allocations
cudaError_t alloc(const char *what, void **p, size_t n) {
  cudaError_t e = op(what);
  if (e != cudaSuccess) return e;
  *p = std::calloc(1, n ? n : 1);
  return *p ? cudaSuccess : (g_last = cudaErrorMemoryAllocation);
}

}  // namespace

void *operator new(size_t n) {
  if (!t_own && g_fail_new.load() >= 0 && g_fail_new.fetch_sub(1) == 0) throw std::bad_alloc();
  if (void *p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }

extern "C" {

// ---- what the tests call ------------------------------------------------------
void fake_clear() {
  std::lock_guard<std::mutex> lock(g_mu);
  g_ops.clear();
  g_fail.clear();
}
// The n-th call of `what` from now (0: the next) fails with `code`.
void fake_fail(const char *what, int n, int code) {
  std::lock_guard<std::mutex> lock(g_mu);
  g_fail[what] = n;
  g_fail_code[what] = (cudaError_t)code;
}
int fake_ops() { return (int)g_ops.size(); }
const char *fake_op(int i, unsigned long long *stream, int *waits) {
  *stream = g_ops[(size_t)i].stream;
  *waits = g_ops[(size_t)i].waits;
  return g_ops[(size_t)i].what.c_str();
}
const void *fake_op_memory(int i, unsigned long long *bytes) {
  *bytes = g_ops[(size_t)i].bytes;
  return g_ops[(size_t)i].at;
}
long long fake_device_bytes() {  // device memory held now
  long long n = 0;
  for (const auto &a : g_device) n += (long long)a.second;
  return n;
}
int fake_device_blocks(long long bytes) {  // device allocations of this size held now
  int n = 0;
  for (const auto &a : g_device) n += a.second == (size_t)bytes;
  return n;
}
int fake_last_error() { return g_last; }
// The n-th host allocation from now fails; -1: none.  Returns the count still to go.
int fake_fail_new(int n) { return (int)g_fail_new.exchange(n); }

// ---- the runtime ----------------------------------------------------------------
cudaError_t cudaMalloc(void **p, size_t n) {
  cudaError_t e = alloc("cudaMalloc", p, n);
  std::lock_guard<std::mutex> lock(g_mu);
  t_own = true;
  if (e == cudaSuccess) {
    g_device[*p] = n;
    g_ops.back().at = *p;
    g_ops.back().bytes = n;
  }
  t_own = false;
  return e;
}
cudaError_t cudaMallocHost(void **p, size_t n) { return alloc("cudaMallocHost", p, n); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return alloc("cudaHostAlloc", p, n); }
cudaError_t cudaFree(void *p) {
  std::lock_guard<std::mutex> lock(g_mu);
  g_device.erase(p);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
// A plain copy to the device may return with its last part under way; one to the host is complete.
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k) {
  cudaError_t e = op("cudaMemcpy", nullptr, k == cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && n) std::memmove(d, s, n);
  return e;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  cudaError_t e = op("cudaMemcpyAsync", st);
  if (e == cudaSuccess && n) std::memmove(d, s, n);
  return e;
}
cudaError_t cudaMemset(void *d, int v, size_t n) {
  cudaError_t e = op("cudaMemset", nullptr, 0, d, n);
  if (e == cudaSuccess && n) std::memset(d, v, n);
  return e;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) {
  cudaError_t e = op("cudaMemsetAsync", st, 0, d, n);
  if (e == cudaSuccess && n) std::memset(d, v, n);
  return e;
}
cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t s) { return op("launch", s); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *, void **) { return op("launch", c->stream); }
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
const char *cudaGetErrorString(cudaError_t) { return "a fake error"; }
cudaError_t cudaDeviceSynchronize() { return op("cudaDeviceSynchronize", nullptr, 1); }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : 1;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int) {  // the header maps the name to its current version
  std::memset(p, 0, sizeof(*p));
  p->major = 10;
  p->multiProcessorCount = 148;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *) { return alloc("cudaMalloc", p, 1 << 20); }
cudaError_t cudaStreamCreate(cudaStream_t *s) { return handle("cudaStreamCreate", s); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return handle("cudaStreamCreate", s); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return op("cudaStreamSynchronize", s, 1); }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return handle("cudaEventCreate", e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return handle("cudaEventCreate", e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }

// ---- registration and <<<>>> ---------------------------------------------------------
static thread_local struct { dim3 g, b; size_t sm; cudaStream_t s; } t_cfg;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t sm, cudaStream_t s) {
  t_cfg = {g, b, sm, s};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *sm, void *s) {
  *g = t_cfg.g;
  *b = t_cfg.b;
  *sm = t_cfg.sm;
  *static_cast<cudaStream_t *>(s) = t_cfg.s;
  return cudaSuccess;
}
static void *g_handle;
void **__cudaRegisterFatBinary(void *) { return &g_handle; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, void *, void *, void *, void *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}

}  // extern "C"
