// A CUDA runtime for tests of the library's host code without a GPU: device
// memory is host memory, kernels do not run, every call is logged, and a call
// can be made to fail.  Linked with the library's own objects in place of
// libcudart (tests/_fakecuda.py).
//
// Log lines: "<function> <arguments> = <error>".
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

namespace {

struct Fail {
  int after, times, err;
};
struct Block {
  size_t bytes;
  int dev;
  unsigned long long id;
};
std::mutex mtx;
std::string logbuf;
std::map<std::string, Fail> fails;
std::map<void *, Block> live;
size_t capacity = (size_t)1 << 40, used = 0;
int cur_dev = 0, nsm = 148;
unsigned long long allocations = 0;
thread_local cudaError_t last = cudaSuccess;

void logf(const char *fmt, ...) {
  char b[256];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(b, sizeof b, fmt, ap);
  va_end(ap);
  logbuf += b;
  logbuf += '\n';
}
// the error that `fn` is to return now
cudaError_t want(const char *fn) {
  auto it = fails.find(fn);
  if (it == fails.end() || !it->second.times) return cudaSuccess;
  if (it->second.after > 0) { --it->second.after; return cudaSuccess; }
  --it->second.times;
  return (cudaError_t)it->second.err;
}
cudaError_t done(const char *fn, const char *args, cudaError_t e) {
  logf("%s %s = %d", fn, args, (int)e);
  if (e != cudaSuccess) last = e;
  return e;
}
cudaError_t plain(const char *fn, const char *args = "") {
  std::lock_guard<std::mutex> g(mtx);
  return done(fn, args, want(fn));
}
cudaError_t alloc(const char *fn, void **p, size_t n, bool device) {
  std::lock_guard<std::mutex> g(mtx);
  cudaError_t e = want(fn);
  if (e == cudaSuccess && device && used + n > capacity) e = cudaErrorMemoryAllocation;
  if (e == cudaSuccess) {
    *p = std::calloc(n ? n : 1, 1);
    live[*p] = Block{device ? n : 0, cur_dev, ++allocations};
    if (device) used += n;
  }
  char a[64];
  std::snprintf(a, sizeof a, "%zu", n);
  return done(fn, a, e);
}
cudaError_t release(const char *fn, void *p) {
  std::lock_guard<std::mutex> g(mtx);
  cudaError_t e = want(fn);
  size_t n = 0;
  if (e == cudaSuccess && p) {
    auto it = live.find(p);
    if (it == live.end()) {
      e = cudaErrorInvalidValue;
    } else {
      n = it->second.bytes;
      used -= n;
      live.erase(it);
      std::free(p);
    }
  }
  char a[64];
  std::snprintf(a, sizeof a, "%zu%s", n, p ? "" : " null");
  return done(fn, a, e);
}

}  // namespace

extern "C" {

// ---- control
void fake_reset() {
  std::lock_guard<std::mutex> g(mtx);
  fails.clear();
  logbuf.clear();
  capacity = (size_t)1 << 40;
  cur_dev = 0;
  nsm = 148;
  last = cudaSuccess;
}
void fake_fail(const char *fn, int after, int times, int err) {
  std::lock_guard<std::mutex> g(mtx);
  fails[fn] = Fail{after, times, err};
}
const char *fake_log() { return logbuf.c_str(); }
void fake_clear_log() { logbuf.clear(); }
size_t fake_used() { return used; }
void fake_capacity(size_t n) { capacity = n; }
void fake_sms(int n) { nsm = n; }
// what a device held goes with its context
void fake_device_reset() {
  std::lock_guard<std::mutex> g(mtx);
  live.clear();
  used = 0;
}

// ---- registration (called when the library is loaded)
void **__cudaRegisterFatBinary(void *) {
  static void *h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, void *, void *, void *, void *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
thread_local struct { dim3 g, b; size_t smem; void *s; } cfg;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void *s) {
  cfg = {g, b, smem, s};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *s) {
  *g = cfg.g; *b = cfg.b; *smem = cfg.smem; *(void **)s = cfg.s;
  return cudaSuccess;
}

// ---- runtime
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaGetDevice(int *d) { *d = cur_dev; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) {
  cur_dev = d;
  char a[16];
  std::snprintf(a, sizeof a, "%d", d);
  return plain("cudaSetDevice", a);
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? nsm : 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
  char a[16];
  std::snprintf(a, sizeof a, "%d", cur_dev);
  return plain("cudaDeviceSynchronize", a);
}
cudaError_t cudaMalloc(void **p, size_t n) { return alloc("cudaMalloc", p, n, true); }
cudaError_t cudaFree(void *p) { return release("cudaFree", p); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return alloc("cudaHostAlloc", p, n, false); }
cudaError_t cudaMallocHost(void **p, size_t n) { return alloc("cudaMallocHost", p, n, false); }
cudaError_t cudaFreeHost(void *p) { return release("cudaFreeHost", p); }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) {
  *d = nullptr;
  const cudaError_t e = plain("cudaHostGetDevicePointer");
  if (e == cudaSuccess) *d = h;
  return e;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
  std::memcpy(d, s, n);
  return plain("cudaMemcpy");
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  return plain("cudaMemcpyAsync");
}
cudaError_t cudaMemset(void *p, int v, size_t n) {
  std::memset(p, v, n);
  return plain("cudaMemset");
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) {
  std::memset(p, v, n);
  return plain("cudaMemsetAsync");
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  *s = (cudaStream_t)1;
  return plain("cudaStreamCreateWithFlags");
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return plain("cudaStreamDestroy"); }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return plain("cudaStreamSynchronize"); }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return plain("cudaStreamBeginCapture"); }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
  *g = (cudaGraph_t)1;
  return plain("cudaStreamEndCapture");
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t, unsigned long long) {
  *x = (cudaGraphExec_t)1;
  return plain("cudaGraphInstantiate");
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return plain("cudaGraphLaunch"); }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return plain("cudaGraphDestroy"); }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return plain("cudaGraphExecDestroy"); }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)1; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **, const void *) { return cudaErrorInvalidSymbol; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return plain("cudaFuncSetAttribute"); }
// as many blocks as 2048 threads and 227 KB of shared memory hold
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int threads, size_t smem,
                                                                  unsigned) {
  *n = 2048 / threads;
  if (smem) *n = std::min(*n, (int)(232448 / (smem + 1024)));
  return cudaSuccess;
}
static cudaError_t launch(dim3 g, dim3 b) {
  char a[64];
  std::snprintf(a, sizeof a, "%u x %u", g.x * g.y * g.z, b.x * b.y * b.z);
  return plain("launch", a);
}
cudaError_t cudaLaunchKernel(const void *, dim3 g, dim3 b, void **, size_t, cudaStream_t) { return launch(g, b); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *, void **) {
  return launch(c->gridDim, c->blockDim);
}

// ---- driver functions, asked for by name
static CUresult context(CUcontext *c) { *c = (CUcontext)(size_t)(1 + cur_dev); return CUDA_SUCCESS; }
static CUresult attribute(void *out, CUpointer_attribute a, CUdeviceptr p) {
  std::lock_guard<std::mutex> g(mtx);
  const auto it = live.find((void *)p);
  if (it == live.end()) return CUDA_ERROR_INVALID_VALUE;
  if (a == CU_POINTER_ATTRIBUTE_CONTEXT) *(CUcontext *)out = (CUcontext)(size_t)(1 + it->second.dev);
  else *(unsigned long long *)out = it->second.id;
  return CUDA_SUCCESS;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char *name, void **f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult *q) {
  *f = !std::strcmp(name, "cuCtxGetCurrent") ? (void *)&context : (void *)&attribute;
  *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}

}  // extern "C"
