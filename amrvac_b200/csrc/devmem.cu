// Device memory of contexts and ensembles (devmem.cuh).
#include "devmem.cuh"

#include <cuda.h>

#include <iterator>
#include <list>
#include <mutex>
#include <unordered_map>
#include <vector>

namespace amrvac {

namespace {

// The driver's identity of an allocation: its context, and an id that no other
// allocation of the process ever has.  A kept register whose identity is not
// what it was went with its context (cudaDeviceReset) and is only forgotten;
// the address may be another's by now.
struct Identity {
  CUcontext ctx = nullptr;
  unsigned long long id = 0;
  bool operator==(const Identity &o) const { return ctx == o.ctx && id == o.id; }
};
template <class F>
F driver_function(const char *name) {
  void *f = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPointByVersion(name, &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
      q != cudaDriverEntryPointSuccess)
    f = nullptr;
  return reinterpret_cast<F>(f);
}
bool identity(void *p, Identity *out) {
  using Get = CUresult (*)(void *, CUpointer_attribute, CUdeviceptr);
  static const Get get = driver_function<Get>("cuPointerGetAttribute");
  const CUdeviceptr d = reinterpret_cast<CUdeviceptr>(p);
  return get && get(&out->ctx, CU_POINTER_ATTRIBUTE_CONTEXT, d) == CUDA_SUCCESS &&
         get(&out->id, CU_POINTER_ATTRIBUTE_BUFFER_ID, d) == CUDA_SUCCESS;
}
CUcontext current_context() {
  using Get = CUresult (*)(CUcontext *);
  static const Get get = driver_function<Get>("cuCtxGetCurrent");
  CUcontext c = nullptr;
  cudaFree(nullptr);  // a thread's first call makes the device's context current
  return get && get(&c) == CUDA_SUCCESS ? c : nullptr;
}

struct Reg {
  double *p;
  size_t bytes;
  int dev;
  Identity is;
  bool there() const {
    Identity now;
    return identity(p, &now) && now == is;
  }
};
struct Registers {
  std::mutex m;
  std::unordered_map<double *, Reg> used;
  std::list<Reg> kept;  // newest first
  size_t kept_bytes = 0;

  void drop(std::list<Reg>::iterator it) {
    kept_bytes -= it->bytes;
    if (it->there()) cudaFree(it->p);
    kept.erase(it);
  }
  // cudaMalloc; with the device short of memory the registers kept there go
  // first (the lock is held)
  cudaError_t alloc(void **p, size_t bytes, int dev) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation && !kept.empty()) {
      cudaGetLastError();
      for (auto it = kept.begin(); it != kept.end();) {
        auto cur = it++;
        if (cur->dev == dev) drop(cur);
      }
      e = cudaMalloc(p, bytes);
    }
    if (e != cudaSuccess) *p = nullptr;
    return e;
  }
};
// (never destroyed: the driver may be gone before static objects are)
Registers &registers() {
  static Registers *r = new Registers;
  return *r;
}

}  // namespace

// The smallest kept register that holds `bytes` with at most a quarter to
// spare (a register is a block count with 25 % headroom), else a new one.
cudaError_t register_alloc(double **p, size_t bytes) {
  *p = nullptr;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  Registers &R = registers();
  std::lock_guard<std::mutex> lock(R.m);
  const CUcontext ctx = R.kept.empty() ? nullptr : current_context();
  for (;;) {
    auto best = R.kept.end();
    for (auto it = R.kept.begin(); it != R.kept.end(); ++it)
      if (it->is.ctx == ctx && it->bytes >= bytes && it->bytes <= bytes + bytes / 4 &&
          (best == R.kept.end() || it->bytes < best->bytes))
        best = it;
    if (best == R.kept.end()) break;
    const Reg r = *best;
    R.kept_bytes -= r.bytes;
    R.kept.erase(best);
    if (!r.there()) continue;
    R.used[r.p] = r;
    *p = r.p;
    return cudaSuccess;
  }
  e = R.alloc(reinterpret_cast<void **>(p), bytes, dev);
  if (e == cudaSuccess) {
    Reg r{*p, bytes, dev, {}};
    if (!identity(*p, &r.is)) r.is.ctx = nullptr;  // not told apart: not kept
    R.used[*p] = r;
  }
  return e;
}

cudaError_t device_alloc(void **p, size_t bytes) {
  *p = nullptr;
  int dev = 0;
  const cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  Registers &R = registers();
  std::lock_guard<std::mutex> lock(R.m);
  return R.alloc(p, bytes, dev);
}

void register_free(double *p) {
  if (!p) return;
  Registers &R = registers();
  std::lock_guard<std::mutex> lock(R.m);
  const auto it = R.used.find(p);
  if (it == R.used.end()) return;
  const Reg r = it->second;
  R.used.erase(it);
  if (!r.is.ctx) {
    cudaFree(p);
    return;
  }
  if (!r.there()) return;
  R.kept.push_front(r);
  R.kept_bytes += r.bytes;
  // the oldest go first; one above the bound by itself takes no other with it
  if (R.kept.front().bytes > REGISTER_KEEP) R.drop(R.kept.begin());
  while (R.kept_bytes > REGISTER_KEEP) R.drop(std::prev(R.kept.end()));
}

namespace {

struct HostPage {
  static constexpr int SLOTS = 256;
  double *p;
  Identity is;  // none: not told apart
  std::vector<int> free;
  bool there() const {
    Identity now;
    return !is.ctx || (identity(p, &now) && now == is);
  }
};
struct HostPages {
  std::mutex m;
  std::list<HostPage> pages;
};
HostPages &host_pages() {
  static HostPages *h = new HostPages;
  return *h;
}

}  // namespace

cudaError_t host_words_alloc(double **host, double **dev) {
  HostPages &H = host_pages();
  std::lock_guard<std::mutex> lock(H.m);
  for (auto it = H.pages.begin(); it != H.pages.end();) {
    auto cur = it++;
    if (!cur->there()) H.pages.erase(cur);  // went with its context
  }
  auto page = H.pages.begin();
  while (page != H.pages.end() && page->free.empty()) ++page;
  if (page == H.pages.end()) {
    HostPage n;
    const cudaError_t e = cudaHostAlloc(reinterpret_cast<void **>(&n.p), sizeof(double) * 2 * HostPage::SLOTS,
                                        cudaHostAllocMapped | cudaHostAllocPortable);
    if (e != cudaSuccess) return e;
    if (!identity(n.p, &n.is)) n.is = Identity();
    for (int q = HostPage::SLOTS; q-- > 0;) n.free.push_back(q);
    H.pages.push_front(n);
    page = H.pages.begin();
  }
  double *const p = page->p + 2 * page->free.back();
  const cudaError_t e = cudaHostGetDevicePointer(reinterpret_cast<void **>(dev), p, 0);
  if (e != cudaSuccess) return e;
  page->free.pop_back();
  *host = p;
  return cudaSuccess;
}

void host_words_free(double *host) {
  if (!host) return;
  HostPages &H = host_pages();
  std::lock_guard<std::mutex> lock(H.m);
  for (HostPage &g : H.pages)
    if (host >= g.p && host < g.p + 2 * HostPage::SLOTS) g.free.push_back((int)(host - g.p) / 2);
}

}  // namespace amrvac
