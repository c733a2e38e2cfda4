// Device memory of contexts and ensembles (devmem.cuh).
#include "devmem.cuh"

#include <list>
#include <mutex>
#include <unordered_map>

namespace amrvac {

namespace {

struct Reg {
  double *p;
  size_t bytes;
  int dev;
};
struct Registers {
  std::mutex m;
  std::unordered_map<double *, Reg> used;
  std::list<Reg> kept;  // newest first
  size_t kept_bytes = 0;

  void drop(std::list<Reg>::iterator it) {
    kept_bytes -= it->bytes;
    cudaFree(it->p);
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
  auto best = R.kept.end();
  for (auto it = R.kept.begin(); it != R.kept.end(); ++it)
    if (it->dev == dev && it->bytes >= bytes && it->bytes <= bytes + bytes / 4 &&
        (best == R.kept.end() || it->bytes < best->bytes))
      best = it;
  if (best != R.kept.end()) {
    *p = best->p;
    R.used[best->p] = *best;
    R.kept_bytes -= best->bytes;
    R.kept.erase(best);
    return cudaSuccess;
  }
  e = R.alloc(reinterpret_cast<void **>(p), bytes, dev);
  if (e == cudaSuccess) R.used[*p] = Reg{*p, bytes, dev};
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
  R.kept.push_front(it->second);
  R.kept_bytes += it->second.bytes;
  R.used.erase(it);
  // the oldest go first; one above the bound by itself takes no other with it
  if (R.kept.front().bytes > REGISTER_KEEP) R.drop(R.kept.begin());
  while (R.kept_bytes > REGISTER_KEEP) R.drop(std::prev(R.kept.end()));
}

}  // namespace amrvac
