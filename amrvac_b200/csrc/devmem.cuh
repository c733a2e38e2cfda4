// Device memory of contexts and ensembles.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace amrvac {

// The large registers of contexts (block registers, the adjoint's, the copy of
// 'average').  Plain cudaMalloc memory, of which the library keeps up to
// REGISTER_KEEP bytes that no context uses: a program that makes and closes
// contexts (adjoint.solve makes two per gradient) otherwise pays for mapping
// and unmapping the same sizes each time.
//
// register_free expects that the caller has waited for all work on the register:
// it is idle, so any context on any stream may have it next.  One larger than
// the bound goes back to the driver at once, as do the oldest above it.
constexpr size_t REGISTER_KEEP = (size_t)256 << 20;
cudaError_t register_alloc(double **p, size_t bytes);
void register_free(double *p);

// cudaMalloc for everything else of the library's: with the device short of
// memory the registers kept on it are given back and it is tried again.
cudaError_t device_alloc(void **p, size_t bytes);
template <class T>
cudaError_t device_alloc(T **p, size_t bytes) {
  return device_alloc(reinterpret_cast<void **>(p), bytes);
}

// Two words of page-locked host memory that kernels write, and their address
// on the current device.  From pages made once per process: a page of a
// context's own cost 2.2 ms to make and 0.3 ms to free.
cudaError_t host_words_alloc(double **host, double **dev);
void host_words_free(double *host);

}  // namespace amrvac
