// devbuf.cuh -- device scratch of one call, from the stream-ordered pool.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>

#include "common.cuh"

namespace lkg {

// Device scratch from the stream-ordered pool: allocation and release are queued on the stream (no device-wide
// synchronisation when many submodels predict concurrently), and the device's default pool keeps up to 8 GiB of
// released memory for reuse (raised from its default of none, never lowered).
inline void keep_pool_memory() {
  static std::once_flag once;
  std::call_once(once, [] {
    int dev = 0;
    LKG_CUDA(cudaGetDevice(&dev));
    cudaMemPool_t pool;
    LKG_CUDA(cudaDeviceGetDefaultMemPool(&pool, dev));
    uint64_t keep = 0;
    LKG_CUDA(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    const uint64_t want = (uint64_t)8 << 30;
    if (keep < want) LKG_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, (void*)&want));
  });
}

struct DevBuf {
  double* p = nullptr;
  cudaStream_t st;
  DevBuf(size_t n, cudaStream_t s) : st(s) {
    keep_pool_memory();
    LKG_CUDA(cudaMallocAsync((void**)&p, sizeof(double) * std::max<size_t>(n, 1), st));
  }
  ~DevBuf() {
    if (p) cudaFreeAsync(p, st);
  }
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
};

}  // namespace lkg
