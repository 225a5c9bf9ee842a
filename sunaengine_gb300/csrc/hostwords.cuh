// Words in host memory that the device writes (mapped): an engine's digests,
// chains and error word.
#pragma once
#include <cuda_runtime.h>
#include <unistd.h>
#include <cstdint>
#include <cstdlib>
#include <cstring>

namespace sn {

// Whole pages of its own, registered: 14 us to make and give back, where
// cudaHostAlloc and cudaFreeHost took 270 of a small engine's 2 ms.
struct HostWords {
  uint32_t *host = nullptr, *dev = nullptr;
  HostWords() = default;
  HostWords(const HostWords&) = delete;
  HostWords& operator=(const HostWords&) = delete;
  ~HostWords() { release(); }
  cudaError_t alloc(size_t words) {
    const size_t page = (size_t)sysconf(_SC_PAGESIZE), bytes = (words * 4 + page - 1) / page * page;
    void* p = std::aligned_alloc(page, bytes);
    if (!p) return cudaErrorMemoryAllocation;
    std::memset(p, 0, bytes);
    cudaError_t e = cudaHostRegister(p, bytes, cudaHostRegisterMapped);
    if (e != cudaSuccess) {
      std::free(p);
      return e;
    }
    host = static_cast<uint32_t*>(p);
    return cudaHostGetDevicePointer((void**)&dev, host, 0);
  }
  // after the last launch that writes them
  void release() {
    if (!host) return;
    cudaHostUnregister(host);
    std::free(host);
    host = nullptr;
  }
};

}  // namespace sn
