// Device memory of one owner (an engine, one tree build): allocations of up to
// 2 MB are cut from 8 MB slabs, larger ones are their own, all are freed
// together.  A cudaMalloc / cudaFree pair costs 20 to 100 us of driver work and
// a free waits for the device; a setup makes over a hundred small ones.
#pragma once

#include <cuda_runtime.h>

#include <vector>

namespace kifmm {

class DeviceArena {
 public:
  DeviceArena() = default;
  DeviceArena(const DeviceArena&) = delete;
  DeviceArena& operator=(const DeviceArena&) = delete;
  ~DeviceArena() { clear(); }
  // frees everything (each free waits for the device)
  void clear() {
    for (void* p : blocks_) cudaFree(p);
    blocks_.clear();
    cur_ = nullptr;
    left_ = 0;
  }
  // `bytes` (at least one) of device memory at a 256-byte boundary
  cudaError_t get(size_t bytes, void** out) {
    constexpr size_t kSlab = (size_t)8 << 20, kSmall = (size_t)2 << 20;
    bytes = (bytes + 255) / 256 * 256;
    if (bytes == 0) bytes = 256;
    if (bytes <= kSmall && bytes <= left_) {
      *out = cur_;
      cur_ += bytes;
      left_ -= bytes;
      return cudaSuccess;
    }
    void* p = nullptr;
    const cudaError_t e = cudaMalloc(&p, bytes <= kSmall ? kSlab : bytes);
    if (e != cudaSuccess) return e;
    blocks_.push_back(p);
    *out = p;
    if (bytes <= kSmall) {  // the rest of the last slab is left unused
      cur_ = (char*)p + bytes;
      left_ = kSlab - bytes;
    }
    return cudaSuccess;
  }

 private:
  std::vector<void*> blocks_;
  char* cur_ = nullptr;
  size_t left_ = 0;
};

}  // namespace kifmm
