// Pinned memory of a model for the small arrays of a host-pointer run.
//
// Ordinary (pageable) arrays cost a synchronising copy of the driver's each, 10-15 us whatever their size.  Small
// inputs, the results and the status word go through this memory instead: a memcpy here, an asynchronous copy there,
// one synchronisation for the whole run (ResNet-18 int8, one 64x64 image: 226 -> 208 us).  Larger inputs stay with the
// driver, which copies a piece while the GPU fetches the one before it.  Whole calls of one small convolution, driver
// against this memory, us: 75 KB 59.0 / 57.1, 127 KB 63.4 / 60.1, 192 KB 68.8 / 66.5, 243 KB 74.3 / 72.5, 363 KB
// 85.6 / 85.4, 432 KB 92.8 / 102.9, 631 KB 114.6 / 135.4, 2 MB 306 / 337.  So the lines cross near 350 KB; up to there 2-3 us
// are left on the table for a quarter of the pinned memory per model.  Pieces of 64-512 KB filled by one to four threads were
// slower than the driver too (0.6 MB: 240 against 254-290 us, 3.7 MB: 480 against 700 us).
#pragma once

#include <cstdint>
#include <cstring>

#include <cuda_runtime.h>

namespace nb {

class HostStage {
 public:
  static constexpr size_t kInputBytes = 64u << 10;  // all inputs of a run together
  static constexpr size_t kResultBytes = 4u << 20;  // status word and results of a run together

  HostStage() = default;
  HostStage(const HostStage&) = delete;
  HostStage& operator=(const HostStage&) = delete;
  ~HostStage() {
    if (first_ != nullptr) cudaFreeHost(first_);
    if (large_ != nullptr) cudaFreeHost(large_);
  }

  static bool pageable(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
  }

  // The inputs of the next run start at the front again (the run before has ended: its copies are done).
  void begin_run() { used_ = 0; }

  // Queues the copy of one input to the device.
  cudaError_t upload(void* dst, const void* src, size_t bytes, cudaStream_t st) {
    const size_t room = (bytes + 63) / 64 * 64;
    if (used_ + room <= kInputBytes && pageable(src) && open()) {
      uint8_t* at = first_ + used_;
      used_ += room;
      std::memcpy(at, src, bytes);
      src = at;
    }
    return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
  }

  // Pinned memory for the results of one run, or null when it cannot be had.
  uint8_t* result(size_t bytes) {
    if (bytes <= kSmallResult) return open() ? first_ + kInputBytes : nullptr;
    if (bytes <= large_bytes_) return large_;
    size_t want = 2 * kSmallResult;
    while (want < bytes) want *= 2;
    if (want > kResultBytes) return nullptr;
    if (large_ != nullptr) cudaFreeHost(large_);
    large_ = allocate(want);
    large_bytes_ = large_ != nullptr ? want : 0;
    return large_;
  }

 private:
  static constexpr size_t kSmallResult = 64u << 10;
  static uint8_t* allocate(size_t bytes) {
    void* p = nullptr;
    if (cudaHostAlloc(&p, bytes, cudaHostAllocPortable) == cudaSuccess) return static_cast<uint8_t*>(p);
    cudaGetLastError();
    return nullptr;
  }
  // (inputs and small results in one piece: an allocation is a large part of a model's first run)
  bool open() {
    if (first_ == nullptr) first_ = allocate(kInputBytes + kSmallResult);
    return first_ != nullptr;
  }

  uint8_t* first_ = nullptr;
  uint8_t* large_ = nullptr;
  size_t large_bytes_ = 0, used_ = 0;
};

}  // namespace nb
