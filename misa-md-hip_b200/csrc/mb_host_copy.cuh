// Copies between device memory and a caller's pageable buffer (mb_host_copy.cu).
#pragma once

#include "mb_common.cuh"

namespace mb {

// One per simulation or ensemble: 8 MiB of page-locked memory from the time that its copies
// have moved enough for it to pay until release().  Calls on one object must not overlap.
struct HostCopy {
  static constexpr int kSlots = 8;
  static constexpr size_t kChunk = 1u << 20;
  static constexpr size_t kMinBytes = 2u << 20; // below: one plain copy is as fast
  // The slots are taken once this much has been moved by an object's copies: to lock 8 MiB
  // takes 6.5 ms, and they save 8 ms of a copy of 54 MiB into fresh pages but 0.3 ms of one of
  // 17 MiB (2.0 against 2.3 ms).
  static constexpr size_t kBigBytes = 32u << 20, kSlotBytes = 64u << 20, kSlotBytesSmall = 512u << 20;
  size_t moved = 0;
  char *slots = nullptr;
  cudaEvent_t ev[kSlots] = {};
  // `bytes` between dev and host, after the work queued on s; done when it returns.
  int to_host(void *host, const void *dev, size_t bytes, cudaStream_t s) {
    return copy(host, const_cast<void *>(dev), bytes, true, s);
  }
  int to_device(void *dev, const void *host, size_t bytes, cudaStream_t s) {
    return copy(const_cast<void *>(host), dev, bytes, false, s);
  }
  void release();

 private:
  int ensure();
  int copy(void *host, void *dev, size_t bytes, bool to_host, cudaStream_t s);
};

} // namespace mb
