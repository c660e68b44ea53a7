// Copies between device records and a caller's pageable buffer.
//
// cudaMemcpyAsync on pageable memory goes through the driver's own staging buffer on one
// thread: 4.7 GB/s into freshly allocated pages, so that reading 4.2 M records (436 MB) back
// took 92 ms, as long as 45 timesteps.  Here a few host threads share the copy in chunks,
// each with a page-locked slot: the chunk crosses PCIe into the slot while the other threads
// move (and first touch) their parts of the caller's buffer.
#include <string.h>

#include <algorithm>
#include <mutex>
#include <thread>

#include "mb_host_copy.cuh"

namespace mb {

static bool page_locked(const void *host) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type != cudaMemoryTypeUnregistered;
}

// All of it or nothing: a later copy finds the slots with their events, or tries again.
int HostCopy::ensure() {
  if (slots) return MB_OK;
  void *p = nullptr;
  MB_CUDA(cudaHostAlloc(&p, kSlots * kChunk, cudaHostAllocDefault));
  slots = (char *)p;
  for (auto &e : ev) {
    const cudaError_t r = cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
    if (r != cudaSuccess) {
      e = nullptr;
      release();
      return cuda_fail(r, "cudaEventCreateWithFlags");
    }
  }
  return MB_OK;
}

void HostCopy::release() {
  if (slots) cudaFreeHost(slots);
  slots = nullptr;
  for (auto &e : ev)
    if (e) cudaEventDestroy(e), e = nullptr;
}

// Fewer than kMinBytes, a page-locked buffer, or too little moved yet to pay for the slots:
// one plain copy.
int HostCopy::copy(void *host, void *dev, size_t bytes, bool to_host, cudaStream_t s) {
  const cudaMemcpyKind kind = to_host ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice;
  unsigned hw = std::thread::hardware_concurrency();
  const int n_chunks = (int)((bytes + kChunk - 1) / kChunk);
  const int workers = std::min({kSlots, n_chunks, (int)std::max(1u, hw / 2)});
  bool plain = bytes < kMinBytes || workers < 2 || page_locked(host);
  if (!plain && !slots)
    plain = (moved += bytes) < (bytes >= kBigBytes ? kSlotBytes : kSlotBytesSmall) || ensure() != MB_OK;
  if (plain) {
    cudaGetLastError();
    MB_CUDA(to_host ? cudaMemcpyAsync(host, dev, bytes, kind, s) : cudaMemcpyAsync(dev, host, bytes, kind, s));
    MB_CUDA(cudaStreamSynchronize(s));
    return MB_OK;
  }
  int device = 0;
  MB_CUDA(cudaGetDevice(&device));
  std::mutex order; // a slot's copy and its event go into the stream together
  cudaError_t first = cudaSuccess;
  auto worker = [&](int t) {
    cudaError_t r = cudaSetDevice(device);
    char *slot = slots + (size_t)t * kChunk;
    for (int c = t; c < n_chunks && r == cudaSuccess; c += workers) {
      char *h = (char *)host + (size_t)c * kChunk, *d = (char *)dev + (size_t)c * kChunk;
      const size_t n = std::min(kChunk, bytes - (size_t)c * kChunk);
      if (!to_host) {
        if (c != t) r = cudaEventSynchronize(ev[t]); // the slot's last chunk has left
        if (r == cudaSuccess) memcpy(slot, h, n);
      }
      if (r == cudaSuccess) {
        std::lock_guard<std::mutex> lk(order);
        r = to_host ? cudaMemcpyAsync(slot, d, n, kind, s) : cudaMemcpyAsync(d, slot, n, kind, s);
        if (r == cudaSuccess) r = cudaEventRecord(ev[t], s);
      }
      if (to_host) {
        if (r == cudaSuccess) r = cudaEventSynchronize(ev[t]);
        if (r == cudaSuccess) memcpy(h, slot, n);
      }
    }
    if (r != cudaSuccess) {
      std::lock_guard<std::mutex> lk(order);
      if (first == cudaSuccess) first = r;
    }
  };
  // No allocation here but a thread's own, and no exception leaves: a share whose thread
  // does not start (no thread, no memory) is done by this one.
  std::thread threads[kSlots];
  bool own[kSlots] = {true};
  for (int t = 1; t < workers; t++) {
    try {
      threads[t] = std::thread(worker, t);
    } catch (...) {
      own[t] = true;
    }
  }
  for (int t = 0; t < workers; t++)
    if (own[t]) worker(t);
  for (auto &th : threads)
    if (th.joinable()) th.join();
  const cudaError_t end = cudaStreamSynchronize(s); // the slots are free again
  MB_CUDA(first);
  MB_CUDA(end);
  return MB_OK;
}

} // namespace mb
