// The shared host copies (csrc/mb_host_copy.cu) on a stand-in CUDA runtime without a device:
// "device" memory is host memory, copies are done at once, and a call can be made to fail.
// Usage: driver SCENARIO; prints one line per copy: its status and whether the bytes are right.
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <atomic>
#include <new>
#include <string>
#include <vector>

template <class T>
T __ldg(const T *p) { return *p; } // named by device code of the header
#include "mb_host_copy.cuh"

static int events_made = 0, event_to_fail = -1; // the event creation that fails
static int events_open = 0, slots_open = 0;
static std::atomic<int> pieces{0}; // copies that crossed to the device and back
static thread_local int news_left = -1; // allocations of this thread until one fails (< 0: none does)

void *operator new(size_t n) {
  if (news_left == 0) throw std::bad_alloc();
  if (news_left > 0) news_left--;
  return malloc(n);
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }

extern "C" {
void **__cudaRegisterFatBinary(void *) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
  if (events_made++ == event_to_fail) return cudaErrorMemoryAllocation;
  events_open++;
  *e = (cudaEvent_t)malloc(1);
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  events_open--;
  free(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { return e ? cudaSuccess : cudaErrorInvalidResourceHandle; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { return e ? cudaSuccess : cudaErrorInvalidResourceHandle; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
  slots_open++;
  *p = malloc(n);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
  slots_open--;
  free(p);
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
  a->type = cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  pieces++;
  memcpy(d, s, n);
  return cudaSuccess;
}
}
namespace mb {
int cuda_fail(cudaError_t e, const char *) { return 1000 + (int)e; }
} // namespace mb

static void copies(mb::HostCopy &c, int times, size_t bytes, int news) {
  std::vector<char> host(bytes), dev(bytes);
  for (int k = 0; k < times; k++) {
    for (size_t i = 0; i < bytes; i++) host[i] = (char)(i * 31 + i / 4096 + k), dev[i] = 0;
    news_left = news;
    const int up = c.to_device(dev.data(), host.data(), bytes, nullptr);
    const bool up_ok = host == dev;
    memset(host.data(), 0, bytes);
    news_left = news;
    const int down = c.to_host(host.data(), dev.data(), bytes, nullptr);
    news_left = -1;
    printf("%d %d %d %d\n", up, (int)up_ok, down, (int)(host == dev));
  }
}

int main(int, char **argv) {
  const std::string scenario = argv[1];
  mb::HostCopy c;
  const size_t big = 40u << 20;
  if (scenario == "event") event_to_fail = 2; // the slots are taken, the third event is not
  // "memory N": every allocation of a copy but the first N fails
  copies(c, 3, big, scenario == "memory" ? atoi(argv[2]) : -1);
  if (scenario == "sizes") // in bytes beyond argv[2], argv[3], ... MiB
    for (int k = 2; argv[k]; k++) {
      pieces = 0;
      copies(c, 1, ((size_t)atoi(argv[k]) << 20) + 12345, -1);
      printf("pieces %d\n", pieces.load());
    }
  c.release();
  printf("left %d %d\n", events_open, slots_open);
  return 0;
}
