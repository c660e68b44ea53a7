// Stand-in CUDA runtime without a device: each device keeps its own limit of dynamic shared
// memory per kernel, as the driver does, and a launch beyond it is refused.
#include <cuda_runtime_api.h>

#include <map>
#include <utility>
#include <vector>

int device = 0;
static std::map<std::pair<int, const void *>, int> limits;
static cudaError_t launch(const void *f, size_t smem) {
  auto l = limits.find({device, f});
  return smem <= (size_t)(l == limits.end() ? 48 * 1024 : l->second) ? cudaSuccess : cudaErrorInvalidValue;
}
struct Call {
  dim3 grid, block;
  size_t smem;
  cudaStream_t s;
};
static std::vector<Call> calls;
static cudaError_t last = cudaSuccess;

extern "C" {
void **__cudaRegisterFatBinary(void *) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t s) {
  calls.push_back({g, b, smem, s});
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *s) {
  const Call c = calls.back();
  calls.pop_back();
  *g = c.grid, *b = c.block, *smem = c.smem, *(cudaStream_t *)s = c.s;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) { return *d = device, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 148, cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute, int v) {
  if (v > 227 * 1024) return cudaErrorInvalidValue;
  return limits[{device, f}] = v, cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3, dim3, void **, size_t smem, cudaStream_t) {
  return last = launch(f, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **) {
  return launch(f, c->dynamicSmemBytes);
}
cudaError_t cudaGetLastError() {
  const cudaError_t r = last;
  last = cudaSuccess;
  return r;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int, size_t smem, unsigned) {
  return *n = 1, launch(f, smem);
}
const char *cudaGetErrorString(cudaError_t) { return "refused"; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
}
