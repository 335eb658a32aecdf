// For the tests: fills the shared memory of every SM with one value, so that a kernel launched next finds that where nothing has been
// written (shared memory is not cleared between launches).  One block takes all the shared memory of an SM; four times as many
// blocks as SMs, so that every SM gets one.
#include <cstdint>
#include <cuda_runtime.h>

namespace {
constexpr int kBytes = 227 * 1024;

__global__ void fill_shared_kernel(uint32_t value) {
  extern __shared__ uint32_t words[];
  volatile uint32_t* w = words;
  for (int i = threadIdx.x; i < kBytes / 4; i += blockDim.x) w[i] = value;
}
}  // namespace

extern "C" __attribute__((visibility("default"))) int test_fill_shared(uint32_t value, void* stream) {
  int device = 0, sms = 0;
  cudaGetDevice(&device);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  cudaError_t e = cudaFuncSetAttribute(fill_shared_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
  if (e != cudaSuccess) return int(e);
  fill_shared_kernel<<<4 * sms, 1024, kBytes, static_cast<cudaStream_t>(stream)>>>(value);
  return int(cudaGetLastError());
}
