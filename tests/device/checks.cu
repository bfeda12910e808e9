// Device functions of the reader on values that a test chooses.  Built by tests/device/__init__.py.
#include "cfm_device.cuh"

namespace {

__global__ void activate(const float* x, float* out, int n, int activation) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = cfm::pinned_activate(x[i], activation);
}

__global__ void divide(const float* x, const float* d, const float* reciprocal, float* out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = cfm::divide_by_reciprocal(x[i], d[i], reciprocal[i]);
}

int finished() {
  const cudaError_t launched = cudaGetLastError();
  return static_cast<int>(launched != cudaSuccess ? launched : cudaDeviceSynchronize());
}

}  // namespace

extern "C" int check_activate(const float* x, float* out, int n, int activation) {
  activate<<<(n + 255) / 256, 256>>>(x, out, n, activation);
  return finished();
}

extern "C" int check_divide(const float* x, const float* d, const float* reciprocal, float* out, int n) {
  divide<<<(n + 255) / 256, 256>>>(x, d, reciprocal, out, n);
  return finished();
}
