// phys::rcp and phys::root over an array (tests/test_gpu_rcp_root.py)
#include "device/physics.cuh"

__global__ void apply(int what, int n, const double* x, double* y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = what == 0 ? dgb::phys::rcp(x[i]) : dgb::phys::root(x[i]);
}

extern "C" int rcp_root(int what, int n, const double* x_dev, double* y_dev) {
  apply<<<(n + 255) / 256, 256>>>(what, n, x_dev, y_dev);
  return (int)cudaDeviceSynchronize();
}
