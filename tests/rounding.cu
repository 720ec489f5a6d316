// The device arithmetic that stands in for CUDA's division and square root, called element by element.
#include <cuda_runtime.h>

#include "rb_device.cuh"

namespace {

__global__ void k_ratio_sqrt(const double* a, const double* v, double* out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = rb::ratio_sqrt(a[i], v[i]);
}
__global__ void k_quotient(const double* a, const double* d, double* out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = rb::quotient(a[i], d[i], 1.0 / d[i]);
}
__global__ void k_sqrt_chain(const double* v, double* out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = rb::sqrt_chain(v[i]);
}

}  // namespace

// device pointers, n elements; waits for the result and returns the CUDA error code
extern "C" int rounding(int what, const double* a, const double* b, double* out, int n) {
    const int blocks = (n + 255) / 256;
    if (what == 0) k_ratio_sqrt<<<blocks, 256>>>(a, b, out, n);
    else if (what == 1) k_quotient<<<blocks, 256>>>(a, b, out, n);
    else k_sqrt_chain<<<blocks, 256>>>(a, out, n);
    const cudaError_t e = cudaGetLastError();
    return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
