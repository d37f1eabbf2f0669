// Device build of the step loops' reciprocal and square root (rt_fast_math.h) with the
// hardware's seeds, beside the device's own IEEE operations.  Test-only.
#include <cuda_runtime.h>

#include "rt_fast_math.h"

__global__ void fast_kernel(const double* v, long n, double* out) {
    const long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
    if (i >= n) return;
    out[i] = relsim::fast_rcp(v[i]);
    out[n + i] = relsim::fast_sqrt(v[i]);
    out[2 * n + i] = __drcp_rn(v[i]);
    out[3 * n + i] = __dsqrt_rn(v[i]);
}

// out: [4][n]; 0 on success.
extern "C" int device_fast(const double* v, long n, double* out) {
    double* d = nullptr;
    if (n <= 0 || cudaMalloc(&d, sizeof(double) * 5 * n) != cudaSuccess) return 1;
    cudaMemcpy(d, v, sizeof(double) * n, cudaMemcpyHostToDevice);
    fast_kernel<<<static_cast<unsigned>((n + 255) / 256), 256>>>(d, n, d + n);
    const cudaError_t e = cudaMemcpy(out, d + n, sizeof(double) * 4 * n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return static_cast<int>(e);
}
