// Test-only harness: the quotients of the device code (co_quot, over_t of unicorn_b200/csrc/uc_device.cuh) and the
// compiler's divisions of the same operands.
#include "../unicorn_b200/csrc/uc_device.cuh"

__global__ void quotients_kernel(int n, const double *num, const double *den, double *co, double *over, double *div)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        co[i] = uc::co_quot(num[i], den[i]);
        over[i] = uc::over_t(num[i], den[i], 1.0 / den[i]);
        div[i] = num[i] / den[i];
    }
}

// host arrays of n; returns the CUDA error (0: none)
extern "C" int harness_quotients(int n, const double *num, const double *den, double *co, double *over, double *div)
{
    double *d = nullptr;
    const size_t b = (size_t)n * sizeof(double);
    cudaError_t e = cudaMalloc((void **)&d, 5 * b);
    if (e != cudaSuccess) return (int)e;
    if (e == cudaSuccess) e = cudaMemcpy(d, num, b, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d + n, den, b, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        quotients_kernel<<<256, 256>>>(n, d, d + n, d + 2 * (size_t)n, d + 3 * (size_t)n, d + 4 * (size_t)n);
        e = cudaGetLastError();
    }
    double *const out[3] = {co, over, div};
    for (int i = 0; i < 3 && e == cudaSuccess; ++i) e = cudaMemcpy(out[i], d + (2 + i) * (size_t)n, b, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}
