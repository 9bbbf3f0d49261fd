// The refined reciprocals and roots of the device code at given arguments, for tests/test_gpu_cubic.py.
#include "kemcu_device.cuh"
#include "kemcu_kernels.cuh"
#include "kemcu_axisym.cuh"

__global__ void eval(const double* x, int n, double* out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        out[i] = kemcu::rsqrt_cubic(x[i]);
        out[n + i] = kemcu::rcp_cubic(x[i]);
        out[2 * n + i] = kemcu::sqrt_cubic(x[i]);
        out[3 * n + i] = 0.5 * kemcu::rsqrt2_fast(x[i]);
    }
}

extern "C" int cubic_dev(const double* x, int n, double* out)
{
    double *dx = nullptr, *dout = nullptr;
    int bad = cudaMalloc(&dx, n * sizeof(double)) != cudaSuccess || cudaMalloc(&dout, 4 * n * sizeof(double)) != cudaSuccess;
    if (!bad) {
        bad |= cudaMemcpy(dx, x, n * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess;
        eval<<<(n + 255) / 256, 256>>>(dx, n, dout);
        bad |= cudaMemcpy(out, dout, 4 * n * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess;
    }
    cudaFree(dx);
    cudaFree(dout);
    return bad;
}
