// Test-only: the device forms of the functions of kiwi_b200/csrc/fastmath.cuh over arrays, for
// tests/test_gpu_functions.py.
#include "../kiwi_b200/csrc/fastmath.cuh"

using namespace kiwi_b200;

__global__ void k_apply(int which, int n, const double* x, double* y) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double v = x[i];
    y[i] = which == 0 ? fm_rcp(v) : (which == 1 ? fm_rsqrt(v) : (which == 2 ? fm_log(v) : fm_atan01(v)));
}

extern "C" int fm_apply(int which, int n, const double* x, double* y) {
    if (n <= 0 || which < 0 || which > 3) return -1;
    double* d = nullptr;
    if (cudaMalloc(&d, 2 * sizeof(double) * (size_t)n) != cudaSuccess) return -2;
    int rc = cudaMemcpy(d, x, sizeof(double) * (size_t)n, cudaMemcpyHostToDevice) == cudaSuccess ? 0 : -3;
    if (rc == 0) {
        k_apply<<<(n + 255) / 256, 256>>>(which, n, d, d + n);
        if (cudaGetLastError() != cudaSuccess) rc = -4;
    }
    if (rc == 0 && cudaMemcpy(y, d + n, sizeof(double) * (size_t)n, cudaMemcpyDeviceToHost) != cudaSuccess) rc = -5;
    cudaFree(d);
    return rc;
}
