// the engine's scalar device functions over arrays, for tests/test_gpu_device_functions.py
#include "engine.cuh"
#include "atm_device.cuh"

using namespace komd;

__global__ void k_roots(int n, const double *x, double *y, double *s) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    y[i] = rsqrt_d(x[i]);
    s[i] = sqrt_d(x[i], y[i]);
}
__global__ void k_fix(int n, const float *x, long long *q) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) q[i] = fix32_rn(x[i]);
}

template <typename T>
static T *up(const T *h, size_t n) {
    T *d = nullptr;
    if (cudaMalloc(reinterpret_cast<void **>(&d), sizeof(T) * n) != cudaSuccess) return nullptr;
    if (h) cudaMemcpy(d, h, sizeof(T) * n, cudaMemcpyHostToDevice);
    return d;
}

extern "C" int roots(int n, const double *x, double *y, double *s) {
    double *dx = up(x, n), *dy = up<double>(nullptr, n), *ds = up<double>(nullptr, n);
    if (!dx || !dy || !ds) return 1;
    k_roots<<<(n + 255) / 256, 256>>>(n, dx, dy, ds);
    int rc = cudaMemcpy(y, dy, sizeof(double) * n, cudaMemcpyDeviceToHost);
    rc |= cudaMemcpy(s, ds, sizeof(double) * n, cudaMemcpyDeviceToHost);
    cudaFree(dx);
    cudaFree(dy);
    cudaFree(ds);
    return rc;
}
extern "C" int fix(int n, const float *x, long long *q) {
    float *dx = up(x, n);
    long long *dq = up<long long>(nullptr, n);
    if (!dx || !dq) return 1;
    k_fix<<<(n + 255) / 256, 256>>>(n, dx, dq);
    const int rc = cudaMemcpy(q, dq, sizeof(long long) * n, cudaMemcpyDeviceToHost);
    cudaFree(dx);
    cudaFree(dq);
    return rc;
}
