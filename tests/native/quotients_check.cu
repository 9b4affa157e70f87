// The short quotients and square roots of div64.cuh beside the device's own operators, over
// operand arrays from the caller (see tests/test_quotients_gpu.py).
#include <cuda_runtime.h>

#include "div64.cuh"

// op 0: 1 / b, 1: a / b, 2: sqrt(a).  hard: whether the short form handed the case on.
__global__ void k_quotients(int op, const double *a, const double *b, double *got, double *want, unsigned char *hard,
                            int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    bool h = false;
    double v = 0.0, w = 0.0;
    if (op == 0) {
        v = vx::rcp_rn(b[i], h);
        w = 1.0 / b[i];
        if (h) v = w;
    } else if (op == 1) {
        v = vx::div_rn(a[i], b[i], vx::rcp_ulp(b[i]), h);
        w = a[i] / b[i];
        if (h) v = w;
    } else {
        v = vx::sqrt_rn(a[i], h);
        w = sqrt(a[i]);
        if (h) v = w;
    }
    got[i] = v;
    want[i] = w;
    hard[i] = h;
}

extern "C" int quotients_check(int op, const double *a, const double *b, double *got, double *want,
                               unsigned char *hard, int n) {
    double *da = nullptr, *out = nullptr;
    unsigned char *dh = nullptr;
    const size_t bytes = (size_t)n * sizeof(double);
    if (cudaMalloc(&da, 2 * bytes) || cudaMalloc(&out, 2 * bytes) || cudaMalloc(&dh, n)) return 1;
    cudaMemcpy(da, a, bytes, cudaMemcpyHostToDevice);
    cudaMemcpy(da + n, b, bytes, cudaMemcpyHostToDevice);
    k_quotients<<<(n + 255) / 256, 256>>>(op, da, da + n, out, out + n, dh, n);
    cudaMemcpy(got, out, bytes, cudaMemcpyDeviceToHost);
    cudaMemcpy(want, out + n, bytes, cudaMemcpyDeviceToHost);
    cudaMemcpy(hard, dh, n, cudaMemcpyDeviceToHost);
    const int rc = (int)cudaGetLastError();
    cudaFree(da);
    cudaFree(out);
    cudaFree(dh);
    return rc;
}
