// The straight-line FP64 quotients of eu3d_b200/csrc/common.cuh on host arrays
// (compiled by test_gpu_quotients.py).
#include "../eu3d_b200/csrc/common.cuh"

using namespace eu3d;

__global__ void k_quotients(const double *a, const double *b, long long n, double *q, double *r, double *s)
{
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= n) return;
    q[t] = div_rn(a[t], b[t]);
    r[t] = rcp_rn(fabs(b[t]));
    s[t] = sqrt_rn(fabs(a[t]));
}

extern "C" int quotients(const double *a, const double *b, long long n, double *q, double *r, double *s)
{
    double *d = nullptr;
    if (cudaMalloc(&d, 5 * n * sizeof(double)) != cudaSuccess) return 1;
    cudaMemcpy(d, a, n * sizeof(double), cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, b, n * sizeof(double), cudaMemcpyHostToDevice);
    k_quotients<<<(unsigned)((n + 255) / 256), 256>>>(d, d + n, n, d + 2 * n, d + 3 * n, d + 4 * n);
    cudaMemcpy(q, d + 2 * n, n * sizeof(double), cudaMemcpyDeviceToHost);
    cudaMemcpy(r, d + 3 * n, n * sizeof(double), cudaMemcpyDeviceToHost);
    cudaMemcpy(s, d + 4 * n, n * sizeof(double), cudaMemcpyDeviceToHost);
    const int rc = cudaDeviceSynchronize() != cudaSuccess;
    cudaFree(d);
    return rc;
}
