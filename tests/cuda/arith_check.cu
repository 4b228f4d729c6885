// The square root of a float pair and the quotient of arith.cuh over arrays of
// operands (host pointers), for the test that compares them with IEEE results.
#include "arith.cuh"

namespace {

__global__ void sqrt_kernel(const float *x, float *out, long n) {
    const long i = 2 * ((long)blockIdx.x * blockDim.x + threadIdx.x);
    if (i + 1 >= n) return;
    const fpb::F2 r = fpb::sqrt2(fpb::pk(x[i], x[i + 1]));
    out[i] = fpb::lo(r);
    out[i + 1] = fpb::hi(r);
}

__global__ void div_kernel(const double *x, const double *y, double *out, long n) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = fpb::div_by(x[i], y[i], 1.0 / y[i]);
}

}  // namespace

// n even. 0 where every call succeeded.
extern "C" int check_sqrt2(const float *x, float *out, long n) {
    float *d = nullptr;
    if (cudaMalloc(&d, 2 * n * sizeof(float)) != cudaSuccess) return 1;
    cudaMemcpy(d, x, n * sizeof(float), cudaMemcpyHostToDevice);
    sqrt_kernel<<<(unsigned)((n / 2 + 255) / 256), 256>>>(d, d + n, n);
    const cudaError_t e = cudaMemcpy(out, d + n, n * sizeof(float), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? 0 : 2;
}

extern "C" int check_div_by(const double *x, const double *y, double *out, long n) {
    double *d = nullptr;
    if (cudaMalloc(&d, 3 * n * sizeof(double)) != cudaSuccess) return 1;
    cudaMemcpy(d, x, n * sizeof(double), cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, y, n * sizeof(double), cudaMemcpyHostToDevice);
    div_kernel<<<(unsigned)((n + 255) / 256), 256>>>(d, d + n, d + 2 * n, n);
    const cudaError_t e = cudaMemcpy(out, d + 2 * n, n * sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? 0 : 2;
}
