// The cell models' double functions (mb_math.cuh) on host arrays, for
// test_cell_math_gpu.py: fn 0 mexp(x), 1 mrcp(x), 2 mdiv(x, y).  Built beside the product
// library by its Makefile, not part of it.
#include "mb_math.cuh"

using namespace mb;

__global__ void k_math_eval(int fn, int n, const double *x, const double *y, double *out) {
    exp_table_fill();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = fn == 0 ? mexp(x[i]) : (fn == 1 ? mrcp(x[i]) : mdiv(x[i], y[i]));
}

extern "C" int math_eval(int fn, int n, const double *x, const double *y, double *out) {
    if (n <= 0) return 0;
    double *d = nullptr;
    const size_t b = (size_t)n * sizeof(double);
    cudaError_t e = cudaMalloc((void **)&d, 3 * b);
    if (e == cudaSuccess) e = cudaMemcpy(d, x, b, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d + n, y, b, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        k_math_eval<<<148, 128>>>(fn, n, d, d + n, d + 2 * (size_t)n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d + 2 * (size_t)n, b, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}
