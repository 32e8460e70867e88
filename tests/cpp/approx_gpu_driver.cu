// The reciprocal and the reciprocal square root of csrc/common.cuh on a file of
// doubles: approx_gpu_driver (0 reciprocal | 1 rsqrt) IN OUT writes the
// hardware's approximations, then the corrected values.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "common.cuh"

__global__ void evaluate(const double *x, double *raw, double *out, size_t n, int which)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        raw[i] = which ? jsvd::hw_rsqrt(x[i]) : jsvd::hw_reciprocal(x[i]);
        out[i] = which ? jsvd::approx_rsqrt(x[i]) : jsvd::approx_reciprocal(x[i]);
    }
}

int main(int argc, char **argv)
{
    if (argc != 4) return 2;
    FILE *f = fopen(argv[2], "rb");
    if (!f) return 2;
    fseek(f, 0, SEEK_END);
    const size_t n = (size_t)ftell(f) / sizeof(double);
    rewind(f);
    std::vector<double> x(n), y(2 * n);
    if (fread(x.data(), sizeof(double), n, f) != n) return 2;
    fclose(f);
    double *d = nullptr;
    if (cudaMalloc(&d, 3 * n * sizeof(double)) != cudaSuccess) return 1;
    cudaMemcpy(d, x.data(), n * sizeof(double), cudaMemcpyHostToDevice);
    evaluate<<<592, 256>>>(d, d + n, d + 2 * n, n, atoi(argv[1]));
    const cudaError_t e = cudaMemcpy(y.data(), d + n, 2 * n * sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) return 1;
    f = fopen(argv[3], "wb");
    if (!f || fwrite(y.data(), sizeof(double), 2 * n, f) != 2 * n) return 2;
    return fclose(f);
}
