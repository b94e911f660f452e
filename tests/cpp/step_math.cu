// The FP64 step's exponential, reciprocal and logarithm (tpord_f64.cuh) on
// arrays: step_math <ex2|rcp|lg2> <doubles in> <doubles out>.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>
#include <vector>

#include "tpord.cuh"

__global__ void k_eval(int op, const double *x, double *y, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = op == 0 ? lqt::ex2d(x[i]) : (op == 1 ? lqt::rcpd(x[i]) : lqt::lg2d(x[i]));
}

int main(int argc, char **argv)
{
    if (argc != 4) return 2;
    const int op = !std::strcmp(argv[1], "ex2") ? 0 : (!std::strcmp(argv[1], "rcp") ? 1 : 2);
    std::vector<double> v;
    FILE *f = std::fopen(argv[2], "rb");
    if (!f) return 3;
    for (double d; std::fread(&d, 8, 1, f) == 1;) v.push_back(d);
    std::fclose(f);
    const int n = (int)v.size();
    double *x = nullptr, *y = nullptr;
    if (n == 0 || cudaMalloc((void **)&x, n * 8) != cudaSuccess || cudaMalloc((void **)&y, n * 8) != cudaSuccess) return 4;
    if (cudaMemcpy(x, v.data(), n * 8, cudaMemcpyHostToDevice) != cudaSuccess) return 4;
    k_eval<<<(n + 255) / 256, 256>>>(op, x, y, n);
    if (cudaMemcpy(v.data(), y, n * 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 5;
    f = std::fopen(argv[3], "wb");
    if (!f || (int)std::fwrite(v.data(), 8, n, f) != n) return 6;
    std::fclose(f);
    cudaFree(x);
    cudaFree(y);
    return 0;
}
