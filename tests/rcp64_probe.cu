// Test helper: the FP64 sweep's reciprocal (rcp64 of csrc/sweep.cuh) of n doubles.  Usage: rcp64_probe <in> <out>
#include <cstdio>
#include <vector>

#include "sweep.cuh"

__global__ void k_rcp(const double *x, double *r, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) r[i] = tcsem::rcp64(x[i]);
}

int main(int argc, char **argv) {
    if (argc < 3) return 2;
    FILE *f = std::fopen(argv[1], "rb");
    if (!f) return 2;
    std::fseek(f, 0, SEEK_END);
    const size_t n = (size_t)std::ftell(f) / sizeof(double);
    std::rewind(f);
    std::vector<double> h(n);
    if (std::fread(h.data(), sizeof(double), n, f) != n) return 2;
    std::fclose(f);
    double *x = nullptr, *r = nullptr;
    if (cudaMalloc(&x, n * sizeof(double)) != cudaSuccess || cudaMalloc(&r, n * sizeof(double)) != cudaSuccess ||
        cudaMemcpy(x, h.data(), n * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess)
        return 1;
    k_rcp<<<(unsigned)((n + 255) / 256), 256>>>(x, r, (int)n);
    if (cudaGetLastError() != cudaSuccess || cudaMemcpy(h.data(), r, n * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess)
        return 1;
    f = std::fopen(argv[2], "wb");
    const bool ok = f && std::fwrite(h.data(), sizeof(double), n, f) == n && std::fclose(f) == 0;
    return ok ? 0 : 1;
}
