// The FP32 form's quotient beside the approximate division of its unit's flags,
// for tests/test_arith.py.
#include "solve.cuh"

using namespace rrsw;

__global__ void k_quot(int n, const float* a, const float* b, float* own, float* cuda) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        own[i] = quot(a[i], b[i]);
        cuda[i] = a[i] / b[i];
    }
}

extern "C" int arith32(int n, const float* a, const float* b, float* own, float* cuda) {
    float* d[4] = {nullptr, nullptr, nullptr, nullptr};
    for (float*& p : d)
        if (cudaMalloc(&p, n * sizeof(float)) != cudaSuccess) return 1;
    cudaMemcpy(d[0], a, n * sizeof(float), cudaMemcpyHostToDevice);
    cudaMemcpy(d[1], b, n * sizeof(float), cudaMemcpyHostToDevice);
    k_quot<<<512, 256>>>(n, d[0], d[1], d[2], d[3]);
    cudaMemcpy(own, d[2], n * sizeof(float), cudaMemcpyDeviceToHost);
    cudaMemcpy(cuda, d[3], n * sizeof(float), cudaMemcpyDeviceToHost);
    for (float* p : d) cudaFree(p);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}
