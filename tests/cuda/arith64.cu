// The FP64 form's and the adjoint's own arithmetic on arrays, beside CUDA's
// functions, for tests/test_arith.py.
#include <cmath>
#include <vector>

#include "ad.cuh"

using namespace rrsw;

__global__ void k_arith(int n, const double* x, const double* tab, double* own, double* cuda) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double k, rk;
        root64(x[i], k, rk);
        own[0 * n + i] = rcp64(x[i]);
        own[1 * n + i] = sqrt64(x[i]);
        own[2 * n + i] = k;
        own[3 * n + i] = rk;
        cuda[0 * n + i] = 1.0 / x[i];
        cuda[1 * n + i] = cuda[2 * n + i] = ::sqrt(x[i]);
        cuda[3 * n + i] = ::rsqrt(x[i]);
    }
}

__global__ void k_exp(int n, const double* x, const double* tab, double* own, double* cuda) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        expm64(x[i], tab, own[i], own[n + i]);
        cuda[i] = ::exp(-x[i]);
        cuda[n + i] = -::expm1(-x[i]);
    }
}

__global__ void k_index(int n, const double* x, const double*, double* own, double* cuda) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        own[i] = tbl_index64(x[i]);
        cuda[i] = (int)(10000.0 * (x[i] / (cT.bpade + x[i])) + 0.5);
    }
}

// what 0: reciprocals and roots (4 results), 1: exponentials (2), 2: table index (1)
extern "C" int arith64(int what, int n, const double* x, double* own, double* cuda) {
    std::vector<double> tab(2 * EXP2_N);
    for (int j = 0; j < EXP2_N; ++j) {
        tab[2 * j] = std::exp2(-j / 1024.0);
        tab[2 * j + 1] = -std::expm1(-j * (std::log(2.0) / 1024.0));
    }
    static DevTables T{};
    T.exp2 = 0;
    T.total = (int)tab.size();
    T.bpade = 1.0 / 0.278;
    const int nres = what == 0 ? 4 : what == 1 ? 2 : 1;
    double *dx = nullptr, *dt = nullptr, *da = nullptr, *db = nullptr;
    if (cudaMemcpyToSymbol(cT, &T, sizeof(T)) != cudaSuccess) return 1;
    if (cudaMalloc(&dx, n * sizeof(double)) != cudaSuccess) return 1;
    if (cudaMalloc(&dt, tab.size() * sizeof(double)) != cudaSuccess) return 1;
    if (cudaMalloc(&da, (size_t)nres * n * sizeof(double)) != cudaSuccess) return 1;
    if (cudaMalloc(&db, (size_t)nres * n * sizeof(double)) != cudaSuccess) return 1;
    cudaMemcpy(dx, x, n * sizeof(double), cudaMemcpyHostToDevice);
    cudaMemcpy(dt, tab.data(), tab.size() * sizeof(double), cudaMemcpyHostToDevice);
    (what == 0 ? k_arith : what == 1 ? k_exp : k_index)<<<512, 256>>>(n, dx, dt, da, db);
    cudaMemcpy(own, da, (size_t)nres * n * sizeof(double), cudaMemcpyDeviceToHost);
    cudaMemcpy(cuda, db, (size_t)nres * n * sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(dx);
    cudaFree(dt);
    cudaFree(da);
    cudaFree(db);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}
