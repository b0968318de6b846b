// One product of the build's digit GEMM on host arrays: C (M x N) = A (M x K) B (K x N), row-major.
#include "../../ellipticforest_gb300/csrc/ef_gemm64.cu"

#include <atomic>

namespace efgb {
std::atomic<long long> g_kernel_launches{0};
}

extern "C" int digit_product(const double* A, const double* B, double* C, int M, int N, int K) {
    using namespace efgb;
    const size_t a = size_t(M) * K, b = size_t(K) * N, c = size_t(M) * N;
    auto steps = [&](Runner& R, const void* table) {
        const MatView va{PtrTable{table, 0}, 0, K}, vb{PtrTable{table, 0}, (long long)a, N}, vc{PtrTable{table, 0}, (long long)(a + b), N};
        const auto da = R.split(va, M, K, 0), db = R.split(vb, N, K, 1);
        R.gemm(da, db, vc, false, ADD_NONE);
        R.flush();
    };
    Runner dry(nullptr, nullptr, nullptr, 1, true);
    steps(dry, nullptr);
    double* dev = nullptr;
    char* ws = nullptr;
    int err = 1;
    // matrices, then their pointer and the error word
    if (cudaMalloc(&dev, (a + b + c + 2) * sizeof(double)) == cudaSuccess && cudaMalloc(&ws, dry.peak()) == cudaSuccess) {
        double** table = reinterpret_cast<double**>(dev + a + b + c);
        int* word = reinterpret_cast<int*>(table + 1);
        cudaMemcpy(dev, A, a * sizeof(double), cudaMemcpyHostToDevice);
        cudaMemcpy(dev + a, B, b * sizeof(double), cudaMemcpyHostToDevice);
        cudaMemcpy(table, &dev, sizeof(dev), cudaMemcpyHostToDevice);
        cudaMemset(word, 0, sizeof(int));
        Runner R(nullptr, ws, word, 1, false);
        steps(R, table);
        if (cudaMemcpy(C, dev + a + b, c * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess ||
            cudaMemcpy(&err, word, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)
            err = 1;
    }
    cudaFree(ws);
    cudaFree(dev);
    return err;
}
