// Quotients and square roots of fcb_arith.cuh beside the operators', elementwise
// (built and driven by test_gpu_arith.py).
#include "fcb_arith.cuh"

__global__ void check(const double* a, const double* b, int n, double* q, double* q0, double* s, double* s0, double* p,
                      double* p0, int* okq, int* oks) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    bool ok = true;
    const fcb::Dv<double> d(b[k], ok);
    q[k] = d(a[k], ok);
    okq[k] = ok;
    q0[k] = a[k] / b[k];
    ok = true;
    s[k] = fcb::sqrt_ok(b[k], ok);
    oks[k] = ok;
    s0[k] = sqrt(b[k]);
    p[k] = fcb::div_pi(a[k]);
    p0[k] = a[k] / 3.141592653589793;
}

extern "C" int run_check(const double* a, const double* b, int n, double* out, int* ok) {
    double *da, *db, *dout;
    int* dok;
    const size_t bytes = (size_t)n * sizeof(double);
    if (cudaMalloc(&da, bytes) || cudaMalloc(&db, bytes) || cudaMalloc(&dout, 6 * bytes) ||
        cudaMalloc(&dok, 2 * (size_t)n * sizeof(int)))
        return 1;
    cudaMemcpy(da, a, bytes, cudaMemcpyHostToDevice);
    cudaMemcpy(db, b, bytes, cudaMemcpyHostToDevice);
    check<<<(n + 255) / 256, 256>>>(da, db, n, dout, dout + n, dout + 2 * n, dout + 3 * n, dout + 4 * n, dout + 5 * n,
                                    dok, dok + n);
    cudaMemcpy(out, dout, 6 * bytes, cudaMemcpyDeviceToHost);
    cudaMemcpy(ok, dok, 2 * (size_t)n * sizeof(int), cudaMemcpyDeviceToHost);
    const int rc = (int)cudaDeviceSynchronize();
    cudaFree(da);
    cudaFree(db);
    cudaFree(dout);
    cudaFree(dok);
    return rc;
}
