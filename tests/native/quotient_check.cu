// Test-only CUDA build: the branch-free quotients, square roots and WENO5-Z
// interpolations of emergence_b200/csrc/quotient.cuh beside the compiler's
// division and square root, on the same operands. Built with -fmad=false like
// the plain FP64 sweeps.
#include "../../emergence_b200/csrc/quotient.cuh"

#include <stddef.h>

namespace {

// out per operand pair: quotient, a/b, flag; signed quotient a/−b, its flag;
// 1/b (recip_rn), √b (sqrt_rn), its flag, and the compiler's
__global__ void quotient_kernel(const double* a, const double* b, double* out, size_t n) {
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    double* o = out + 10 * i;
    bool bad = false;
    const emg::RecipRn r = emg::den_rn(b[i], bad);
    o[0] = emg::div_rn(a[i], r, bad);
    o[1] = a[i] / b[i];
    o[2] = bad ? 1.0 : 0.0;
    bad = false;
    o[3] = emg::div_signed_rn(a[i], -b[i], bad);
    o[4] = a[i] / -b[i];
    o[5] = bad ? 1.0 : 0.0;
    o[6] = r.y;
    bad = false;
    o[7] = emg::sqrt_rn(b[i], bad);
    o[8] = bad ? 1.0 : 0.0;
    o[9] = sqrt(b[i]);
}
// out per operand pair: quotient by recip_sq, a/b
__global__ void square_kernel(const double* a, const double* b, double* out, size_t n) {
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[2 * i] = emg::quot_rn(a[i], emg::recip_sq(b[i]));
    out[2 * i + 1] = a[i] / b[i];
}
// six stencil values in; both interpolations, the plain ones, flag out
__global__ void weno_kernel(const double* v, double* out, size_t n) {
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    double c[6];
    for (int k = 0; k < 6; k++) c[k] = v[6 * i + k];
    double* o = out + 5 * i;
    bool bad = false;
    emg::weno5z_pair_rn(c, o[0], o[1], bad);
    o[2] = emg::weno5z_interp(c[0], c[1], c[2], c[3], c[4]);
    o[3] = emg::weno5z_interp(c[5], c[4], c[3], c[2], c[1]);
    o[4] = bad ? 1.0 : 0.0;
}

int run(const double* in0, size_t n0, const double* in1, size_t n1, double* out_host, size_t nout, size_t n, int what) {
    double *a = nullptr, *b = nullptr, *out = nullptr;
    int rc = cudaMalloc(&a, n0 * sizeof(double)) || cudaMalloc(&b, n1 * sizeof(double)) || cudaMalloc(&out, nout * sizeof(double));
    if (!rc) rc = cudaMemcpy(a, in0, n0 * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess;
    if (!rc && in1) rc = cudaMemcpy(b, in1, n1 * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess;
    if (!rc) {
        const unsigned g = (unsigned)((n + 255) / 256);
        if (what == 1)
            weno_kernel<<<g, 256>>>(a, out, n);
        else if (what == 2)
            square_kernel<<<g, 256>>>(a, b, out, n);
        else
            quotient_kernel<<<g, 256>>>(a, b, out, n);
        rc = cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess;
    }
    if (!rc) rc = cudaMemcpy(out_host, out, nout * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(a);
    cudaFree(b);
    cudaFree(out);
    return rc;
}

}  // namespace

extern "C" int quotient_check(const double* a, const double* b, double* out, size_t n) {
    return run(a, n, b, n, out, 10 * n, n, 0);
}
extern "C" int weno_check(const double* v, double* out, size_t n) { return run(v, 6 * n, nullptr, 1, out, 5 * n, n, 1); }
extern "C" int square_check(const double* a, const double* b, double* out, size_t n) {
    return run(a, n, b, n, out, 2 * n, n, 2);
}
