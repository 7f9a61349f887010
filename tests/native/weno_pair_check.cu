// Test-only CUDA build: the paired WENO5-Z interpolations of the fast and mixed
// forms (emergence_b200/csrc/physics.cuh) beside the plain one. Built with the
// mixed sweep's flags.
#include "../../emergence_b200/csrc/physics.cuh"

#include <stddef.h>

namespace {
// out per stencil: fast left, right; mixed left, right; plain left, right
__global__ void pair_kernel(const double* v, double* out, size_t n) {
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    double c[6];
    for (int k = 0; k < 6; k++) c[k] = v[6 * i + k];
    double* o = out + 6 * i;
    emg::weno5z_pair_f(c, o[0], o[1]);
    emg::weno5z_pair_m(c, o[2], o[3]);
    o[4] = emg::weno5z_interp(c[0], c[1], c[2], c[3], c[4]);
    o[5] = emg::weno5z_interp(c[5], c[4], c[3], c[2], c[1]);
}
}  // namespace

extern "C" int pair_check(const double* v_host, double* out_host, size_t n) {
    double *v = nullptr, *out = nullptr;
    int rc = cudaMalloc(&v, 6 * n * sizeof(double)) || cudaMalloc(&out, 6 * n * sizeof(double));
    if (!rc) rc = cudaMemcpy(v, v_host, 6 * n * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess;
    if (!rc) {
        pair_kernel<<<(unsigned)((n + 255) / 256), 256>>>(v, out, n);
        rc = cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess;
    }
    if (!rc) rc = cudaMemcpy(out_host, out, 6 * n * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(v);
    cudaFree(out);
    return rc;
}
