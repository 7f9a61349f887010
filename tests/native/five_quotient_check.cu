// Test-only CUDA build: the five-equation closure, maps and HLLC flux in the
// branch-free form (FORM_RN) beside the compiler's division (FORM_DIV), on the
// same primitive states. Built with -fmad=false like the plain sweeps.
#include "../../emergence_b200/csrc/five_physics.cuh"

#include <stddef.h>

namespace {

template <int F> __device__ void evaluate(const emg::Five& s, const double* wl, const double* wr, int un, double* o) {
    using namespace emg;
    const Five::St a = s.state<F>(wl), b = s.state<F>(wr);
    o[0] = a.d;
    o[1] = a.b;
    o[2] = a.rc2;
    o[3] = s.kapila_k<F>(wl);
    o[4] = s.sound_speed_rc2<F>(wl, a.rc2);
    double u[NF], w[NF], d, e;
    s.to_cons<F>(wl, u);
    for (int k = 0; k < NF; k++) o[5 + k] = u[k];
    s.to_prim_db<F>(u, w, d, e);
    for (int k = 0; k < NF; k++) o[12 + k] = w[k];
    double f[NF];
    o[19] = s.riemann_st<F>(wl, wr, a, b, un, f);
    for (int k = 0; k < NF; k++) o[20 + k] = f[k];
    o[27] = s.nc_coef<F>(wr);
}

__global__ void five_kernel(const double* w, double* out, size_t n, emg::FiveSysD sd) {
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const emg::Five s = emg::Five::from(sd);
    double wl[emg::NF], wr[emg::NF];
    for (int k = 0; k < emg::NF; k++) {
        wl[k] = w[14 * i + k];
        wr[k] = w[14 * i + 7 + k];
    }
    double* o = out + 57 * i;
    const int un = emg::F_IU + (int)(i % 3);
    s.begin();
    evaluate<emg::FORM_RN>(s, wl, wr, un, o);
    o[56] = s.bad ? 1.0 : 0.0;
    evaluate<emg::FORM_DIV>(s, wl, wr, un, o + 28);
}

}  // namespace

// w: n pairs of primitive states; eos: (γ, p∞, b, q) of both phases; out: per
// pair 28 values, the same 28 with the compiler's division, range flag
extern "C" int five_check(const double* w_host, double* out_host, size_t n, const double* eos, int kapila) {
    emg::FiveSysD sd{};
    for (int k = 0; k < 2; k++) sd.e[k] = emg::EosD{eos[4 * k], eos[4 * k + 1], eos[4 * k + 2], eos[4 * k + 3]};
    sd.kapila = kapila;
    double *w = nullptr, *out = nullptr;
    int rc = cudaMalloc(&w, 14 * n * sizeof(double)) || cudaMalloc(&out, 57 * n * sizeof(double));
    if (!rc) rc = cudaMemcpy(w, w_host, 14 * n * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess;
    if (!rc) {
        five_kernel<<<(unsigned)((n + 127) / 128), 128>>>(w, out, n, sd);
        rc = cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess;
    }
    if (!rc) rc = cudaMemcpy(out_host, out, 57 * n * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(w);
    cudaFree(out);
    return rc;
}
