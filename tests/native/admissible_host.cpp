// Test-only host build of the limiter's division-free admissibility test
// (surely_admissible, emergence_b200/csrc/physics.cuh), compiled by g++ without
// contraction; its fused multiply-adds are explicit.
#include "../../emergence_b200/csrc/physics.cuh"

extern "C" void admissible_check(const double* a, size_t n, unsigned char* out) {
    for (size_t i = 0; i < n; i++) out[i] = emg::surely_admissible(a + 5 * i);
}
