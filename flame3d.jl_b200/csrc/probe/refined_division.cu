// refined_division.cu — common.cuh's refined reciprocals, quotient and reciprocal square root beside
// CUDA's own operators, element by element, for tests/test_refined_division.py.  Built into
// libflame3d_probe.so.
#include "../common.cuh"

namespace {

__global__ void __launch_bounds__(256) k_refined(int op, long long n, const double *a, const double *b,
                                                 double *got, double *want) {
    const long long i = blockIdx.x * 256LL + threadIdx.x;
    if (i >= n) return;
    const double x = a[i], y = b[i];
    switch (op) {
        case 0: got[i] = flame::fast_rcp(x), want[i] = 1.0 / x; break;
        case 1: got[i] = flame::full_rcp(x), want[i] = 1.0 / x; break;
        case 2: got[i] = flame::fast_div(x, y), want[i] = x / y; break;
        case 3: got[i] = flame::fast_rsqrt(x), want[i] = 1.0 / sqrt(x); break;
        case 4: got[i] = flame::rule_sqrt(x), want[i] = sqrt(x); break;
        case 5: got[i] = flame::rule_div(x, y), want[i] = x / y; break;
        default: got[i] = flame::full_div(x, y), want[i] = x / y; break;
    }
}

}  // namespace

// op: 0 fast_rcp, 1 full_rcp, 2 fast_div, 3 fast_rsqrt, 4 rule_sqrt, 5 rule_div, 6 full_div; got from it, want
// from CUDA.  Returns 0, or -1 on a launch error.
extern "C" int flame_probe_refined_division(int op, long long n, const double *a, const double *b,
                                            double *got, double *want, cudaStream_t stream) {
    k_refined<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(op, n, a, b, got, want);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}
