// The arithmetic of the solves (rt_fastmath.cuh) beside the operators it stands
// for, elementwise, for tests/test_arithmetic_gpu.py.
#include "../legacy-mars-global-climate-model_b200/csrc/rt_fastmath.cuh"

namespace {

// op 0: 1/b, b > 0; 1: 1/b; 2: a/b; 3: sqrt(b); 4: exp(b).
// out[2i]: the fast form, out[2i + 1]: the operator or mgcm_rt_exp.
__global__ void probe(int op, long long n, const double *__restrict__ a, const double *__restrict__ b,
                      double *__restrict__ out) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double x = a[i], y = b[i];
    double f, g;
    switch (op) {
        case 0: f = mgcm::rcp_n(y); g = 1.0 / y; break;
        case 1: f = mgcm::rcp_s(y); g = 1.0 / y; break;
        case 2: f = mgcm::quot(x, y, mgcm::rcp_s(y)); g = x / y; break;
        case 3: f = mgcm::sqrt_n(y); g = sqrt(y); break;
        default: f = mgcm::exp_r(y); g = mgcm_rt_exp(y); break;
    }
    out[2 * i] = f;
    out[2 * i + 1] = g;
}

}  // namespace

// Device pointers; returns the CUDA error code.
extern "C" int arith_probe(int op, long long n, const double *a, const double *b, double *out) {
    if (n <= 0) return 0;
    probe<<<(unsigned)((n + 255) / 256), 256>>>(op, n, a, b, out);
    const cudaError_t e = cudaGetLastError();
    return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
