// dev_math.cu -- test harness: evaluates the FP64 helpers of csrc/tns_device.cuh and
// csrc/tns_adjoint.cuh on the GPU, elementwise, in the forms the kernels call.  Test
// infrastructure only: nothing in the library calls it.
#include "../../2d-turbulent-navier-stokes_b200/csrc/tns_adjoint.cuh"
#include "../../2d-turbulent-navier-stokes_b200/csrc/tns_params.h"

using namespace tns;

__global__ void k_eval(int fn, Params P, long long n, const double* a, const double* b, double* out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double x = a[i], y = b[i];
    double r = 0.0;
    switch (fn) {
        case 0: r = recip(x); break;
        case 1: r = root(x); break;
        case 2: r = quot(x, y); break;
        case 3: r = fifth_roots(x).m04; break;
        case 4: r = fifth_roots(x).m06; break;
        case 5: r = damping(P, x).fmu; break;
        case 6: r = damping(P, x).fr2; break;
        case 7: r = damping_fmu(x); break;
        case 8: r = adj::tanh_work(x).t; break;
        case 9: r = adj::tanh_work(x).inv; break;
        case 10: r = adj::tanh_work(x).d; break;
        case 11: r = inlet_density(P, x); break;
        case 12: r = expm1_nonneg(x); break;
    }
    out[i] = r;
}

// fn over n elements of host arrays; returns the CUDA error (0: none)
extern "C" int dev_math(int fn, const tns_params* prm, long long n, const double* a, const double* b, double* out) {
    double* d = nullptr;
    const size_t bytes = (size_t)n * sizeof(double);
    cudaError_t e = cudaMalloc((void**)&d, 3 * bytes);
    if (e != cudaSuccess) return (int)e;
    if ((e = cudaMemcpy(d, a, bytes, cudaMemcpyHostToDevice)) == cudaSuccess &&
        (e = cudaMemcpy(d + n, b, bytes, cudaMemcpyHostToDevice)) == cudaSuccess) {
        k_eval<<<(unsigned)((n + 255) / 256), 256>>>(fn, make_params(*prm), n, d, d + n, d + 2 * n);
        if ((e = cudaGetLastError()) == cudaSuccess) e = cudaMemcpy(out, d + 2 * n, bytes, cudaMemcpyDeviceToHost);
    }
    cudaFree(d);
    return (int)e;
}

extern "C" double dev_math_fr2k(const tns_params* prm) { return make_params(*prm).fr2k; }
