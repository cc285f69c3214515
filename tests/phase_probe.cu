// Outputs of the quadrature kernels' phase factors and reciprocal square roots
// beside CUDA's own, for test_gpu_phase.py.
#include "phase.cuh"

namespace {

using namespace sieb200;

// out: cos, sin of k x by phase_cs, then by sincos (n of each)
__global__ void phase_kernel(int n, Wave w, const double* __restrict__ x, double* __restrict__ out) {
    __shared__ __align__(16) double2 tab[kTurn * kTurnCopies];
    fill_turn_table(tab);
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double c, s;
    phase_cs(tab + (threadIdx.x & (kTurnCopies - 1)), w, x[i], c, s);
    out[i] = c;
    out[n + i] = s;
    sincos(w.k * x[i], &s, &c);
    out[2 * n + i] = c;
    out[3 * n + i] = s;
}

// out: rsqrt_refined, then rsqrt
__global__ void rsqrt_kernel(int n, const double* __restrict__ x, double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = rsqrt_refined(x[i]);
    out[n + i] = rsqrt(x[i]);
}

}  // namespace

extern "C" int probe_phase(int n, double k, const double* x, double* out) {
    phase_kernel<<<(n + 255) / 256, 256>>>(n, make_wave(k), x, out);
    return (int)cudaDeviceSynchronize();
}

extern "C" int probe_rsqrt(int n, const double* x, double* out) {
    rsqrt_kernel<<<(n + 255) / 256, 256>>>(n, x, out);
    return (int)cudaDeviceSynchronize();
}
