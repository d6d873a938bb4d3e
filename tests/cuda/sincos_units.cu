// Sine and cosine of the checkers' fast form (near_sincos) and of the
// clearance (clr::sin_cos, value = high + low), element by element.
#include "clearance_eval.cuh"
#include "near_check.cuh"

__global__ void k_sincos(const float *x, int n, float *near, double *pair)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    prrtc::near_sincos(x[i], near + 2 * i, near + 2 * i + 1);
    prrtc::clr::Dd s, c;
    prrtc::clr::sin_cos(x[i], &s, &c);
    pair[2 * i] = prrtc::clr::to_double(s);
    pair[2 * i + 1] = prrtc::clr::to_double(c);
}

// device pointers; 0 or a CUDA error
extern "C" int units_sincos(const float *x, int n, float *near, double *pair)
{
    k_sincos<<<(n + 127) / 128, 128>>>(x, n, near, pair);
    const cudaError_t e = cudaGetLastError();
    return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
