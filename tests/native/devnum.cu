// Device instantiations of the kernels' short reciprocal, inverse root, wave speed and half-space functions
// on arrays, beside CUDA's own operations where there are any.  Test infrastructure only.
#include "sweep_impl.cuh"

using namespace gkm;
using namespace gkm::sweep_detail;

namespace {
__global__ void recip_kernel(const double* x, long n, double* mine, double* cuda)
{
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    mine[i] = recip<double>(x[i]);
    cuda[i] = 1.0 / x[i];
}
__global__ void rsqrt_kernel(const double* x, long n, double* mine, double* cuda)
{
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    mine[i] = rsqrt_t<double>(x[i]);
    cuda[i] = rsqrt(x[i]);
}
// w: n states of five; the square root of wave_speed_sq beside wave_speed
__global__ void wave_kernel(const double* w, long n, double* mine, double* cuda)
{
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    mine[i] = sqrt(wave_speed_sq(w + 5 * i, 1.4, 1.4 - 1.0));
    cuda[i] = wave_speed(w + 5 * i, 1.4, 1.4 - 1.0);
}
// exp(-x^2/2) and erf(x / sqrt(2)) / 2 of gauss_small
__global__ void gauss_kernel(const double* x, long n, double* ex, double* herf)
{
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    gauss_small<double>(x[i], x[i] * x[i], ex[i], herf[i]);
}
__global__ void gauss_kernel_f32(const double* x, long n, double* ex, double* herf)
{
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float v = (float)x[i];
    float e, h;
    gauss_small<float>(v, v * v, e, h);
    ex[i] = e;
    herf[i] = h;
}
}  // namespace

// which: 0 recip, 1 rsqrt, 2 wave speed, 3 gauss_small, 4 the same in single precision; device arrays
extern "C" int dn_run(int which, const double* in, long n, double* a, double* b)
{
    const unsigned blocks = (unsigned)((n + 255) / 256);
    if (which == 0) recip_kernel<<<blocks, 256>>>(in, n, a, b);
    else if (which == 1) rsqrt_kernel<<<blocks, 256>>>(in, n, a, b);
    else if (which == 2) wave_kernel<<<blocks, 256>>>(in, n, a, b);
    else if (which == 3) gauss_kernel<<<blocks, 256>>>(in, n, a, b);
    else gauss_kernel_f32<<<blocks, 256>>>(in, n, a, b);
    const cudaError_t e = cudaGetLastError();
    return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
