// Single device functions of the solver behind plain C calls, for
// test_gpu_device_functions.py.  Built twice (flash-x_b200/Makefile), the way
// the kernels are: with -fmad=false for FP64 and with fused multiply-adds for
// the mixed path (FXB_TEST_MIXED).
#include "../flash-x_b200/csrc/fxb_device.cuh"

using namespace fxb;

#ifndef FXB_TEST_MIXED
namespace {
template <int N> __global__ void recips_kernel(const double *b, double *y, long n)
{
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    double d[N], r[N];
    for (int q = 0; q < N; q++) d[q] = b[i * N + q];
    recips(d, r);
    for (int q = 0; q < N; q++) y[i * N + q] = r[q];
}
} // namespace
// n groups of `group` (2 or 3) values: recips of each group
extern "C" int fxt_recips(int group, const double *b, double *y, long n)
{
    const unsigned grid = (unsigned)((n + 255) / 256);
    if (group == 2) recips_kernel<2><<<grid, 256>>>(b, y, n);
    else recips_kernel<3><<<grid, 256>>>(b, y, n);
    return (int)cudaDeviceSynchronize();
}
#else
namespace {
__global__ void weno_kernel(int method, const float *I, float *r, float *l, long n)
{
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    weno_scalar(method, I[5 * i], I[5 * i + 1], I[5 * i + 2], I[5 * i + 3], I[5 * i + 4], r[i], l[i]);
}
} // namespace
// n stencils of five values: the interface values at i + 1/2 (r) and i - 1/2 (l)
extern "C" int fxt_weno_mixed(int method, const float *I, float *r, float *l, long n)
{
    weno_kernel<<<(unsigned)((n + 255) / 256), 256>>>(method, I, r, l, n);
    return (int)cudaDeviceSynchronize();
}
#endif
