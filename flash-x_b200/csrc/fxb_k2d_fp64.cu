// FP64 instantiation of the 2-D fused kernel (built with -fmad=false).
#include "fxb_launch.h"
namespace fxb {
cudaError_t setup_hydro2d_fp64()
{
    return each_hydro2d<double>([](auto *k) {
        return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem2d_bytes<double>());
    });
}
void launch_hydro2d_fp64(const Args2D &a, dim3 grid, cudaStream_t s) { launch_hydro2d_t<double>(a, grid, s); }
} // namespace fxb
