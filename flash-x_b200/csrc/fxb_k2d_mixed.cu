// Mixed-precision instantiation of the 2-D fused kernel: FP32 reconstruction,
// characteristic projection and Riemann solve; FP64 conserved update,
// internal-energy recovery, Eos and CFL rate.
#include "fxb_launch.h"
namespace fxb {
cudaError_t setup_hydro2d_mixed()
{
    return each_hydro2d<float>([](auto *k) {
        return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem2d_bytes<float>());
    });
}
void launch_hydro2d_mixed(const Args2D &a, dim3 grid, cudaStream_t s) { launch_hydro2d_t<float>(a, grid, s); }
} // namespace fxb
