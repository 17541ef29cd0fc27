// Mixed-precision hydro: the KT reconstruction and flux in FP32 (FMA
// allowed in this translation unit), fluxes stored in FP64 for the FP64
// coarse-fine correction and conservative update.
#include "flux_kernel.cuh"
#include "kernels.h"
#include "launch.cuh"

namespace amr {

template <int R>
__global__ void __launch_bounds__(FluxBlock<true>::THREADS, 2) k_flux_f32(Geom g, DevState st, const int* __restrict__ slots) {
    extern __shared__ float flux_smem_f32[];
    flux_staged<float, R>(g, st, slots[blockIdx.x], flux_smem_f32);
}

namespace {
template <int R>
void flux_fp32(const Geom& g, const DevState& st, const int* slots, int n, cudaStream_t s) {
    const size_t smem = staged_smem<float, R>(g);
    if (smem > 48 * 1024)
        cudaFuncSetAttribute((const void*)k_flux_f32<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    launch_k(k_flux_f32<R>, dim3(n, 3), PENCIL_PARTS * g.nx * g.nx, smem, s, g, st, slots);
}
}  // namespace

void launch_flux_f32(const Geom& g, const DevState& st, const int* slots, int n, cudaStream_t s) {
    if (n <= 0) return;
    if (g.recon == RECON_PPM)
        flux_fp32<RECON_PPM>(g, st, slots, n, s);
    else
        flux_fp32<RECON_MINMOD>(g, st, slots, n, s);
}

}  // namespace amr
