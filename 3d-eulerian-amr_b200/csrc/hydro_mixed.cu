// Mixed-precision hydro: the KT reconstruction and flux in FP32 (FMA
// allowed in this translation unit), fluxes stored in FP64 for the FP64
// coarse-fine correction and conservative update.
#include "flux_kernel.cuh"
#include "kernels.h"
#include "launch.cuh"

namespace amr {

template <int R, FluxBricks B>
__global__ void __launch_bounds__(FluxBlock<OF_12>::THREADS, 2)
    k_flux_f32(Geom g, DevState st, const int* __restrict__ slots, int group) {
    extern __shared__ float flux_smem_f32[];
    flux_staged<float, R, B>(g, st, slots[blockIdx.x], flux_smem_f32, group);
}

namespace {
// one instance for bricks up to 12^3, whose pencils are staged at once
template <int R, FluxBricks B>
void flux_fp32(const Geom& g, const DevState& st, const int* slots, int n, cudaStream_t s) {
    const int group = pencil_group<float, R>(g);
    const size_t smem = staged_smem<float, R>(g, group);
    if (smem > 48 * 1024)
        cudaFuncSetAttribute((const void*)k_flux_f32<R, B>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    launch_k(k_flux_f32<R, B>, dim3(n, 3), PENCIL_PARTS * group, smem, s, g, st, slots, group);
}
template <int R>
void flux_fp32(const Geom& g, const DevState& st, const int* slots, int n, cudaStream_t s) {
    (g.nx <= 12 ? flux_fp32<R, OF_12> : flux_fp32<R, IN_GROUPS>)(g, st, slots, n, s);
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
