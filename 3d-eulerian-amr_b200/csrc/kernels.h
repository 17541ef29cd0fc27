// Launch wrappers of the device kernels (host-callable).
#pragma once

#include <cuda_runtime.h>

#include "amr_internal.h"

namespace amr {

// hydro_kernels.cu
void launch_ghost_fill(const Geom& g, const BrickTable& bt, const DevState& st, const int* slots, int n,
                       cudaStream_t s);
// every level in one launch (trees whose coarse-fine ghosts read none)
void launch_ghost_fill_all(const Geom& g, const BrickTable& bt, const DevState& st, const int* slots, int n,
                           cudaStream_t s);
void launch_flux(const Geom& g, const DevState& st, const int* slots, int n, cudaStream_t s);
// hydro_mixed.cu: FP32 reconstruction + flux (used by launch_flux when g.precision is mixed)
void launch_flux_f32(const Geom& g, const DevState& st, const int* slots, int n, cudaStream_t s);
// every level: items = those whose child's face no item corrects; fixes[6
// slot + face] = items that correct a face, done[6 slot + face] zero between
// launches; with null fixes the items given and no others (one coarse level)
void launch_reflux(const Geom& g, const BrickTable& bt, const DevState& st, const RefluxItem* items, int n,
                   const unsigned char* fixes, unsigned* done, cudaStream_t s);
// with the root's flow-off; dtp: when non-null the step is read from device
// memory (captured graphs)
void launch_add_difs(const Geom& g, const DevState& st, const int* slots, int n, const double* hs, double dt,
                     double beta, int gravity, int root, double* fo, cudaStream_t s, const double* dtp = nullptr);
// whole tree: starts = bricks whose children are all leaves, refined[slot] =
// children of a brick that have children, done[slot] zero between launches
void launch_inject(const Geom& g, const BrickTable& bt, const DevState& st, const int* starts, int n,
                   const int* refined, unsigned* done, cudaStream_t s);
void launch_prolong(const Geom& g, const BrickTable& bt, const DevState& st, const int* slots, int n,
                    cudaStream_t s);
// largest eigenvalue of each direction, lam[3 slot + d]
void launch_max_dt(const Geom& g, const DevState& st, const int* slots, int n, double* lam, cudaStream_t s);
// Grid::max_dt's step of a brick from its three eigenvalues (grid.cpp:470-483)
__host__ __device__ inline double cfl_step(const double* lam, double h, double cfl) {
    double m = 0.0 > lam[0] ? 0.0 : lam[0];
    m = m > lam[1] ? m : lam[1];
    m = m > lam[2] ? m : lam[2];
    double dtinv = m / h;
    if (dtinv == 0.0) dtinv = 1.0E-10;
    double dt = 1.0 / dtinv;
    dt *= cfl;
    return dt;
}
void launch_refine_flags(const Geom& g, const DevState& st, const int* slots, int n, double thr,
                         unsigned char* flags, cudaStream_t s);
void launch_state_max(const Geom& g, const BrickTable& bt, const DevState& st, const int* slots, int n, int field,
                      double* out, cudaStream_t s);

}  // namespace amr

namespace amr {
void launch_gather(const double* src, const int* slots, int n, int count, double* dst, cudaStream_t s);
void launch_scatter(const double* src, const int* slots, int n, int count, double* dst, cudaStream_t s);
}  // namespace amr
