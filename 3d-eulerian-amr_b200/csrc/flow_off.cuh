// Root flow-off: Grid::sum_{x,y,z}_flow_off (grid.cpp:346-404) in the
// sequential order of a one-thread OpenMP run, then the FO update of
// Grid::add_difs (grid.cpp:419).  fo = [FO(nf), FO0(nf)].
//
// One block: its threads form a chunk of the terms, then thread l adds field
// l's in order.  The chain of additions is all that is left of the 28 us that
// one thread per field took over loads and additions, and it runs beside the
// update of the bricks where that is the same launch.
#pragma once

#include "amr_internal.h"
#include "flux_kernel.cuh"

namespace amr {

__device__ __forceinline__ void flow_off_block(const Geom& g, const DevState& st, int root, double h, double dt,
                                               double beta, double* fo) {
    constexpr int CHUNK = 64, NFMAX = 13;
    __shared__ double term[NFMAX][CHUNK];
    const int nx = g.nx, npen = nx * nx, fstride = npen * (nx + 1), l = threadIdx.x;
    double dfo = 0.0;
    for (int d = 0; d < 3; d++) {
        const double* F = (d == 0 ? st.Fx : (d == 1 ? st.Fy : st.Fz)) + (size_t)root * g.nf * fstride;
        for (int p0 = 0; p0 < npen; p0 += CHUNK) {
            const int n = npen - p0 < CHUNK ? npen - p0 : CHUNK;
            for (int q = threadIdx.x; q < g.nf * n; q += blockDim.x) {
                const int f = q / n, p = p0 + q % n, t1 = p % nx, t2 = p / nx;
                const double* Ff = F + f * fstride;
                const double hi = Ff[flux_index(d, nx, nx, t1, t2)];
                term[f][q % n] = d == 2 && g.z_reflect ? hi * h * h
                                                       : (hi - Ff[flux_index(d, nx, 0, t1, t2)]) * h * h;
            }
            __syncthreads();
            if (l < g.nf)
                for (int q = 0; q < n; q++) dfo += term[l][q];
            __syncthreads();
        }
    }
    if (l < g.nf) fo[l] = (fo[l] + dfo * dt) * beta + fo[g.nf + l] * (1.0 - beta);
}

}  // namespace amr
