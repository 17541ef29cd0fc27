// KT/Rusanov face fluxes, Grid::compute_{x,y,z}_flux (grid.cpp:215-302),
// with minmod-theta (reconstruct.cpp:60-71) or PPM (reconstruct.cpp:22-58)
// reconstruction, templated on the arithmetic type: double is the plain form
// (instantiated in hydro_kernels.cu, no FMA contraction), float the mixed
// form's FP32 reconstruction and flux (hydro_mixed.cu) whose fluxes are
// stored in FP64 and accumulated in FP64 by the conservative update.
//
// Block = (brick, direction), three threads a pencil of nx + 1 faces; the
// pencils' primitives are formed once a cell and staged in shared memory (37
// KB for 8^3 bricks of bw 2, 44 KB of bw 3), and each thread streams the
// reconstruction (recon.cuh) over its part.  The latency of FP64 divisions and
// square roots with few warps in flight bounds it, not memory.  One thread a
// pencil over all its cells from global memory, a block a brick, took 25.6 us
// for 25 bricks and 69 us for 527 (minmod), 101 us for 541 (PPM), against
// 11.8, 51.8 and 90 us now.
#pragma once

#include "recon.cuh"

namespace amr {

// index of flux array element for direction d: face index fi (0..nx) along d,
// transverse interior indices t1 (lower axis) and t2 (higher axis).
__device__ __forceinline__ int flux_index(int d, int nx, int fi, int t1, int t2) {
    if (d == 0) return (t2 * nx + t1) * (nx + 1) + fi;
    if (d == 1) return (t2 * (nx + 1) + fi) * nx + t1;
    return (fi * nx + t2) * nx + t1;
}

__device__ __forceinline__ int cell_index(int gnx, int i, int j, int k) { return (k * gnx + j) * gnx + i; }

// KT flux of one face from its reconstructed primitive states, to F (stride
// fstride between fields).
template <typename T, int d>
__device__ __forceinline__ void kt_flux(T* ql, T* qr, T gam, double* F, int fstride) {
    st_to_con(ql);
    st_to_con(qr);
    T fl[NF_EULER], fr[NF_EULER];
    const T al = st_flux(ql, d, gam, fl);
    const T ar = st_flux(qr, d, gam, fr);
    const T a = r_max(al, ar);
#pragma unroll
    for (int l = 0; l < NF_EULER; l++)
        F[l * fstride] = (double)(((fl[l] + fr[l]) - (qr[l] - ql[l]) * a) * T(0.5));
}

// Cells on each side of a face's two that its reconstruction reads, and the
// threads of a pencil in the staged kernels.
template <int R>
__host__ __device__ constexpr int recon_reach() { return R == 1 ? 2 : 1; }
constexpr int PENCIL_PARTS = 3;
// Which bricks an instance is for, and its register budget: 4^3 and 8^3 ones
// in blocks of at most 192 threads, three to an SM (96 registers: of the 18
// warps five share a quarter of the SM; fluxes spill 256 bytes with minmod, 612
// with PPM, the PPM eigenvalues 528); 12^3 ones in blocks of 432, one to an SM
// (128 registers, PPM fluxes spill 116 bytes); larger ones in groups of at most 64 pencils, one group after
// the other in a block of 192 (all of a 16^3 brick's pencils would be 768
// threads and 247 KB).  THREADS is whole warps, as the CFL kernel is launched
// (its 432 are 448).
enum FluxBricks { UP_TO_8, OF_12, IN_GROUPS };
template <FluxBricks B>
struct FluxBlock {
    static constexpr int THREADS = (PENCIL_PARTS * (B == OF_12 ? 144 : 64) + 31) / 32 * 32, PER_SM = B == OF_12 ? 1 : 3;
};

// Shared memory of a block that stages `group` pencils, [field][cell of the
// pencil][pencil] with the pencils padded so that staging x pencils has no
// bank conflicts.
template <typename T, int R>
inline size_t staged_smem(const Geom& g, int group) {
    const int cells = g.nx + 2 * (recon_reach<R>() + 1);
    return sizeof(T) * NF_EULER * cells * (size_t)(group + 1);
}
// Pencils that a block stages at a time: all of a direction's up to 12^3
// bricks, else as many of 64 as shared memory has room for (64 up to 68^3).
template <typename T, int R>
inline int pencil_group(const Geom& g) {
    if (g.nx <= 12) return g.nx * g.nx;
    int group = 64;
    while (group > 1 && staged_smem<T, R>(g, group) > 226 * 1024) group /= 2;
    return group;
}

// Stages the primitives of every cell that the faces read (grid cells
// bw - reach - 1 ...) of direction d's pencils p0 .. p0 + np - 1.
template <typename T, int d, int R>
__device__ __forceinline__ void stage_pencils(const Geom& g, const double* Ub, T* P, int p0, int np) {
    const int nx = g.nx, first = g.bw - recon_reach<R>() - 1, cells = nx + 2 * (recon_reach<R>() + 1);
    for (int q = threadIdx.x; q < np * cells; q += blockDim.x) {
        // neighbouring threads on neighbouring cells in memory
        const int n = d == 0 ? q % cells : q / np, p = d == 0 ? q / cells : q % np;
        const int t1 = (p0 + p) % nx + g.bw, t2 = (p0 + p) / nx + g.bw, m = first + n;
        const int ci = d == 0 ? cell_index(g.gnx, m, t1, t2)
                              : (d == 1 ? cell_index(g.gnx, t1, m, t2) : cell_index(g.gnx, t1, t2, m));
        T w[NF_EULER];
#pragma unroll
        for (int l = 0; l < NF_EULER; l++) w[l] = (T)Ub[l * g.gnx3 + ci];
        st_to_prim(w);
#pragma unroll
        for (int l = 0; l < NF_EULER; l++) P[(l * cells + n) * (np + 1) + p] = w[l];
    }
    __syncthreads();
}

// Cell n of a staged pencil; the reconstructions start as at face
// recon_reach + 1 of a pencil whose cell 0 is the first one they read.
template <typename T>
struct StagedLoad {
    const T* P;  // cell 0 of this thread's first face
    int row, field;
    __device__ __forceinline__ void operator()(int n, T* q) const {
#pragma unroll
        for (int l = 0; l < NF_EULER; l++) q[l] = P[l * field + n * row];
    }
};

// Calls f(face 0..nx, ql, qr) for this thread's part of its pencil's faces, np
// pencils being staged.
template <typename T, int R, class F>
__device__ __forceinline__ void staged_faces(const Geom& g, const T* P, int np, F f) {
    const int nx = g.nx, cells = nx + 2 * (recon_reach<R>() + 1);
    const int p = threadIdx.x % np, part = threadIdx.x / np;
    const int each = (nx + PENCIL_PARTS) / PENCIL_PARTS;
    const int f0 = part * each, f1 = min(f0 + each, nx + 1);
    if (f0 >= f1) return;
    StagedLoad<T> load{P + f0 * (np + 1) + p, np + 1, cells * (np + 1)};
    constexpr int START = recon_reach<R>() + 1;  // the face f0 in load's frame
    PencilRecon<T, R> rec;
    rec.begin(load, START, (T)g.theta);
    for (int q = f0; q < f1; q++) {
        T ql[NF_EULER], qr[NF_EULER];
        rec.next(load, START + q - f0, ql, qr);
        f(q, ql, qr);
    }
}

// Fluxes of direction d's pencils p0 .. p0 + np - 1, staged together.
template <typename T, int d, int R>
__device__ __forceinline__ void flux_pencils(const Geom& g, const DevState& st, int b, T* P, int p0, int np) {
    const int nx = g.nx, fstride = nx * nx * (nx + 1);
    stage_pencils<T, d, R>(g, st.U + (size_t)b * g.ucount, P, p0, np);
    double* F = (d == 0 ? st.Fx : (d == 1 ? st.Fy : st.Fz)) + (size_t)b * g.nf * fstride;
    const int t1 = (p0 + threadIdx.x % np) % nx, t2 = (p0 + threadIdx.x % np) / nx;
    staged_faces<T, R>(g, P, np, [&](int q, T* ql, T* qr) {
        kt_flux<T, d>(ql, qr, (T)g.gamma, F + flux_index(d, nx, q, t1, t2), fstride);
    });
}

// ... of every pencil
template <typename T, int d, int R, FluxBricks B>
__device__ __forceinline__ void flux_staged_dir(const Geom& g, const DevState& st, int b, T* P, int group) {
    if constexpr (B != IN_GROUPS) {
        flux_pencils<T, d, R>(g, st, b, P, 0, g.nx * g.nx);
    } else {
        const int npen = g.nx * g.nx;
        for (int p0 = 0; p0 < npen; p0 += group) {
            if (p0) __syncthreads();  // the last group's faces are done with the staged cells
            flux_pencils<T, d, R>(g, st, b, P, p0, min(group, npen - p0));
        }
    }
}

// grid = (bricks, 3 directions), PENCIL_PARTS threads for each pencil staged
template <typename T, int R, FluxBricks B>
__device__ __forceinline__ void flux_staged(const Geom& g, const DevState& st, int b, T* P, int group) {
    if (blockIdx.y == 0) flux_staged_dir<T, 0, R, B>(g, st, b, P, group);
    else if (blockIdx.y == 1) flux_staged_dir<T, 1, R, B>(g, st, b, P, group);
    else flux_staged_dir<T, 2, R, B>(g, st, b, P, group);
}

// Largest face eigenvalue of those pencils ...
template <int d, int R>
__device__ __forceinline__ double max_eigen_pencils(const Geom& g, const DevState& st, int b, double* P, int p0,
                                                    int np) {
    stage_pencils<double, d, R>(g, st.U + (size_t)b * g.ucount, P, p0, np);
    double lam = 0.0;
    staged_faces<double, R>(g, P, np, [&](int, double* ql, double* qr) {
        st_to_con(ql);
        st_to_con(qr);
        lam = r_max(lam, r_max(st_eigen(ql, d, g.gamma), st_eigen(qr, d, g.gamma)));
    });
    return lam;
}

// ... of every pencil
template <int d, int R, FluxBricks B>
__device__ __forceinline__ double max_eigen_staged(const Geom& g, const DevState& st, int b, double* P, int group) {
    const int npen = g.nx * g.nx;
    if constexpr (B != IN_GROUPS) return max_eigen_pencils<d, R>(g, st, b, P, 0, npen);
    double lam = 0.0;
    for (int p0 = 0; p0 < npen; p0 += group) {
        if (p0) __syncthreads();
        lam = r_max(lam, max_eigen_pencils<d, R>(g, st, b, P, p0, min(group, npen - p0)));
    }
    return lam;
}

}  // namespace amr
