// One hydro substep of every brick in one persistent launch: ghost zones,
// minmod-theta reconstruction, KT flux, coarse-fine flux correction, flux
// differences and the RK combination with floor, fused per brick.
//
// The reference runs this as level-ordered ghost fills
// (GridNode::enforce_boundaries, grid_node.cpp:59-112), Grid::compute_*_flux
// (grid.cpp:215-302) and the coarse-fine corrections (grid_node.cpp:1076-1274),
// then Grid::add_difs (grid.cpp:304-420).  Here each block takes bricks from
// a device work list, finest level first:
//  * ghost cells are not stored: a pencil's two ghost cells at each end are
//    computed where they are needed, from the neighbour's interior, the
//    parent's cells with the minmod slope (a parent ghost cell resolved the
//    same way), or the brick's own cells at a domain face -- the values the
//    level-ordered ghost fill would have written;
//  * a brick whose faces a coarser brick corrects publishes those face fluxes
//    and stamps itself done; the coarse brick waits (bounded) for the stamp
//    and replaces its own face flux by the mean of the four child faces;
//  * the updated state goes to a second state array, so no block reads a
//    brick another block is writing.
// The arithmetic of every value is that of the one-launch-per-step kernels,
// so with FT = double the result is bitwise that of amr_sub_step.
#pragma once

#include "flow_off.cuh"
#include "flux_kernel.cuh"
#include "hydro_cell.cuh"
#include "hydro_fused.h"

namespace amr {


__device__ __forceinline__ void fused_wait(const FusedArgs& A, int child) {
    unsigned long long spins = 0;
    while (*(volatile const int*)(A.done + child) != A.epoch) {
        if (++spins > A.wait_limit) {
            atomicOr(A.err, 1);
            break;
        }
        __nanosleep(64);
    }
    __threadfence();
}

// Block layout: per brick the "cross" -- the 8^3 interior and the six 2-deep
// ghost slabs the dimension-split stencil reads -- is held in shared memory as
// primitives (FT), and one direction's 576 face fluxes (FP64) at a time.  288
// threads take the faces in two full rounds; 256 left a third round with a
// quarter of them.  Faces are numbered so that neighbouring threads read and
// write neighbouring words in every direction (with the pencil fastest in x,
// two thirds of the shared-memory wavefronts were bank conflicts).  Two blocks
// an SM are 18 warps, five on a quarter of it: 96 registers, 160 bytes of
// spills in FP64.
constexpr int FUSED_BLOCK = 288;
constexpr int CROSS = 512 + 6 * 2 * 64;  // interior + ghost slabs
constexpr int FACES = 9 * 64;            // faces of one direction

// cross index of the cell at position n (0..11) along direction d of pencil
// (t1, t2): interior (z*8 + y)*8 + x, or slab ((face*2 + depth)*8 + t2)*8 + t1
__device__ __forceinline__ int cross_index(int d, int n, int t1, int t2) {
    if (n < 2) return 512 + (((2 * d) * 2 + n) * 8 + t2) * 8 + t1;
    if (n >= 10) return 512 + (((2 * d + 1) * 2 + (n - 10)) * 8 + t2) * 8 + t1;
    const int i = n - 2;
    const int x = d == 0 ? i : t1, y = d == 1 ? i : (d == 0 ? t1 : t2), z = d == 2 ? i : t2;
    return (z * 8 + y) * 8 + x;
}
// face number q of direction d <-> its position fi along d and its pencil
__device__ __forceinline__ void face_of(int d, int q, int& fi, int& t1, int& t2) {
    if (d == 0) {
        fi = q % 9, t1 = (q / 9) % 8, t2 = q / 72;
    } else if (d == 1) {
        t1 = q % 8, fi = (q / 8) % 9, t2 = q / 72;
    } else {
        t1 = q % 8, t2 = (q / 8) % 8, fi = q / 64;
    }
}
// the lower face of cell (x, y, z) along d, and the step to its upper face
__device__ __forceinline__ int cell_face(int d, int x, int y, int z) {
    return d == 0 ? (z * 8 + y) * 9 + x : (d == 1 ? z * 72 + y * 8 + x : (z * 8 + y) * 8 + x);
}
__device__ __forceinline__ int face_step(int d) { return d == 0 ? 1 : (d == 1 ? 8 : 64); }

template <typename FT>
__device__ __forceinline__ void fused_brick(const FusedArgs& A, int b, int vr, FT* P, double* Fs) {
    const Geom& g = A.g;
    const int nx = 8, gnx = 12, bw = 2, npen = 64, half = 4;
    const int tid = threadIdx.x;
    // (a) the cross as primitives: interior cells, then ghost cells resolved
    //     as the level-ordered ghost fill would have set them (one call: its
    //     code is long, and the block runs through all of this kernel's)
#pragma unroll 1
    for (int q = tid; q < CROSS; q += FUSED_BLOCK) {
        int x = q % 8 + bw, y = (q / 8) % 8 + bw, z = q / 64 + bw;
        if (q >= 512) {
            const int r = q - 512, t1 = x, t2 = (r / 8) % 8 + bw, depth = (r / 64) % 2, face = r / 128;
            const int ax = face >> 1;
            const int n = (face & 1) ? gnx - bw + depth : depth;
            x = ax == 0 ? n : t1;
            y = ax == 1 ? n : (ax == 0 ? t1 : t2);
            z = ax == 2 ? n : t2;
        }
        Cell6 u;
        ghost_cell<1, 2, 12>(A.g, A.bt, A.Uin, b, x, y, z, u, A.err);
        FT w[NF_EULER];
#pragma unroll
        for (int l = 0; l < NF_EULER; l++) w[l] = (FT)u.v[l];
        st_to_prim(w);
#pragma unroll
        for (int l = 0; l < NF_EULER; l++) P[l * CROSS + q] = w[l];
    }
    __syncthreads();
    const double hinv = 1.0 / A.bt.h[b];
    const FT th = (FT)g.theta, gam = (FT)g.gamma;
    const unsigned char pm = A.pubmask[b];
    double* pubb = A.pub + (size_t)b * 6 * NF_EULER * npen;
    const int* rg = vr >= 0 ? A.vranges + 4 * vr : nullptr;
    double D[2][NF_EULER];  // this thread's cells tid, tid + 288: flux differences, x then y then z
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
        for (int l = 0; l < NF_EULER; l++) D[h][l] = 0.0;
    // unrolled: the direction is a compile-time constant in each copy, so the
    // state arrays indexed by it (normal velocity, normal momentum flux) stay
    // in registers (one copy with the direction chosen by selects is smaller
    // but spills: 449 against 424 us for 2505 bricks)
#pragma unroll
    for (int d = 0; d < 3; d++) {
        // (b) face fluxes of direction d, one thread per face
#pragma unroll 1
        for (int q = tid; q < FACES; q += FUSED_BLOCK) {
            int fi, t1, t2;
            face_of(d, q, fi, t1, t2);
            const int p = t2 * nx + t1;
            FT w[4][NF_EULER];  // cells f-2 .. f+1 (f = fi + bw)
#pragma unroll
            for (int m = 0; m < 4; m++) {
                const int ci = cross_index(d, fi + m, t1, t2);
#pragma unroll
                for (int l = 0; l < NF_EULER; l++) w[m][l] = P[l * CROSS + ci];
            }
            FT ql[NF_EULER], qr[NF_EULER];
#pragma unroll
            for (int l = 0; l < NF_EULER; l++) {
                const FT sL = minmod_theta(w[2][l] - w[1][l], w[1][l] - w[0][l], th);  // slope of cell f-1
                const FT sR = minmod_theta(w[3][l] - w[2][l], w[2][l] - w[1][l], th);  // slope of cell f
                ql[l] = w[1][l] + sL / FT(2);
                qr[l] = w[2][l] - sR / FT(2);
            }
            st_to_con(ql);
            st_to_con(qr);
            FT fl[NF_EULER], fr[NF_EULER];
            const FT al = st_flux(ql, d, gam, fl);
            const FT ar = st_flux(qr, d, gam, fr);
            const FT a = r_max(al, ar);
            double F[NF_EULER];
#pragma unroll
            for (int l = 0; l < NF_EULER; l++) F[l] = (double)(((fl[l] + fr[l]) - (qr[l] - ql[l]) * a) * FT(0.5));
            // coarse-fine correction: mean of the child's four faces
            if (rg) {
                for (int it_q = rg[d]; it_q < rg[d + 1]; it_q++) {
                    const RefluxItem it = A.vitems[it_q];
                    const int aa = t1 - it.cj * half, cc = t2 - it.ck * half;
                    if (it.i0 - bw != fi || aa < 0 || aa >= half || cc < 0 || cc >= half) continue;
                    fused_wait(A, it.child);
                    const int side = it.ic == bw ? 0 : 1;
                    const double* Fc = A.pub + ((size_t)it.child * 6 + 2 * d + side) * NF_EULER * npen;
                    const int j = 2 * aa, k = 2 * cc;
#pragma unroll
                    for (int l = 0; l < NF_EULER; l++) {
                        const double* C = Fc + l * npen;
                        double v = +__ldcg(C + k * nx + j);
                        v += __ldcg(C + k * nx + j + 1);
                        v += __ldcg(C + (k + 1) * nx + j);
                        v += __ldcg(C + (k + 1) * nx + j + 1);
                        F[l] = v * 0.25;
                    }
                }
            }
            if (fi == 0 && (pm & (1u << (2 * d))))
#pragma unroll
                for (int l = 0; l < NF_EULER; l++) pubb[(2 * d * NF_EULER + l) * npen + p] = F[l];
            if (fi == nx && (pm & (1u << (2 * d + 1))))
#pragma unroll
                for (int l = 0; l < NF_EULER; l++) pubb[((2 * d + 1) * NF_EULER + l) * npen + p] = F[l];
            if (b == A.root) {
                double* Fr = (d == 0 ? A.Fx : (d == 1 ? A.Fy : A.Fz)) + (size_t)b * g.nf * npen * (nx + 1);
#pragma unroll
                for (int l = 0; l < NF_EULER; l++) Fr[l * npen * (nx + 1) + flux_index(d, nx, fi, t1, t2)] = F[l];
            }
#pragma unroll
            for (int l = 0; l < NF_EULER; l++) Fs[l * FACES + q] = F[l];
        }
        __syncthreads();
        // (c) this thread's cell: D -= (F(i+1) - F(i)) / h along d
        {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int cc = tid + h * FUSED_BLOCK;
                if (cc >= 512) break;
                const int lo = cell_face(d, cc % 8, (cc / 8) % 8, cc / 64), up = lo + face_step(d);
#pragma unroll
                for (int l = 0; l < NF_EULER; l++) D[h][l] -= (Fs[l * FACES + up] - Fs[l * FACES + lo]) * hinv;
            }
        }
        __syncthreads();
    }
    // faces published: stamp the brick done for the coarser bricks
    __threadfence();
    __syncthreads();
    if (tid == 0 && pm) atomicExch(A.done + b, A.epoch);
    // (d) Grid::add_difs (grid.cpp:406-420) for this thread's cells
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int cc = tid + h * FUSED_BLOCK;
        if (cc >= 512) break;
        const int x = cc % 8, y = (cc / 8) % 8, z = cc / 64;
        const int ci = cell_index(gnx, x + bw, y + bw, z + bw);
        const double* U = A.Uin + (size_t)b * g.ucount;
        const double* U0 = A.U0 + (size_t)b * g.ucount;
        double* Uo = A.Uout + (size_t)b * g.ucount;
        double u[NF_EULER];
#pragma unroll
        for (int l = 0; l < NF_EULER; l++) {
            const double Dl = D[h][l] + 0.0;  // State::source() is zero for the Euler state
            u[l] = (U[(size_t)l * g.gnx3 + ci] + Dl * A.dt) * A.beta + U0[(size_t)l * g.gnx3 + ci] * (1.0 - A.beta);
        }
        st_floor(u, g.gamma, g.rho_floor, g.ei_floor);
#pragma unroll
        for (int l = 0; l < NF_EULER; l++) Uo[(size_t)l * g.gnx3 + ci] = u[l];
    }
}

template <typename FT>
__global__ void __launch_bounds__(FUSED_BLOCK, 2) k_substep_fused(FusedArgs A) {
    extern __shared__ double smem[];  // [nf][CROSS] primitives (FT), then [nf][FACES] fluxes (FP64)
    FT* P = reinterpret_cast<FT*>(smem);
    double* Fs = smem + (NF_EULER * CROSS * sizeof(FT) + sizeof(double) - 1) / sizeof(double);
    __shared__ int s_item;
    for (;;) {
        if (threadIdx.x == 0) s_item = (int)atomicAdd(A.next, 1u);
        __syncthreads();
        const int w = s_item;
        if (w >= A.nwork) break;
        const int b = A.work[w].x;
        fused_brick<FT>(A, b, A.work[w].y, P, Fs);
        __syncthreads();
        // the root's fluxes are this block's own: their flow-off with them
        if (b == A.root) flow_off_block(A.g, DevState{.Fx = A.Fx, .Fy = A.Fy, .Fz = A.Fz}, b, A.bt.h[b], A.dt, A.beta, A.fo);
    }
}

template <typename FT>
constexpr size_t fused_smem_bytes() {
    return ((NF_EULER * CROSS * sizeof(FT) + sizeof(double) - 1) / sizeof(double)) * sizeof(double) +
           sizeof(double) * NF_EULER * FACES;
}

}  // namespace amr
