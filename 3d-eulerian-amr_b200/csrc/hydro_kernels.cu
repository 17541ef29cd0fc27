// Hydro kernels, plain FP64 form.  One CUDA block per brick (or per brick
// face / correction item); bricks of any level run in one launch wherever
// the reference's recursion order does not create a dependency.
//
// Layouts (see amr_internal.h):
//   U  [slot][f][k][j][i], GNX^3 per field, ghosts included
//   Fx [slot][f][k'][j'][i'] faces i'=0..nx (grid face bw+i'), j',k' interior
//   Fy [slot][f][k'][j'][i'] faces j'=0..nx
//   Fz [slot][f][k'][j'][i'] faces k'=0..nx
#include "euler_state.cuh"
#include "flux_kernel.cuh"
#include "flow_off.cuh"
#include "hydro_cell.cuh"
#include "kernels.h"
#include "launch.cuh"

#include <algorithm>

namespace amr {

// ---------------------------------------------------------------------------
// ghost zones: GridNode::enforce_boundaries (grid_node.cpp:59-112) with the
// three kinds of face source (same level, GridAMRBound, GridPhysBound).
// grid = (bricks of one level, 6 faces); thread per ghost cell of the face
// slab (bw x nx x nx, transverse interior only; edges/corners untouched).
// ---------------------------------------------------------------------------
__global__ void k_ghost_fill(Geom g, BrickTable bt, DevState st, const int* __restrict__ slots) {
    const int b = slots[blockIdx.x];
    const int face = blockIdx.y;
    const int ax = face >> 1, upper = face & 1;
    const int bw = g.bw, gnx = g.gnx, nx = g.nx;
    const int kind = bt.ftype[6 * b + face];
    const int nbr = bt.fnbr[6 * b + face];
    double* U = st.U + (size_t)b * g.ucount;
    for (int t = threadIdx.x; t < bw * nx * nx; t += blockDim.x) {
        const int n = t % bw;             // depth into the ghost layer
        const int t1 = (t / bw) % nx + bw;  // lower transverse axis
        const int t2 = (t / bw) / nx + bw;  // higher transverse axis
        const int gi = upper ? gnx - bw + n : n;  // ghost index along ax
        int c[3];
        c[ax] = gi;
        c[ax == 0 ? 1 : 0] = t1;
        c[ax == 2 ? 1 : 2] = t2;
        const int dst = cell_index(gnx, c[0], c[1], c[2]);
        double u[NF_EULER];
        if (kind == FACE_SIB) {
            // (*sib)(GNX-2bw+i, j, k) for the lower face, (i-GNX+2bw) upper.
            int s[3] = {c[0], c[1], c[2]};
            s[ax] = upper ? gi - (gnx - 2 * bw) : gi + (gnx - 2 * bw);
            const double* V = st.U + (size_t)nbr * g.ucount;
            const int src = cell_index(gnx, s[0], s[1], s[2]);
#pragma unroll
            for (int l = 0; l < NF_EULER; l++) u[l] = V[l * g.gnx3 + src];
        } else if (kind == FACE_OUTFLOW) {
            // GridPhysBound map (grid_phys_bound.cpp:60-169): copy the first
            // interior cell, then enforce_outflow with the proxy's face.
            int s[3] = {c[0], c[1], c[2]};
            s[ax] = upper ? gnx - bw - 1 : bw;
            const int src = cell_index(gnx, s[0], s[1], s[2]);
#pragma unroll
            for (int l = 0; l < NF_EULER; l++) u[l] = U[l * g.gnx3 + src];
            st_enforce_outflow(u, face ^ 1);
        } else if (kind == FACE_REFLECT) {
            // Z_REFLECT at z=0: ghost k <- cell 2*bw-1-k, sz -> -sz
            // (grid_phys_bound.cpp:140-155, State::reflect_on_z).
            int s[3] = {c[0], c[1], c[2]};
            s[ax] = 2 * bw - 1 - gi;
            const int src = cell_index(gnx, s[0], s[1], s[2]);
#pragma unroll
            for (int l = 0; l < NF_EULER; l++) u[l] = U[l * g.gnx3 + src];
            u[3] = -u[3];
        } else {
            // GridAMRBound::operator() (grid_amr_bound.cpp:27-78): parent cell
            // at half the fine index, minus a quarter of the face-normal
            // minmod slope, sign by the fine cell's parity.
            const double* P = st.U + (size_t)nbr * g.ucount;
            int pi[3], par = 0;
            for (int d = 0; d < 3; d++) {
                const int fine = bt.off[3 * b + d] - 2 * bt.off[3 * nbr + d] + c[d];
                pi[d] = fine / 2;
                if (d == ax) par = fine % 2;
            }
            int pp[3] = {pi[0], pi[1], pi[2]}, pm[3] = {pi[0], pi[1], pi[2]};
            pp[ax] += 1;
            pm[ax] -= 1;
            const int i0 = cell_index(gnx, pi[0], pi[1], pi[2]);
            const int ip = cell_index(gnx, pp[0], pp[1], pp[2]);
            const int im = cell_index(gnx, pm[0], pm[1], pm[2]);
#pragma unroll
            for (int l = 0; l < NF_EULER; l++) {
                const double uc = P[l * g.gnx3 + i0];
                double m = minmod2(P[l * g.gnx3 + ip] - uc, uc - P[l * g.gnx3 + im]);
                if (par == 1) m = -m;
                u[l] = uc - m * 0.25;
            }
        }
#pragma unroll
        for (int l = 0; l < NF_EULER; l++) U[l * g.gnx3 + dst] = u[l];
    }
}

// The same for every level in one launch: every ghost value is computed from
// interior cells (ghost_cell), so no level waits for another.  Needs a tree
// whose coarse-fine ghosts read no coarse-fine ghosts (the host looks at
// every such stencil, amr_ctx::ghost_chain, and runs the level-ordered fill
// otherwise: proper nesting alone is not enough for 4^3 bricks).  A launch of a
// small level is 5 us of latency; one per level was 18 to 21% of a step.
// grid = (bricks, 6 faces); neighbouring threads on neighbouring cells; the
// brick's sizes at compile time (0: at run time) for the index divisions.
template <int BW, int NX>
__global__ void __launch_bounds__(128) k_ghost_fill_all(Geom g, BrickTable bt, DevState st,
                                                        const int* __restrict__ slots) {
    const int b = slots[blockIdx.x];
    const int face = blockIdx.y;
    const int ax = face >> 1, upper = face & 1;
    const int bw = BW ? BW : g.bw, nx = NX ? NX : g.nx, gnx = nx + 2 * bw, gnx3 = gnx * gnx * gnx;
    const int kind = bt.ftype[6 * b + face];
    const int step = ax == 0 ? 1 : (ax == 1 ? gnx : gnx * gnx);
    for (int t = threadIdx.x; t < bw * nx * nx; t += blockDim.x) {
        const int n = ax == 0 ? t % bw : (t / nx) % bw;
        const int t1 = (ax == 0 ? (t / bw) % nx : t % nx) + bw;
        const int t2 = t / (bw * nx) + bw;
        const int gi = upper ? gnx - bw + n : n;
        const int x = ax == 0 ? gi : t1, y = ax == 1 ? gi : (ax == 0 ? t1 : t2), z = ax == 2 ? gi : t2;
        const int to = cell_index(gnx, x, y, z);
        Cell6 u;
        if (kind == FACE_SIB) {
            const double* V = st.U + (size_t)bt.fnbr[6 * b + face] * g.ucount + to + (upper ? -nx : nx) * step;
#pragma unroll
            for (int l = 0; l < NF_EULER; l++) u.v[l] = V[l * gnx3];
        } else {
            ghost_cell<1, BW, NX ? NX + 2 * BW : 0>(g, bt, st.U, b, x, y, z, u, nullptr);
        }
        double* U = st.U + (size_t)b * g.ucount + to;
#pragma unroll
        for (int l = 0; l < NF_EULER; l++) U[l * gnx3] = u.v[l];
    }
}

// ---------------------------------------------------------------------------
// KT/Rusanov fluxes, Grid::compute_{x,y,z}_flux (grid.cpp:215-302) with
// minmod-theta (reconstruct.cpp:60-71) or PPM (reconstruct.cpp:22-58)
// reconstruction (flux_kernel.cuh).  grid = (bricks, 3 directions)
// ---------------------------------------------------------------------------
template <int R, FluxBricks B>
__global__ void __launch_bounds__(FluxBlock<B>::THREADS, FluxBlock<B>::PER_SM)
    k_flux(Geom g, DevState st, const int* __restrict__ slots, int group) {
    extern __shared__ double flux_smem[];
    flux_staged<double, R, B>(g, st, slots[blockIdx.x], flux_smem, group);
}

// ---------------------------------------------------------------------------
// Coarse-fine flux correction, GridNode::adjust_{x,y,z}_flux
// (grid_node.cpp:1076-1274): the coarse face quadrant takes the mean of the
// child's four faces.  A child's face can itself be corrected (at a domain
// face, where no neighbour decides: elsewhere proper nesting leaves none), so
// the finest coarse level comes first.  One launch for all levels: a block
// starts at an item whose child's face is not corrected and, if it is the
// last of the items that correct the coarse brick's face, goes on to the item
// that reads that face (a counter per brick face, back to zero for the next
// launch); no block waits.  fixes[6 slot + face] = items that correct the
// face.  One block per starting item, thread per (field, face cell).  The
// climb knows one reader of a corrected face, the parent's item.  In a loaded
// tree that is not properly nested the parent's neighbour can read it too:
// there (host: reflux_by_level) fixes is null, a block does its item only,
// and the launches are one per coarse level, finest first.
// ---------------------------------------------------------------------------
__global__ void k_reflux(Geom g, BrickTable bt, DevState st, const RefluxItem* __restrict__ items,
                         const unsigned char* __restrict__ fixes, unsigned* done) {
    __shared__ int s_go;
    RefluxItem it = items[blockIdx.x];
    const int nx = g.nx, bw = g.bw, gnx = g.gnx;
    const int half = nx / 2, fstride = nx * nx * (nx + 1);
    const int t = threadIdx.x;
    const int l = t / (half * half);
    const int q = t % (half * half);
    const int a = q % half, c = q / half;      // by2 indexer: j = bw+2a, k = bw+2c
    const int j = 2 * a, k = 2 * c;            // child interior offsets
    for (;;) {
        if (t < g.nf * half * half) {
            const int j0 = a + it.cj * half, k0 = c + it.ck * half;  // coarse interior offsets
            double* F = (it.dir == 0 ? st.Fx : (it.dir == 1 ? st.Fy : st.Fz));
            const double* Fc = F + ((size_t)it.child * g.nf + l) * fstride;
            double* Fp = F + ((size_t)it.coarse * g.nf + l) * fstride;
            const int ic = it.ic - bw;
            // L2 loads: another block of this launch may have corrected them,
            // and a line of them can be in this SM's first cache already
            double v = +__ldcg(Fc + flux_index(it.dir, nx, ic, j, k));
            v += __ldcg(Fc + flux_index(it.dir, nx, ic, j + 1, k));
            v += __ldcg(Fc + flux_index(it.dir, nx, ic, j, k + 1));
            v += __ldcg(Fc + flux_index(it.dir, nx, ic, j + 1, k + 1));
            v *= 0.25;
            Fp[flux_index(it.dir, nx, it.i0 - bw, j0, k0)] = v;
        }
        // the face just corrected, if it is an outer one, and who reads it
        if (!fixes) return;
        if (it.i0 != bw && it.i0 != gnx - bw) return;
        const int p = it.coarse, side = it.i0 == bw ? 0 : 1, face = 2 * it.dir + side;
        if (bt.parent[p] < 0 || bt.ftype[6 * p + face] == FACE_SIB) return;
        __threadfence();
        __syncthreads();
        if (t == 0) {
            const bool last = atomicAdd(done + 6 * p + face, 1u) == (unsigned)fixes[6 * p + face] - 1u;
            if (last) done[6 * p + face] = 0u;
            s_go = last;
        }
        __syncthreads();
        if (!s_go) return;
        __threadfence();
        const int ta = it.dir == 0 ? 1 : 0, tb = it.dir == 2 ? 1 : 2, ci = bt.cidx[p];
        const bool outer = ((ci >> it.dir) & 1) == side;
        it.child = p;
        it.coarse = bt.parent[p];
        it.ic = side ? gnx - bw : bw;
        it.i0 = outer ? it.ic : gnx / 2;
        it.cj = (ci >> ta) & 1;
        it.ck = (ci >> tb) & 1;
    }
}

// ---------------------------------------------------------------------------
// Flux differences + RK combine + floor: clear_difs, sum_{x,y,z}_difs and
// Grid::add_difs (grid.cpp:201-213, 304-344, 406-420).  With gravity the
// ZSTAR energy work term and the momentum sources of the restated coupling
// (single/single.cpp:49-97, 304-383) are added in the reference order.
// grid = (bricks, cells / 256) + the root's flow-off in the last block of
// the first row; thread per interior cell.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_add_difs(Geom g, DevState st, const int* __restrict__ slots,
                                                  const double* __restrict__ hs, double dt_arg,
                                                  const double* __restrict__ dtp, double beta, int gravity, int root,
                                                  double* fo) {
    const double dt = dtp ? *dtp : dt_arg;  // device-computed step in captured graphs
    if (blockIdx.x == gridDim.x - 1) {
        if (blockIdx.y == 0) flow_off_block(g, st, root, hs[root], dt, beta, fo);
        return;
    }
    const int b = slots[blockIdx.x];
    const int nx = g.nx, gnx = g.gnx, bw = g.bw, pnx = g.pnx;
    const int npen = nx * nx, fstride = npen * (nx + 1);
    const double h = hs[b];
    const double hinv = 1.0 / h;
    const int t = blockIdx.y * blockDim.x + threadIdx.x;
    if (t < nx * nx * nx) {
        const int i = t % nx, j = (t / nx) % nx, k = t / npen;
        double D[NF_EULER];
#pragma unroll
        for (int l = 0; l < NF_EULER; l++) D[l] = 0.0;
        const double* Fx = st.Fx + (size_t)b * g.nf * fstride;
        const double* Fy = st.Fy + (size_t)b * g.nf * fstride;
        const double* Fz = st.Fz + (size_t)b * g.nf * fstride;
        // Poisson frame: pi = i + 1 (grid index i+bw == pi + BW - 1)
        const size_t pb = (size_t)b * g.pnx3;
        const int pc = ((k + 1) * pnx + (j + 1)) * pnx + (i + 1);
        const int a0 = flux_index(0, nx, i, j, k), a1 = flux_index(0, nx, i + 1, j, k);
#pragma unroll
        for (int l = 0; l < NF_EULER; l++) D[l] -= (Fx[l * fstride + a1] - Fx[l * fstride + a0]) * hinv;
        if (gravity) {
            D[4] += 0.5 * st.fx[pb + pc] * (Fx[a0]);
            D[4] += 0.5 * st.fx[pb + pc + 1] * (Fx[a1]);
        }
        const int b0 = flux_index(1, nx, j, i, k), b1 = flux_index(1, nx, j + 1, i, k);
#pragma unroll
        for (int l = 0; l < NF_EULER; l++) D[l] -= (Fy[l * fstride + b1] - Fy[l * fstride + b0]) * hinv;
        if (gravity) {
            D[4] += 0.5 * st.fy[pb + pc] * (Fy[b0]);
            D[4] += 0.5 * st.fy[pb + pc + pnx] * (Fy[b1]);
        }
        const int c0 = flux_index(2, nx, k, i, j), c1 = flux_index(2, nx, k + 1, i, j);
#pragma unroll
        for (int l = 0; l < NF_EULER; l++) D[l] -= (Fz[l * fstride + c1] - Fz[l * fstride + c0]) * hinv;
        if (gravity) {
            D[4] += 0.5 * st.fz[pb + pc] * (Fz[c0]);
            D[4] += 0.5 * st.fz[pb + pc + pnx * pnx] * (Fz[c1]);
        }
        const int ci = cell_index(gnx, i + bw, j + bw, k + bw);
        double* U = st.U + (size_t)b * g.ucount;
        const double* U0 = st.U0 + (size_t)b * g.ucount;
        double u[NF_EULER];
#pragma unroll
        for (int l = 0; l < NF_EULER; l++) u[l] = U[l * g.gnx3 + ci];
        if (gravity) {
            const double fx0 = 0.5 * u[0] * (st.fx[pb + pc] + st.fx[pb + pc + 1]);
            const double fy0 = 0.5 * u[0] * (st.fy[pb + pc] + st.fy[pb + pc + pnx]);
            const double fz0 = 0.5 * u[0] * (st.fz[pb + pc] + st.fz[pb + pc + pnx * pnx]);
            D[3] += fz0;
            D[1] += fx0;
            D[2] += fy0;
        }
#pragma unroll
        for (int l = 0; l < NF_EULER; l++) {
            D[l] += 0.0;  // State::source() is zero for the Euler state
            u[l] = (u[l] + D[l] * dt) * beta + U0[l * g.gnx3 + ci] * (1.0 - beta);
        }
        st_floor(u, g.gamma, g.rho_floor, g.ei_floor);
#pragma unroll
        for (int l = 0; l < NF_EULER; l++) U[l * g.gnx3 + ci] = u[l];
    }
}

// ---------------------------------------------------------------------------
// Restriction, GridNode::inject_from_children (grid_node.cpp:1035-1074):
// covered parent cell := mean of its 8 child cells, then floor.
// One launch for the whole tree: a block starts at a brick whose children
// have no children, restricts into it, and goes on to its parent if it is the
// last of that brick's refined children to be done (a counter per brick, back
// to zero for the next launch), so children come first as in the recursion
// and no block waits.  A launch per level was 9 us of latency each.
// grid = bricks whose children are all leaves; thread per parent cell.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(512) k_inject(Geom g, BrickTable bt, DevState st, const int* __restrict__ starts,
                                                const int* __restrict__ refined, unsigned* done) {
    __shared__ int s_next;
    const int nx = g.nx, gnx = g.gnx, bw = g.bw, half = nx / 2, h3 = half * half * half;
    int p = starts[blockIdx.x];
    for (;;) {
        double* P = st.U + (size_t)p * g.ucount;
        for (int q = threadIdx.x; q < 8 * h3; q += blockDim.x) {
            const int c = q / h3, t = q % h3;
            const int ch = bt.child[8 * p + c];
            if (ch < 0) continue;
            const int a = t % half, bb = (t / half) % half, cc = t / (half * half);
            const int i = bw + 2 * a, j = bw + 2 * bb, k = bw + 2 * cc;
            const int i0 = bw + a + (c & 1) * half, j0 = bw + bb + ((c >> 1) & 1) * half,
                      k0 = bw + cc + ((c >> 2) & 1) * half;
            const double* C = st.U + (size_t)ch * g.ucount + cell_index(gnx, i, j, k);
            double u[NF_EULER];
#pragma unroll
            for (int l = 0; l < NF_EULER; l++) {
                const double* Cl = C + l * g.gnx3;
                // plain loads, although another block of this launch may have
                // written the child: nothing reads these cells before this
                // block does, so no line of them is in its SM's first cache
                double s = 0.0;
                s += Cl[0];
                s += Cl[1];
                s += Cl[gnx];
                s += Cl[gnx + 1];
                s += Cl[gnx * gnx];
                s += Cl[gnx * gnx + 1];
                s += Cl[gnx * gnx + gnx];
                s += Cl[gnx * gnx + gnx + 1];
                u[l] = s * 0.125;
            }
            st_floor(u, g.gamma, g.rho_floor, g.ei_floor);
            const int dst = cell_index(gnx, i0, j0, k0);
#pragma unroll
            for (int l = 0; l < NF_EULER; l++) P[l * g.gnx3 + dst] = u[l];
        }
        const int up = bt.parent[p];
        if (up < 0) return;
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) {
            const bool last = atomicAdd(done + up, 1u) == (unsigned)refined[up] - 1u;
            if (last) done[up] = 0u;
            s_next = last ? up : -1;
        }
        __syncthreads();
        p = s_next;
        if (p < 0) return;
        __threadfence();
    }
}

// ---------------------------------------------------------------------------
// Prolongation of new bricks, GridNode::inject_from_parent
// (grid_node.cpp:193-233): parent cell +- a quarter of the three minmod
// slopes, then floor.  Thread per parent cell of the child's octant.
// ---------------------------------------------------------------------------
__global__ void k_prolong(Geom g, BrickTable bt, DevState st, const int* __restrict__ slots) {
    const int b = slots[blockIdx.x];
    const int p = bt.parent[b];
    const int c = bt.cidx[b];
    const int nx = g.nx, gnx = g.gnx, bw = g.bw, half = nx / 2;
    const int t = threadIdx.x;
    if (t >= half * half * half) return;
    const int a = t % half, bb = (t / half) % half, cc = t / (half * half);
    const int i = bw + 2 * a, j = bw + 2 * bb, k = bw + 2 * cc;
    const int i0 = bw + a + (c & 1) * half, j0 = bw + bb + ((c >> 1) & 1) * half, k0 = bw + cc + ((c >> 2) & 1) * half;
    const double* P = st.U + (size_t)p * g.ucount;
    double* C = st.U + (size_t)b * g.ucount;
    double out[8][NF_EULER];
#pragma unroll
    for (int l = 0; l < NF_EULER; l++) {
        const double* Pl = P + l * g.gnx3;
        const double u = Pl[cell_index(gnx, i0, j0, k0)];
        const double s1 = minmod2(Pl[cell_index(gnx, i0 + 1, j0, k0)] - u, u - Pl[cell_index(gnx, i0 - 1, j0, k0)]);
        const double s2 = minmod2(Pl[cell_index(gnx, i0, j0 + 1, k0)] - u, u - Pl[cell_index(gnx, i0, j0 - 1, k0)]);
        const double s3 = minmod2(Pl[cell_index(gnx, i0, j0, k0 + 1)] - u, u - Pl[cell_index(gnx, i0, j0, k0 - 1)]);
        out[0][l] = u - (s1 + s2 + s3) * 0.25;
        out[1][l] = u + (s1 - s2 - s3) * 0.25;
        out[2][l] = u - (s1 - s2 + s3) * 0.25;
        out[3][l] = u + (s1 + s2 - s3) * 0.25;
        out[4][l] = u - (s1 + s2 - s3) * 0.25;
        out[5][l] = u + (s1 - s2 + s3) * 0.25;
        out[6][l] = u - (s1 - s2 - s3) * 0.25;
        out[7][l] = u + (s1 + s2 + s3) * 0.25;
    }
#pragma unroll
    for (int o = 0; o < 8; o++) {
        st_floor(out[o], g.gamma, g.rho_floor, g.ei_floor);
        const int dst = cell_index(gnx, i + (o & 1), j + ((o >> 1) & 1), k + ((o >> 2) & 1));
#pragma unroll
        for (int l = 0; l < NF_EULER; l++) C[l * g.gnx3 + dst] = out[o][l];
    }
}

// ---------------------------------------------------------------------------
// CFL time step, Grid::max_dt (grid.cpp:422-483): largest face eigenvalue of
// the reconstructed states of each direction, lam[3 b + d].  (The brick's
// step, cfl / (max lam / h), is formed where the tree's is: cfl_step.)
// ---------------------------------------------------------------------------
__device__ __forceinline__ void store_block_max(double lam, double* out) {
    __shared__ double red[32];
    // block max (max is exact, order-free)
    for (int o = 16; o > 0; o >>= 1) lam = r_max(lam, __shfl_xor_sync(0xffffffffu, lam, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = lam;
    __syncthreads();
    if (threadIdx.x == 0) {
        double m = 0.0;
        for (int w = 0; w < (int)((blockDim.x + 31) >> 5); w++) m = r_max(m, red[w]);
        *out = m;
    }
}
// grid = (bricks, 3 directions): staged pencils (flux_kernel.cuh), threads
// rounded up to whole warps
template <int R, FluxBricks B>
__global__ void __launch_bounds__(FluxBlock<B>::THREADS, FluxBlock<B>::PER_SM)
    k_max_dt(Geom g, DevState st, const int* __restrict__ slots, double* __restrict__ lam_out, int group) {
    extern __shared__ double flux_smem[];
    const int b = slots[blockIdx.x], d = blockIdx.y;
    double lam;
    if (d == 0)
        lam = max_eigen_staged<0, R, B>(g, st, b, flux_smem, group);
    else if (d == 1)
        lam = max_eigen_staged<1, R, B>(g, st, b, flux_smem, group);
    else
        lam = max_eigen_staged<2, R, B>(g, st, b, flux_smem, group);
    store_block_max(lam, lam_out + 3 * b + d);
}

// ---------------------------------------------------------------------------
// Density test of GridNode::set_refine_flags (grid_node.cpp:649-671):
// flag octant c when an interior cell of it has rho > threshold.
// ---------------------------------------------------------------------------
__global__ void k_refine_flags(Geom g, DevState st, const int* __restrict__ slots, double thr,
                               unsigned char* __restrict__ flags) {
    const int b = slots[blockIdx.x];
    __shared__ int f8[8];
    if (threadIdx.x < 8) f8[threadIdx.x] = 0;
    __syncthreads();
    const int nx = g.nx, gnx = g.gnx, bw = g.bw;
    const double* R = st.U + (size_t)b * g.ucount;
    for (int t = threadIdx.x; t < nx * nx * nx; t += blockDim.x) {
        const int i = t % nx + bw, j = (t / nx) % nx + bw, k = t / (nx * nx) + bw;
        if (R[cell_index(gnx, i, j, k)] > thr) {
            const int c = (2 * i / gnx) | ((2 * j / gnx) << 1) | ((2 * k / gnx) << 2);
            f8[c] = 1;
        }
    }
    __syncthreads();
    if (threadIdx.x < 8) flags[8 * blockIdx.x + threadIdx.x] = (unsigned char)f8[threadIdx.x];
}

// Per-brick max of one field over uncovered interior cells
// (GridNode::state_max, grid_node.cpp:1529-1558).
__global__ void k_state_max(Geom g, BrickTable bt, DevState st, const int* __restrict__ slots, int field,
                            double* __restrict__ out) {
    const int b = slots[blockIdx.x];
    const int nx = g.nx, gnx = g.gnx, bw = g.bw;
    const double* R = st.U + (size_t)b * g.ucount + field * g.gnx3;
    __shared__ double red[32];
    double m = -1.0E+99;
    for (int t = threadIdx.x; t < nx * nx * nx; t += blockDim.x) {
        const int i = t % nx + bw, j = (t / nx) % nx + bw, k = t / (nx * nx) + bw;
        const int c = (2 * i / gnx) | ((2 * j / gnx) << 1) | ((2 * k / gnx) << 2);
        if (bt.child[8 * b + c] < 0) m = r_max(R[cell_index(gnx, i, j, k)], m);
    }
    for (int o = 16; o > 0; o >>= 1) m = r_max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        double r = -1.0E+99;
        for (int w = 0; w < (int)((blockDim.x + 31) >> 5); w++) r = r_max(red[w], r);
        out[blockIdx.x] = r;
    }
}

// ---------------------------------------------------------------------------
// launch wrappers
// ---------------------------------------------------------------------------
void launch_ghost_fill(const Geom& g, const BrickTable& bt, const DevState& st, const int* slots, int n,
                       cudaStream_t s) {
    if (n <= 0) return;
    launch_k(k_ghost_fill, dim3(n, 6), 128, 0, s, g, bt, st, slots);
}
void launch_ghost_fill_all(const Geom& g, const BrickTable& bt, const DevState& st, const int* slots, int n,
                           cudaStream_t s) {
    if (n <= 0) return;
    const auto k = g.nx == 8 && g.bw == 2 ? k_ghost_fill_all<2, 8>
                                          : (g.nx == 8 && g.bw == 3 ? k_ghost_fill_all<3, 8> : k_ghost_fill_all<0, 0>);
    launch_k(k, dim3(n, 6), 128, 0, s, g, bt, st, slots);
}
namespace {
template <int R, FluxBricks B>
void flux_fp64(const Geom& g, const DevState& st, const int* slots, int n, cudaStream_t s) {
    const int group = pencil_group<double, R>(g);
    const size_t smem = staged_smem<double, R>(g, group);
    if (smem > 48 * 1024)
        cudaFuncSetAttribute((const void*)k_flux<R, B>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    launch_k(k_flux<R, B>, dim3(n, 3), PENCIL_PARTS * group, smem, s, g, st, slots, group);
}
template <int R>
void flux_fp64(const Geom& g, const DevState& st, const int* slots, int n, cudaStream_t s) {
    (g.nx <= 8 ? flux_fp64<R, UP_TO_8> : g.nx == 12 ? flux_fp64<R, OF_12> : flux_fp64<R, IN_GROUPS>)(g, st, slots, n, s);
}
template <int R, FluxBricks B>
void max_dt_fp64(const Geom& g, const DevState& st, const int* slots, int n, double* lam, cudaStream_t s) {
    const int group = pencil_group<double, R>(g);
    const size_t smem = staged_smem<double, R>(g, group);
    if (smem > 48 * 1024)
        cudaFuncSetAttribute((const void*)k_max_dt<R, B>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const int threads = (PENCIL_PARTS * group + 31) / 32 * 32;
    launch_k(k_max_dt<R, B>, dim3(n, 3), threads, smem, s, g, st, slots, lam, group);
}
template <int R>
void max_dt_fp64(const Geom& g, const DevState& st, const int* slots, int n, double* lam, cudaStream_t s) {
    (g.nx <= 8    ? max_dt_fp64<R, UP_TO_8>
     : g.nx == 12 ? max_dt_fp64<R, OF_12>
                  : max_dt_fp64<R, IN_GROUPS>)(g, st, slots, n, lam, s);
}
}  // namespace
void launch_flux(const Geom& g, const DevState& st, const int* slots, int n, cudaStream_t s) {
    if (n <= 0) return;
    if (g.flux32)
        launch_flux_f32(g, st, slots, n, s);
    else if (g.recon == RECON_PPM)
        flux_fp64<RECON_PPM>(g, st, slots, n, s);
    else
        flux_fp64<RECON_MINMOD>(g, st, slots, n, s);
}
void launch_reflux(const Geom& g, const BrickTable& bt, const DevState& st, const RefluxItem* items, int n,
                   const unsigned char* fixes, unsigned* done, cudaStream_t s) {
    if (n <= 0) return;
    const int half = g.nx / 2;
    launch_k(k_reflux, n, ((g.nf * half * half + 31) / 32) * 32, 0, s, g, bt, st, items, fixes, done);
}
void launch_add_difs(const Geom& g, const DevState& st, const int* slots, int n, const double* hs, double dt,
                     double beta, int gravity, int root, double* fo, cudaStream_t s, const double* dtp) {
    if (n <= 0) return;
    launch_k(k_add_difs, dim3(n + 1, (g.nx * g.nx * g.nx + 255) / 256), 256, 0, s, g, st, slots, hs, dt, dtp, beta,
             gravity, root, fo);
}
void launch_inject(const Geom& g, const BrickTable& bt, const DevState& st, const int* starts, int n,
                   const int* refined, unsigned* done, cudaStream_t s) {
    if (n <= 0) return;
    launch_k(k_inject, n, std::min(512, (g.nx * g.nx * g.nx + 31) / 32 * 32), 0, s, g, bt, st, starts, refined, done);
}
void launch_prolong(const Geom& g, const BrickTable& bt, const DevState& st, const int* slots, int n,
                    cudaStream_t s) {
    if (n <= 0) return;
    const int half = g.nx / 2;
    launch_k(k_prolong, n, ((half * half * half + 31) / 32) * 32, 0, s, g, bt, st, slots);
}
void launch_max_dt(const Geom& g, const DevState& st, const int* slots, int n, double* lam, cudaStream_t s) {
    if (n <= 0) return;
    if (g.recon == RECON_PPM)
        max_dt_fp64<RECON_PPM>(g, st, slots, n, lam, s);
    else
        max_dt_fp64<RECON_MINMOD>(g, st, slots, n, lam, s);
}
void launch_refine_flags(const Geom& g, const DevState& st, const int* slots, int n, double thr,
                         unsigned char* flags, cudaStream_t s) {
    if (n <= 0) return;
    launch_k(k_refine_flags, n, 256, 0, s, g, st, slots, thr, flags);
}
void launch_state_max(const Geom& g, const BrickTable& bt, const DevState& st, const int* slots, int n, int field,
                      double* out, cudaStream_t s) {
    if (n <= 0) return;
    launch_k(k_state_max, n, 256, 0, s, g, bt, st, slots, field, out);
}

}  // namespace amr

namespace amr {
// Host transfer helpers: pack the listed bricks into / out of a contiguous
// staging buffer (count doubles per brick).
__global__ void k_gather(const double* __restrict__ src, const int* __restrict__ slots, int count,
                         double* __restrict__ dst) {
    const int e = blockIdx.y;
    const double* s = src + (size_t)slots[e] * count;
    double* d = dst + (size_t)e * count;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < count; t += gridDim.x * blockDim.x) d[t] = s[t];
}
__global__ void k_scatter(const double* __restrict__ src, const int* __restrict__ slots, int count,
                          double* __restrict__ dst) {
    const int e = blockIdx.y;
    const double* s = src + (size_t)e * count;
    double* d = dst + (size_t)slots[e] * count;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < count; t += gridDim.x * blockDim.x) d[t] = s[t];
}
void launch_gather(const double* src, const int* slots, int n, int count, double* dst, cudaStream_t s) {
    if (n <= 0) return;
    launch_k(k_gather, dim3((count + 255) / 256, n), 256, 0, s, src, slots, count, dst);
}
void launch_scatter(const double* src, const int* slots, int n, int count, double* dst, cudaStream_t s) {
    if (n <= 0) return;
    launch_k(k_scatter, dim3((count + 255) / 256, n), 256, 0, s, src, slots, count, dst);
}
}  // namespace amr
