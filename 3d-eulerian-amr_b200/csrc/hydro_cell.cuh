// One cell of a brick as the level-ordered ghost fill leaves it, without
// reading a stored ghost: the interior value, or the face ghost's value
// computed from its source (GridNode::enforce_boundaries,
// grid_node.cpp:59-112; GridAMRBound, grid_amr_bound.cpp:27-78; GridPhysBound,
// grid_phys_bound.cpp:60-169).  Shared by the one-launch ghost fill and the
// fused substep; the arithmetic of every value is that of the level-ordered
// fill, so the results are the same bits.
#pragma once

#include "euler_state.cuh"
#include "flux_kernel.cuh"

namespace amr {

// Six conserved fields of one cell, indexed only by compile-time constants
// (stays in registers).
struct Cell6 {
    double v[NF_EULER];
};

// State::enforce_outflow (euler/state.cpp:45-84) on a register cell, the
// same arithmetic as st_enforce_outflow without a run-time array index.
__device__ __forceinline__ void cell_outflow(Cell6& u, int bface) {
    const int m = 1 + (bface >> 1);
    const double um = m == 1 ? u.v[1] : (m == 2 ? u.v[2] : u.v[3]);
    bool zero;
    if (bface == ZU || bface == ZL) {
        zero = (bface == ZU) ? (u.v[3] > 0.0) : (u.v[3] < 0.0);
    } else {
        const double v = um / u.v[0];
        zero = (bface & 1) ? (v > 0.0) : (v < 0.0);
    }
    if (zero) {
        u.v[4] = u.v[4] - 0.5 * um * um / u.v[0];
        if (m == 1) u.v[1] = 0.0;
        else if (m == 2) u.v[2] = 0.0;
        else u.v[3] = 0.0;
    }
}

__device__ __forceinline__ int axis_of(int x, int y, int z, int a) { return a == 0 ? x : (a == 1 ? y : z); }

__device__ __forceinline__ void cell_load(const double* U, int ucount, int gnx, int gnx3, int b, int x, int y, int z,
                                          Cell6& u) {
    const double* V = U + (size_t)b * ucount + cell_index(gnx, x, y, z);
#pragma unroll
    for (int l = 0; l < NF_EULER; l++) u.v[l] = V[(size_t)l * gnx3];
}

// Cell (x, y, z) (GNX frame, at most one coordinate outside the interior) of
// brick b.  DEPTH bounds the coarse-fine hops: a coarse-fine ghost reads the
// parent's cells, whose ghosts across the same face are same-level or domain
// ghosts under proper nesting, so DEPTH = 1 suffices unless the stencil is
// wider than an octant (4^3 bricks with bw >= 3) and reads the parent's ghosts
// on its other side.  A deeper chain sets *err bit 1 (and gives 0) where err
// is given; callers that give none must know that the tree has none
// (amr_ctx::ghost_chain).  BW, GNX: the brick's sizes where they are known at
// compile time, else 0.
template <int DEPTH, int BW, int GNX>
__device__ __forceinline__ void ghost_cell(const Geom& g, const BrickTable& bt, const double* U, int b, int x, int y,
                                           int z, Cell6& u, int* err) {
    const int bw = BW ? BW : g.bw, gnx = GNX ? GNX : g.gnx;
    const int ax = (x < bw || x >= gnx - bw) ? 0 : ((y < bw || y >= gnx - bw) ? 1 : ((z < bw || z >= gnx - bw) ? 2 : -1));
    if (ax < 0) {
        cell_load(U, g.ucount, gnx, g.gnx3, b, x, y, z, u);
        return;
    }
    const int gi = axis_of(x, y, z, ax);
    const int upper = gi >= gnx - bw ? 1 : 0;
    const int face = 2 * ax + upper;
    const int kind = bt.ftype[6 * b + face];
    const int nbr = bt.fnbr[6 * b + face];
    int sx = x, sy = y, sz = z, src = b;
    int s;
    if (kind == FACE_SIB) {
        s = upper ? gi - (gnx - 2 * bw) : gi + (gnx - 2 * bw);
        src = nbr;
    } else if (kind == FACE_OUTFLOW) {
        s = upper ? gnx - bw - 1 : bw;
    } else if (kind == FACE_REFLECT) {
        s = 2 * bw - 1 - gi;
    } else {
        s = -1;
    }
    if (s >= 0) {
        if (ax == 0) sx = s;
        else if (ax == 1) sy = s;
        else sz = s;
        cell_load(U, g.ucount, gnx, g.gnx3, src, sx, sy, sz, u);
        if (kind == FACE_OUTFLOW) cell_outflow(u, face ^ 1);
        if (kind == FACE_REFLECT) u.v[3] = -u.v[3];
        return;
    }
    if constexpr (DEPTH == 0) {
        if (err) atomicOr(err, 2);
#pragma unroll
        for (int l = 0; l < NF_EULER; l++) u.v[l] = 0.0;
    } else {
        // GridAMRBound::operator() (grid_amr_bound.cpp:27-78): the parent
        // cell minus a quarter of the face-normal minmod slope, sign by the
        // fine cell's parity
        const int fx = bt.off[3 * b + 0] - 2 * bt.off[3 * nbr + 0] + x;
        const int fy = bt.off[3 * b + 1] - 2 * bt.off[3 * nbr + 1] + y;
        const int fz = bt.off[3 * b + 2] - 2 * bt.off[3 * nbr + 2] + z;
        const int px = fx / 2, py = fy / 2, pz = fz / 2;
        const int par = axis_of(fx, fy, fz, ax) % 2;
        const int dx = ax == 0, dy = ax == 1, dz = ax == 2;
        Cell6 uc, up, um;
        const int pa = axis_of(px, py, pz, ax);
        if (pa - 1 >= bw && pa + 1 < gnx - bw) {  // all three inside the parent: their loads together
            cell_load(U, g.ucount, gnx, g.gnx3, nbr, px, py, pz, uc);
            cell_load(U, g.ucount, gnx, g.gnx3, nbr, px + dx, py + dy, pz + dz, up);
            cell_load(U, g.ucount, gnx, g.gnx3, nbr, px - dx, py - dy, pz - dz, um);
        } else {
            ghost_cell<DEPTH - 1, BW, GNX>(g, bt, U, nbr, px, py, pz, uc, err);
            ghost_cell<DEPTH - 1, BW, GNX>(g, bt, U, nbr, px + dx, py + dy, pz + dz, up, err);
            ghost_cell<DEPTH - 1, BW, GNX>(g, bt, U, nbr, px - dx, py - dy, pz - dz, um, err);
        }
#pragma unroll
        for (int l = 0; l < NF_EULER; l++) {
            double m = minmod2(up.v[l] - uc.v[l], uc.v[l] - um.v[l]);
            if (par == 1) m = -m;
            u.v[l] = uc.v[l] - m * 0.25;
        }
    }
}

}  // namespace amr
