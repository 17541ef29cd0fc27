// Jacobi sweeps of Poisson::vcycle_relax (poisson.cpp:88-130) on one brick
// staged in shared memory.
//
// Each sweep computes tmp0 = dphi1 + lap(dphi)/6 for every cell from the
// previous sweep's values and adds it; the sweep's sum of tmp0^2 decides the
// loop (ratio to the first sweep's > 0.5, at most 16 sweeps).  The two shared
// buffers alternate so one barrier per sweep suffices; every thread forms
// the decision itself from the same numbers, so all threads take the same
// one.  (The reference adds the squares sequentially; the sums differ in the
// last bits only.)
//
// What bounds a sweep is shared-memory loads and the latency of the sum, not
// arithmetic or memory:
//  * a thread owns K cells one above the other in z and keeps them in
//    registers from sweep to sweep, so a sweep loads 4 + 2/K values a cell
//    instead of 7;
//  * a row of the staged brick holds its NX interior cells only, the two x
//    ghost faces lie apart (relax_at): a warp's 32 cells are then 32
//    neighbouring words, where rows of NX + 2 put every access in two
//    wavefronts (a sweep of a 12^3 FP32 brick by 864 threads: 669 cycles
//    before, a sweep and its decision 907);
//  * the FP64 sum (its last stages dependent 64-bit shuffles and adds, 500
//    to 1100 cycles) is formed for the last sweep only.  Before it the loop
//    compares an integer sum: every thread's squares scaled so that the
//    first sweep's sum, formed in FP32, is 2^22, cut to a whole number, and
//    added with one integer warp reduction per stage.  Unless that sum is
//    above the threshold by more than its error bound
//    (RELAX_CLEARLY_ABOVE), the FP64 sums are formed and decide, so every
//    decision is the FP64 sums'.
//
// Thread layout: TH threads (a multiple of 32 that divides NX^3) relax one
// brick, K = NX^3 / TH cells each: thread lt owns the cells of column
// lt % NX^2 (x fastest) at heights K (lt / NX^2) + r, r < K.  In the FP64
// sum cell t's square enters the partial of its 32-cell group t / 32 at lane
// t % 32 whatever TH is, so the partials, their pairwise sum and every loop
// decision are the same bit for bit for every layout: a whole block of 512
// threads on an 8^3 brick, two bricks of 256 threads each in one block, 576
// threads on a 12^3 brick.
#pragma once

namespace amr {

template <int NX, typename CT = double>
struct alignas(16) RelaxSmem {
    static constexpr int P = NX + 2, NT = NX * NX * NX, NW = NT / 32;
    static constexpr int B3 = NX * P * P + 2 * NX * NX;  // entries of a staged brick (relax_at)
    // A plane of 8^2 cells is two whole 32-cell groups, so a warp's cells of
    // one height are a group and its partial needs no other thread's value.
    // A plane of 12^2 is four and a half: the squares' roots then pass
    // through tmp (groups 40 apart, so that four groups lie in 32 banks).
    static constexpr bool DIRECT = (NX * NX) % 32 == 0;
    CT buf[2][B3];
    double red[64];        // partials of the FP64 sum
    unsigned qred[2][32];  // warp sums of the integer sum, by sweep parity
    float fred[32];        // warp sums of the first sweep's FP32 sum
    CT tmp[DIRECT ? 4 : NW * 40];
};

// Entry of cell (i, j, k), each 0..NX+1 with at most one of them a ghost, in
// a staged brick: rows of NX interior cells, then the two x ghost faces.
template <int NX>
__host__ __device__ __forceinline__ int relax_at(int i, int j, int k) {
    constexpr int P = NX + 2, GX = NX * P * P;
    if (i == 0) return GX + (k - 1) * NX + j - 1;
    if (i == NX + 1) return GX + NX * NX + (k - 1) * NX + j - 1;
    return i - 1 + NX * (j + P * k);
}

// Threads of a whole block relaxing one brick of NX^3 interior cells.
template <int NX>
struct RelaxThreads;
template <>
struct RelaxThreads<8> {
    static constexpr int value = 512;  // one cell per thread
};
template <>
struct RelaxThreads<12> {
    static constexpr int value = 576;  // three cells per thread
};

// Barrier over the threads that relax one brick.
struct BlockSync {
    __device__ __forceinline__ void operator()() const { __syncthreads(); }
};
// Barrier over `n` threads with id `id` (1..15; 0 is __syncthreads).
__device__ __forceinline__ void named_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
struct NamedSync {
    int id, n;
    __device__ __forceinline__ void operator()() const { named_sync(id, n); }
};

// Dynamic shared memory of a kernel (one declaration for every kernel).
__device__ __forceinline__ unsigned char* dyn_smem() {
    extern __shared__ __align__(16) unsigned char amr_dyn_smem[];
    return amr_dyn_smem;
}

// Interior cell t in the (NX+2)^3 array of dphi, and in a staged brick.
template <int NX>
__device__ __forceinline__ int relax_cell(int t) {
    constexpr int P = NX + 2;
    return ((t / (NX * NX) + 1) * P + (t / NX) % NX + 1) * P + t % NX + 1;
}
template <int NX>
__device__ __forceinline__ int relax_staged(int t) {
    return t % NX + NX * ((t / NX) % NX + 1 + (NX + 2) * (t / (NX * NX) + 1));
}

// Ghost face cell q (< 6 NX^2): its face, its face coordinates t1, t2
// (1..NX, along the lower and the higher of the two other axes), its index
// in the dphi array and in a staged brick.
template <int NX>
__device__ __forceinline__ void relax_ghost(int q, int& face, int& t1, int& t2, int& cell, int& staged) {
    constexpr int P = NX + 2, F = NX * NX;
    face = q / F;
    const int qq = q % F;
    t1 = qq % NX + 1;
    t2 = qq / NX + 1;
    const int ax = face >> 1, g = (face & 1) ? P - 1 : 0;
    const int i = ax == 0 ? g : t1, j = ax == 1 ? g : (ax == 0 ? t1 : t2), k = ax == 2 ? g : t2;
    cell = (k * P + j) * P + i;
    staged = relax_at<NX>(i, j, k);
}

// Interior index of cell r of thread lt (see the thread layout above).
template <int NX, int TH>
__device__ __forceinline__ int relax_index(int lt, int r) {
    constexpr int K = NX * NX * NX / TH;
    return lt % (NX * NX) + NX * NX * (K * (lt / (NX * NX)) + r);
}

// Sum of the NW group partials p[0..NW-1] (NW <= 64; every partial is a sum
// of squares, so >= 0) along a fixed pairwise tree, identical in every
// thread: partials 0..31 and 32..63 (0.0 where there is none) are each
// added along the xor butterfly (at span s = 1, 2, 4, 8, 16 partial q takes
// q ^ s), and the two halves' sums added last.  IEEE addition is
// commutative and an absent partner adds +0.0, which leaves a non-negative
// value unchanged, so every lane ends with the tree's sum bit for bit.  A
// lane loads the four partials of spans 1 and 2 itself; the other spans, and
// the halves, are shuffles between lanes (two for at most 16 partials, four
// for 64, instead of five and six).  p has room for 16 or 64 entries.
template <int NW>
__device__ __forceinline__ double pairwise_sum(const double* p) {
    static_assert(NW <= 16 || (NW > 32 && NW <= 64), "16 or 64 slots");
    constexpr int LANES = NW <= 16 ? 4 : 16;
    const int q = 4 * (threadIdx.x & (LANES - 1));
    const double2 a = *reinterpret_cast<const double2*>(p + q), b = *reinterpret_cast<const double2*>(p + q + 2);
    double v = ((q < NW ? a.x : 0.0) + (q + 1 < NW ? a.y : 0.0)) + ((q + 2 < NW ? b.x : 0.0) + (q + 3 < NW ? b.y : 0.0));
#pragma unroll
    for (int s = 1; s < LANES; s <<= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
    return v;
}

// resid / resid0 > 0.5, the sweep loop's test, without the division.  For
// resid0 >= 2^-1021 (so that 0.5 resid0 is a normal double, exact) the
// correctly rounded quotient exceeds 0.5 exactly when resid > 0.5 resid0:
// rounding is monotonic and 0.5 is a double, so the two can differ only if
// the exact quotient lay in (0.5, 0.5 + 2^-54], which would need
// 0 < resid - 0.5 resid0 <= 2^-54 resid0; but two different doubles differ
// by at least one unit in the last place of the smaller, here of
// 0.5 resid0, which is more than 2^-53 (0.5 resid0) = 2^-54 resid0.  Zero, subnormal, infinite and NaN values
// give the same answer both ways (any resid0 below the bound takes the
// division).
__device__ __forceinline__ bool above_half(double resid, double resid0) {
    return resid0 >= 0x1p-1021 ? resid > 0.5 * resid0 : resid / resid0 > 0.5;
}

// The integer sum that answers above_half(resid, resid0) for most sweeps: q
// is the sum over the brick's threads of floor(min(f, RELAX_CLEARLY_ABOVE + 1)),
// f the sum over a thread's cells of (s tmp0)^2 in FP32, with s =
// RELAX_SCALE / sqrt(r), r the first sweep's sum of squares formed in FP32, so
// that 2^22 stands for resid0 and 2^21 for the threshold.  Errors, in units of
// the 2^22: r carries one rounding each of a value, its square and at most
// 5 + 10 additions, 18 x 2^-24; s those of the reciprocal square root (2 ulp)
// and a product, twice in the square; a value, its product, square and
// K - 1 <= 5 additions one each: together below 36 x 2^-24 of the sum or 5
// near the threshold; the cuts take off less than one for each of at most 864
// threads.  The FP64 sums are within 2^-40.  So a q more than 1024 above 2^21
// means that the FP64 sum is above half of resid0 as well, and one more than
// 1024 below that it is below.  The minimum changes neither: a thread that it
// cuts short is above the threshold by itself, and so is q.  It keeps q below
// 864 (2^21 + 1025) < 2^31: in exact arithmetic the sum does not grow from
// sweep to sweep (the ghost faces stay fixed), but where a brick's values are
// at rounding level it can, by any factor.  (A finite first sweep stays
// finite: later values are bounded by the same cells'.  An r outside
// [1e-28, 1e28], where FP32 under- or overflows of single squares could
// matter, takes the FP64 sums in every sweep.)
constexpr float RELAX_SCALE = 2048.0f;
constexpr unsigned RELAX_HALF = 1u << 21, RELAX_MARGIN = 1024u;
constexpr unsigned RELAX_CLEARLY_ABOVE = RELAX_HALF + RELAX_MARGIN, RELAX_CLEARLY_BELOW = RELAX_HALF - RELAX_MARGIN;

// The FP64 sum of squares of the values tmp0[r] of every thread's cells:
// group partials, a barrier, and the pairwise sum in every thread.  Cell t's
// square is lane t % 32 of group t / 32; a group is added along the xor
// butterfly with spans 16, 8, 4, 2, 1.
template <int NX, int TH, typename CT, typename Sync>
__device__ __forceinline__ double relax_sum(RelaxSmem<NX, CT>& sm, int lt, const CT* tmp0, Sync sync) {
    using S = RelaxSmem<NX, CT>;
    constexpr int K = NX * NX * NX / TH;
    if constexpr (S::DIRECT) {
        // this warp's cells of height r are group(r).  Two groups' butterflies
        // are taken together: at span 16 the lower lanes keep group r's pair
        // sums and the upper ones group r + 1's, one shuffle carrying the
        // value each lane gives away; spans 8..1 stay within a half.
        const int lane = lt & 31;
        auto group = [&](int r) { return (K * (lt / (NX * NX)) + r) * (NX * NX / 32) + (lt % (NX * NX)) / 32; };
        double sq[K];
#pragma unroll
        for (int r = 0; r < K; r++) sq[r] = double(tmp0[r]) * double(tmp0[r]);
#pragma unroll
        for (int r = 0; r + 1 < K; r += 2) {
            const bool up = lane & 16;
            double v = (up ? sq[r + 1] : sq[r]) + __shfl_xor_sync(0xffffffffu, up ? sq[r] : sq[r + 1], 16);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if ((lane & 15) == 0) sm.red[up ? group(r + 1) : group(r)] = v;
        }
        if constexpr (K & 1) {
            double v = sq[K - 1];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) sm.red[group(K - 1)] = v;
        }
    } else {
        // through tmp: eight lanes a group, each adding the four values of
        // spans 16 and 8 itself, then three shuffles
#pragma unroll
        for (int r = 0; r < K; r++) {
            const int t = relax_index<NX, TH>(lt, r);
            sm.tmp[t + 8 * (t / 32)] = tmp0[r];
        }
        sync();
        constexpr int ALL = (8 * S::NW + 31) / 32 * 32;
        for (int u = lt; u < ALL; u += TH) {
            const int g = u / 8, o = u % 8;
            double v = 0.0;
            if (g < S::NW) {
                const CT* w = sm.tmp + 40 * g + o;
                const double a = double(w[0]), b = double(w[16]), c = double(w[8]), d = double(w[24]);
                v = (a * a + b * b) + (c * c + d * d);
            }
#pragma unroll
            for (int s = 4; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
            if (o == 0 && g < S::NW) sm.red[g] = v;
        }
    }
    sync();
    return pairwise_sum<S::NW>(sm.red);
}

// The sweeps on a brick staged in two buffers x, y (x holds every cell,
// ghosts included; y the same ghost faces), given as entries of CT from the
// start of the dynamic shared memory: the compiler then knows the address
// space and works in 32-bit addresses, where pointers picked at run time
// cost generic loads and 64-bit arithmetic in a loop that issue slots bound.
// Thread lt owns the K cells relax_index(lt, r) with dphi1 values d1[r].  Returns the last sweep's sum
// and the buffer that holds the relaxed brick.  sm holds the sums' scratch (x
// and y need not be its buffers).
template <int NX, int TH, typename CT, typename Sync>
__device__ __forceinline__ double relax_sweeps_in(unsigned x, unsigned y, RelaxSmem<NX, CT>& sm, int lt, const CT* d1,
                                                  unsigned* result, Sync sync, int* sweeps = nullptr) {
    constexpr int P = NX + 2, K = NX * NX * NX / TH, WT = TH / 32, PZ = NX * P;
    static_assert((NX * NX * NX) % TH == 0 && TH % 32 == 0 && NX % K == 0 && WT <= 32, "relaxation layout");
    static_assert(K <= 6 && TH <= 864, "error bound of the integer sum");
    const int lane = lt & 31, wp = lt >> 5;
    CT* S = reinterpret_cast<CT*>(dyn_smem());
    // entries of the lowest own cell and of every own cell's x neighbours (in
    // the row, or in a ghost face), in the buffer read next
    unsigned c = x + relax_staged<NX>(relax_index<NX, TH>(lt, 0));
    const int i = lt % NX + 1, j = (lt / NX) % NX + 1, k = K * (lt / (NX * NX)) + 1;
    unsigned xl[K], xu[K];
#pragma unroll
    for (int r = 0; r < K; r++) {
        xl[r] = x + relax_at<NX>(i - 1, j, k + r);
        xu[r] = x + relax_at<NX>(i + 1, j, k + r);
    }
    unsigned other = y - x;  // from the buffer read next to the one written next
    CT own[K], tmp0[K], first[K];
#pragma unroll
    for (int r = 0; r < K; r++) own[r] = S[c + r * PZ];
    // one sweep: own and tmp0 of this thread's cells; the buffers swap
    auto sweep = [&]() {
        CT below = S[c - PZ];
        const CT above = S[c + K * PZ];
        const unsigned w = c + other;
#pragma unroll
        for (int r = 0; r < K; r++) {
            const CT up = r + 1 < K ? own[r + 1 < K ? r + 1 : r] : above;
            const CT div = (S[xu[r]] + S[xl[r]] + S[c + r * PZ + NX] + S[c + r * PZ - NX] + up + below) - (own[r] * CT(6.0));
            below = own[r];
            tmp0[r] = d1[r] + div * (CT(1.0) / CT(6.0));
            own[r] = own[r] + tmp0[r];
            S[w + r * PZ] = own[r];
            xl[r] += other;
            xu[r] += other;
        }
        c = w;
        other = 0u - other;
    };
    // the first sweep and its sum in FP32
    sweep();
    float r0 = 0.0f;
#pragma unroll
    for (int r = 0; r < K; r++) {
        first[r] = tmp0[r];
        const float t = float(tmp0[r]);
        r0 += t * t;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r0 += __shfl_xor_sync(0xffffffffu, r0, o);
    if (lane == 0) sm.fred[wp] = r0;
    sync();
    r0 = lane < WT ? sm.fred[lane] : 0.0f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r0 += __shfl_xor_sync(0xffffffffu, r0, o);
    const bool scaled = r0 >= 1.0e-28f && r0 <= 1.0e28f;  // so resid0 is neither 0 nor infinite nor NaN
    const float s = scaled ? RELAX_SCALE * rsqrtf(r0) : 0.0f;
    bool exact0 = !scaled;  // resid0 is formed: at once, or when a decision asks for it
    double resid0 = exact0 ? relax_sum<NX, TH, CT>(sm, lt, first, sync) : 0.0;
    double resid = resid0;
    int iters = 1;
    if (scaled || above_half(resid0, resid0)) {
        for (;;) {
            sweep();
            float f = 0.0f;
#pragma unroll
            for (int r = 0; r < K; r++) {
                const float t = float(tmp0[r]) * s;
                f += t * t;
            }
            f = fminf(f, float(RELAX_CLEARLY_ABOVE + 1));  // no 32-bit sum can wrap
            const unsigned part = __reduce_add_sync(0xffffffffu, __float2uint_rz(f));
            if (lane == 0) sm.qred[iters & 1][wp] = part;
            sync();
            const unsigned q = __reduce_add_sync(0xffffffffu, lane < WT ? sm.qred[iters & 1][lane] : 0u);
            iters++;
            if (q > RELAX_CLEARLY_ABOVE && iters < 16) continue;
            resid = relax_sum<NX, TH, CT>(sm, lt, tmp0, sync);
            // far enough below the threshold, or the last sweep allowed
            if ((scaled && q < RELAX_CLEARLY_BELOW) || iters >= 16) break;
            if (!exact0) {
                sync();  // the sums' scratch is free again
                resid0 = relax_sum<NX, TH, CT>(sm, lt, first, sync);
                exact0 = true;
            }
            if (!above_half(resid, resid0)) break;
        }
    }
    *result = iters & 1 ? y : x;
    if (sweeps) *sweeps = iters;
    return resid;
}

// This thread's dphi1 values.
template <int NX, int TH, typename CT>
__device__ __forceinline__ void relax_load_d1(int lt, const CT* __restrict__ dphi1, CT* d1) {
    constexpr int K = NX * NX * NX / TH;
#pragma unroll
    for (int r = 0; r < K; r++) d1[r] = dphi1[relax_cell<NX>(relax_index<NX, TH>(lt, r))];
}

// Stages the brick: dphi's interior into x, its ghost faces into x and y.
template <int NX, int TH, typename CT>
__device__ __forceinline__ void relax_stage(unsigned x, unsigned y, const CT* __restrict__ dphi, int lt) {
    constexpr int K = NX * NX * NX / TH;
    CT* S = reinterpret_cast<CT*>(dyn_smem());
#pragma unroll
    for (int r = 0; r < K; r++) {
        const int t = relax_index<NX, TH>(lt, r);
        S[x + relax_staged<NX>(t)] = dphi[relax_cell<NX>(t)];
    }
    for (int q = lt; q < 6 * NX * NX; q += TH) {
        int face, t1, t2, cell, staged;
        relax_ghost<NX>(q, face, t1, t2, cell, staged);
        const CT v = dphi[cell];
        S[x + staged] = v;
        S[y + staged] = v;
    }
}

// The entry of a brick buffer in the dynamic shared memory.
template <typename CT>
__device__ __forceinline__ unsigned relax_entry(const CT* buf) {
    return (unsigned)(buf - reinterpret_cast<const CT*>(dyn_smem()));
}

// Stages the brick and relaxes it: returns the last sweep's sum and leaves
// the relaxed interior values of this thread's cells relax_index(lt, r) in
// out[r].  CT is the correction's storage and arithmetic type (FP64, or FP32
// in the mixed form); the sums of squares are formed in FP64 either way.
// sm lies in the dynamic shared memory.
template <int NX, int TH, typename CT, typename Sync>
__device__ __forceinline__ double relax_brick(RelaxSmem<NX, CT>& sm, const CT* __restrict__ dphi,
                                              const CT* __restrict__ dphi1, int lt, CT* out, Sync sync) {
    constexpr int K = NX * NX * NX / TH;
    const unsigned x = relax_entry(sm.buf[0]), y = relax_entry(sm.buf[1]);
    relax_stage<NX, TH, CT>(x, y, dphi, lt);
    CT d1[K];
    relax_load_d1<NX, TH, CT>(lt, dphi1, d1);
    sync();
    unsigned res;
    const double s = relax_sweeps_in<NX, TH, CT>(x, y, sm, lt, d1, &res, sync);
#pragma unroll
    for (int r = 0; r < K; r++)
        out[r] = reinterpret_cast<CT*>(dyn_smem())[res + relax_staged<NX>(relax_index<NX, TH>(lt, r))];
    return s;
}

}  // namespace amr
