// Persistent multigrid solve: the whole V-cycle loop of Poisson::solve (the
// drivers' `while (err > toler) vcycle()`, binary_driver.cpp:296-330) in one
// cooperative launch.  Every dependent step of the reference's sequence --
// restriction of phi level by level, the phi ghost faces / edges / vertices
// of each level, the down sweep (vcycle_down + relax_until(1.0)) and the up
// sweep (coarse correction, relax_until(0.05), retire, ghosts) of each
// level, the forces with their coarse-fine averages, the L1 error -- is a
// phase separated from the next by a grid barrier instead of a kernel
// boundary.  The phases run the same device functions as the
// one-launch-per-step kernels (poisson_ops.cuh, graph_ops.cuh), so the
// result is bitwise that of the plain and graph forms.
//
// Loop decisions (relaxation ratio, L1 error > tol) need the reference's
// nested sums over the per-brick values; every block forms them itself, in
// its own scratch, from the same values, so all blocks take the same
// decision without another barrier.  Per-brick values are double-buffered
// by pass so a block still summing one pass cannot see the next pass's.
//
// The grid barrier spins with a bound: a block that waits longer than the
// control block's wait limit (BARRIER_SPINS polls by default) sets the
// abort word, every block leaves at its next barrier, and the host reports
// AMR_ERR_TIMEOUT.
#include <cuda_runtime.h>

#include "graph_ops.cuh"
#include "launch.cuh"
#include "persistent.h"
#include "poisson_ops.cuh"

namespace amr {

namespace {

constexpr unsigned long long BARRIER_SPINS = 1ull << 22;

__device__ __forceinline__ int ld_volatile(const int* p) { return *(const volatile int*)p; }

// Grid-wide barrier of a cooperative launch; false when the solve aborted.
// The arrival counter only grows: barrier k of the launch completes when it
// reaches k * gridDim.x (target, kept by thread 0), so an arrival is one
// fire-and-forget release add and the wait one acquire load per poll.
// A block whose wait runs out sets the abort word and records status 3
// (AMR_ERR_TIMEOUT) in the control block itself, so the timeout is reported
// whichever block meets it and whatever the other solves of a captured step
// record after it (statuses only grow).
__device__ __forceinline__ void give_up(GridBarrier* bar, int* status) {
    atomicExch(&bar->abort, 1);
    atomicMax(status, 3);
}

__device__ __forceinline__ bool grid_sync(GridBarrier* bar, unsigned& target, unsigned long long limit, int* status) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int good = 1;
        target += gridDim.x;
        // the release orders the whole block's writes (made before the block
        // barrier above) before the arrival, at GPU scope
        asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(&bar->count), "r"(1u) : "memory");
        unsigned long long spins = 0;
        for (;;) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&bar->count) : "memory");
            if ((int)(v - target) >= 0) break;
            if ((spins & 63) == 63 && ld_volatile(&bar->abort)) {
                good = 0;
                break;
            }
            if (++spins > limit) {
                give_up(bar, status);
                good = 0;
                break;
            }
            if (spins > 32) __nanosleep(20);
        }
        ok = good;
    }
    __syncthreads();
    return ok != 0;
}

// Block layout of the solve for bricks of NX^3 interior cells: TPB threads
// per block, NX^3 / TPB cells per thread in the relaxation (every layout
// gives the same results bit for bit).  With 8^3 bricks and 512 threads a
// block relaxes two bricks at once (one per half) on levels with more bricks
// than the shared-memory loop takes, so it holds two staged bricks; the other
// layouts take such levels brick by brick.  MINB: blocks per SM the registers are
// budgeted for.  resb: the bricks one block can hold in the shared-memory
// relaxation loop, as many as leave room for MINB blocks per SM (three
// buffers and dphi1 each: 28 KB for an 8^3 brick in FP64, 80 KB for a 12^3
// one, half of that in FP32).  A level of more bricks than that goes through
// the grid barrier once a pass, at 12.7 us a pass for the 408 bricks of the
// 4-level star on 296 blocks, against 7 us for its levels held in shared
// memory.
template <int NX, int TPB_>
struct SolveLayout {
    static constexpr int TPB = TPB_;
    static constexpr bool HALVES = NX == 8 && TPB == 512;
    static constexpr int NSM = HALVES ? 2 : 1;
    template <typename CT>
    static constexpr int resb() {
        if (NX == 8) return TPB == 512 ? (sizeof(CT) == 4 ? 4 : 3) : (sizeof(CT) == 4 ? 2 : 1);
        return TPB == 864 ? (sizeof(CT) == 4 ? 4 : 2) : TPB == 576 && sizeof(CT) == 4 ? 2 : 1;
    }
    static constexpr int MINB = TPB >= 864 ? 1 : (TPB > 288 ? 2 : (TPB > 256 ? 3 : 4));
    // threads per face in the face-ghost phases
    static constexpr int PF = NX * NX <= TPB / 6 ? NX * NX : TPB / 6;
};

template <int NX, int TPB_, typename CT>
struct Solver {
    using Lay = SolveLayout<NX, TPB_>;
    static constexpr int TPB = Lay::TPB;
    const SolveArgs& a;
    RelaxSmem<NX, CT>* sm;  // Lay::NSM staged bricks
    double* red;
    double* nbuf;    // 2 * NEST_SMEM doubles of shared memory for the level sums
    double* nest;    // this block's scratch [cap] (level sums of larger trees)
    int relax_par;   // pres buffer of the next relaxation pass
    int status;
    long long relax_calls;
    int max_outer;
    unsigned bar_target = 0;    // thread 0: arrivals that complete the next barrier
    unsigned lsum_gen = 0;      // level sums published so far in this launch
    unsigned pass_seq = 0;      // last pass word used by the shared-memory relaxation loops
    unsigned long long spin_limit = BARRIER_SPINS;  // polls per bounded wait
    unsigned long long t_last;  // block 0: global time at the last barrier exit
    // block 0's phase accounting, in shared memory
    unsigned long long* ph_ns;
    unsigned* ph_n;
    double* ph_bytes;
    unsigned long long* ph_wait;  // [PH_COUNT], then level-sum time and count
    unsigned* lvl_n;              // relaxation passes per level
    unsigned long long* lvl_ns;   // block 0's time in each level's relaxation loops
    unsigned long long* rsplit;   // block 0: the resident loops' time split [4], passes, sweeps
    double solo_sum = 0.0;        // the sum of a one-brick level's last pass

    __device__ static unsigned long long now() {
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        return t;
    }

    // barrier closing a phase of class ph
    __device__ bool sync(int ph, int units) {
        const unsigned long long t_arrive = (blockIdx.x == 0 && threadIdx.x == 0) ? now() : 0;
        const bool ok = grid_sync(a.bar, bar_target, spin_limit, &a.ctl->status);
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            const unsigned long long t = now();
            ph_wait[ph] += t - t_arrive;
            ph_ns[ph] += t - t_last;
            ph_n[ph]++;
            ph_bytes[ph] += (double)units * phase_bytes(ph);
            t_last = t;
        }
        return ok;
    }

    // Algorithmic HBM bytes of one unit (brick, parent or coarse-fine item)
    // of a phase: the arrays the phase must read and write once, at their
    // storage width (the correction dphi, dphi1 in CT).
    __device__ static double phase_bytes(int ph) {
        constexpr double PNX = NX + 2, H = NX / 2, C = sizeof(CT);
        switch (ph) {
            case PH_SOURCE: return 16 * PNX * PNX * PNX;                                  // rho -> S
            case PH_RESTRICT: return 8 * (8 * PNX * PNX * PNX + 8 * H * H * H);           // 8 children -> parent
            case PH_PHI_FACES: return 16 * 6 * NX * NX;                                   // source cell -> ghost
            case PH_PHI_EDGES: return 16 * 12 * NX;
            case PH_PHI_VERTICES: return 16 * 8;
            case PH_INIT: return 2 * C * PNX * PNX * PNX;                                 // dphi, dphi1 = 0
            case PH_VDOWN: return 8 * (PNX * PNX * PNX + NX * NX * NX) + 2 * C * NX * NX * NX;  // phi, S -> dphi, dphi1
            case PH_DPHI_FACES: return 2 * C * 6 * NX * NX;
            case PH_RELAX_FIRST:
            case PH_RELAX: return C * (PNX * PNX * PNX + 2 * NX * NX * NX + 12 * NX * NX);  // dphi, dphi1 -> dphi, layers
            case PH_CORRECT: return C * (2 * NX * NX * NX + H * H * H);
            case PH_RETIRE: return (16 + C) * NX * NX * NX;                               // phi += dphi
            case PH_FORCES: return 8 * (PNX * PNX * PNX + 3 * (PNX - 1) * (PNX - 1) * (PNX - 1));
            case PH_ADJUST_FORCE: return 8 * 5 * H * H;
            case PH_ERROR: return 8 * (3 * PNX * PNX * PNX + NX * NX * NX) + C * NX * NX * NX;
            default: return 0;
        }
    }

    // this block's share of n items
    template <typename F>
    __device__ void each(int n, F f) {
        for (int q = blockIdx.x; q < n; q += gridDim.x) f(q);
    }

    // one relaxation pass over the n bricks sl[]: one brick per block, or
    // (8^3 bricks) two per block, one per half with two cells per thread,
    // when the level has more bricks than there are blocks; the results are
    // the same either way
    __device__ void relax_pass(const int* sl, int n, int mode, const CT* rd, CT* wr, double* pres) {
        if (!Lay::HALVES || n <= (int)gridDim.x) {
            each(n, [&](int q) {
                op_relax_pass<NX, TPB, CT>(a.g, a.bt, a.st, sl[q], mode, rd, wr, a.stride, pres, sm[0], threadIdx.x,
                                           BlockSync{});
                __syncthreads();
            });
        } else if constexpr (Lay::HALVES) {
            constexpr int HT = TPB / 2;
            const int h = threadIdx.x / HT, lt = threadIdx.x % HT;
            for (int q = 2 * blockIdx.x + h; q < n; q += 2 * gridDim.x) {
                op_relax_pass<NX, HT, CT>(a.g, a.bt, a.st, sl[q], mode, rd, wr, a.stride, pres, sm[h & 1], lt,
                                          NamedSync{1 + h, HT});
                named_sync(1 + h, HT);
            }
        }
    }

    __device__ const int* level(int l) const { return a.L.slots + a.L.off[l]; }

    // enforce_phi_boundaries of one level: faces, then edges (reading the
    // neighbours' face ghosts), then vertices (reading their edge ghosts)
    __device__ bool phi_boundaries(int l) {
        const int* sl = level(l);
        const int n = a.L.cnt[l];
        const int t = threadIdx.x;
        constexpr int PF = Lay::PF;
        each(n, [&](int q) {
            if (t < 6 * PF) op_phi_faces(a.g, a.bt, a.st, a.aux, sl[q], t / PF, t % PF, PF);
        });
        if (!sync(PH_PHI_FACES, n)) return false;
        const int m = a.g.pnx - 2;
        each(n, [&](int q) {
            if (t < 12 * m) op_phi_edge(a.g, a.bt, a.st, a.aux, sl[q], t / m, t % m + 1);
        });
        if (!sync(PH_PHI_EDGES, n)) return false;
        each(n, [&](int q) {
            if (t < 8) op_phi_vertex(a.g, a.bt, a.st, a.aux, sl[q], t);
        });
        return sync(PH_PHI_VERTICES, n);
    }

    // Poisson::vcycle_relax sum over level l (poisson.cpp:107, nested as the
    // recursion adds it) from buffer `buf` of the per-brick sums
    __device__ double level_sum(int l, const double* buf) {
        const unsigned long long t0 = (blockIdx.x == 0 && threadIdx.x == 0) ? now() : 0;
        double r;
        if (l == 0) {
            r = __ldcg(buf + a.L.slots[a.L.off[0]]);
        } else {
            __syncthreads();
            if (a.L.max_cnt <= NEST_SMEM)
                r = nested_sum_smem(a.L, buf, l, false, nbuf);
            else
                r = nested_sum_block(a.L, a.bt.child, buf, nest, l, false);
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            ph_wait[PH_COUNT] += now() - t0;
            ph_wait[PH_COUNT + 1]++;
        }
        return r;
    }

    // the level sum published as generation lsum_gen (block 0 records the
    // time it waits for it).  Its two tagged halves carry the generation they
    // belong to, so a half of another sum is never taken for this one.  Two
    // mailboxes in turn: the server can be one generation ahead of a block
    // that has not read this one yet, never two (serve_sum).
    __device__ bool wait_sum(double& r) {
        const unsigned long long t0 = (blockIdx.x == 0 && threadIdx.x == 0) ? now() : 0;
        __shared__ double s_r;
        __shared__ int s_ok;
        if (threadIdx.x == 0) {
            unsigned hi, lo;
            const int good = tagged_get2(a.bar->lsum_tag + 2 * (lsum_gen & 1), lsum_gen, hi, lo);
            s_r = good ? join_halves(hi, lo) : 0.0;
            s_ok = good;
        }
        __syncthreads();
        r = s_r;
        const bool ok = s_ok != 0;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            ph_wait[PH_COUNT] += now() - t0;
            ph_wait[PH_COUNT + 1]++;
        }
        return ok;
    }

    // relax_until (poisson.cpp:66-70, 74-78): ghosts, one pass, then passes
    // with ghosts from the previous pass's snapshot until the level sum has
    // fallen to `ratio` of the first
    __device__ bool relax_until(int l, double ratio) {
        const unsigned long long t0 = (blockIdx.x == 0 && threadIdx.x == 0) ? now() : 0;
        const bool ok = relax_until_(l, ratio);
        if (blockIdx.x == 0 && threadIdx.x == 0) lvl_ns[l] += now() - t0;
        return ok;
    }
    __device__ bool relax_until_(int l, double ratio) {
        const int* sl = level(l);
        const int n = a.L.cnt[l];
        const int t = threadIdx.x;
        CT* snap = reinterpret_cast<CT*>(a.snap);
        constexpr int PF = Lay::PF;
        each(n, [&](int q) {
            if (t < 6 * PF) op_dphi_faces<CT>(a.g, a.bt, a.st, a.aux, sl[q], t / PF, t % PF, PF);
        });
        if (!sync(PH_DPHI_FACES, n)) return false;
        if (n <= (int)gridDim.x || n <= RESB * ((int)gridDim.x - 1)) return relax_loop_resident(l, ratio, sl, n);
        int par = 0;
        double* pres = a.pres + (size_t)relax_par * a.L.cap;
        relax_pass(sl, n, 0, snap, snap, pres);
        if (!sync(PH_RELAX_FIRST, n)) return false;
        const double r0 = level_sum(l, pres);
        relax_par ^= 1;
        relax_calls++;
        if (blockIdx.x == 0 && threadIdx.x == 0) lvl_n[l]++;
        int outer = 0;
        for (;;) {
            pres = a.pres + (size_t)relax_par * a.L.cap;
            const CT* rd = snap + (size_t)par * a.snap_half;
            CT* wr = snap + (size_t)(par ^ 1) * a.snap_half;
            relax_pass(sl, n, 1, rd, wr, pres);
            if (!sync(PH_RELAX, n)) return false;
            par ^= 1;
            const double r = level_sum(l, pres);
            relax_par ^= 1;
            relax_calls++;
            if (blockIdx.x == 0 && threadIdx.x == 0) lvl_n[l]++;
            ++outer;
            bool again = r / r0 > ratio;
            if (again && outer > max_outer) {
                again = false;
                status = 1;
            }
            if (!again) break;
        }
        return true;
    }

    // A pass's face layers and its sum travel as tagged entries: 32 bits of
    // the value and the pass word in one 64-bit store (tagged_put; an FP64
    // value is two such words).  A reader waits on the very words it reads, so
    // a pass needs neither a block barrier nor a release fence before its
    // layers are visible, nor a flag.  The buffers are zeroed before every
    // launch and pass words start at 1.
    static constexpr int RESB = Lay::template resb<CT>();
    static constexpr int WORDS = sizeof(CT) / 4;  // tagged words of a layer entry
    __device__ unsigned long long* tagged_snap(int p, int b) const {
        return a.tsnap + ((size_t)p * a.snap_half + (size_t)b * a.stride) * WORDS;
    }
    __device__ unsigned long long* tagged_sum(const double* pres, int b) const {
        return a.tpres + ((size_t)((pres - a.pres) / a.L.cap) * a.L.cap + b) * 2;
    }

    // Publishes the first interior layers of the relaxed brick `res` to
    // snapshot buffer `wpar` as pass word `seq`: those a same-level neighbour
    // reads (the other faces' ghosts come from the parent, the mirror or the
    // outflow value).
    __device__ void put_layers(int b, unsigned res, int wpar, unsigned seq) {
        constexpr int K = NX * NX * NX / TPB;
        unsigned long long* sw = tagged_snap(wpar, b);
        unsigned sib = 0;
#pragma unroll
        for (int f = 0; f < 6; f++) sib |= a.bt.ftype[6 * b + f] == FACE_SIB ? 1u << f : 0u;
#pragma unroll
        for (int r = 0; r < K; r++) {
            const int t = relax_index<NX, TPB>(threadIdx.x, r);
            relax_layer_put_tagged<NX, CT>(sw, t, smem()[res + relax_staged<NX>(t)], seq, sib);
        }
    }

    // Publishes brick b's sum of a pass (to the tagged twin of buffer pres).
    __device__ void put_sum(int b, const double* pres, double resid, unsigned seq) {
        if (threadIdx.x != 0) return;
        unsigned long long* w = tagged_sum(pres, b);
        const unsigned long long bits = (unsigned long long)__double_as_longlong(resid);
        tagged_put(w, (unsigned)(bits >> 32), seq);
        tagged_put(w + 1, (unsigned)bits, seq);
    }

    // Two adjacent tagged words (the halves of an FP64 value): waits until
    // both carry pass word `tag`, loading the two together in every poll;
    // false when the solve aborted or the wait ran out.
    __device__ bool tagged_get2(const unsigned long long* p, unsigned tag, unsigned& hi, unsigned& lo) {
        unsigned long long spins = 0;
        for (;;) {
            unsigned long long w0, w1;
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w0) : "l"(p) : "memory");
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w1) : "l"(p + 1) : "memory");
            if ((unsigned)(w0 >> 32) == tag && (unsigned)(w1 >> 32) == tag) {
                hi = (unsigned)w0;
                lo = (unsigned)w1;
                return true;
            }
            if ((spins & 63) == 63 && ld_volatile(&a.bar->abort)) return false;
            if (++spins > spin_limit) {
                give_up(a.bar, &a.ctl->status);
                return false;
            }
            if (spins > 8) __nanosleep(20);
        }
    }

    // The FP64 value of two 32-bit halves.
    __device__ static double join_halves(unsigned hi, unsigned lo) {
        return __longlong_as_double((long long)(((unsigned long long)hi << 32) | lo));
    }

    // A same-level neighbour's layer value of pass word `tag`; false when the
    // solve aborted or the wait ran out.
    __device__ bool tagged_get(const unsigned long long* p, unsigned tag, CT& v) {
        if constexpr (WORDS == 2) {
            unsigned hi, lo;
            if (!tagged_get2(p, tag, hi, lo)) return false;
            v = CT(join_halves(hi, lo));
            return true;
        }
        unsigned long long spins = 0;
        for (;;) {
            unsigned long long w;
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
            if ((unsigned)(w >> 32) == tag) {
                v = CT(__uint_as_float((unsigned)w));
                return true;
            }
            if ((spins & 63) == 63 && ld_volatile(&a.bar->abort)) return false;
            if (++spins > spin_limit) {
                give_up(a.bar, &a.ctl->status);
                return false;
            }
            if (spins > 8) __nanosleep(20);
        }
    }

    // One pass of brick b from its committed values in `base`, ghost faces
    // from snapshot `rpar` as pass word `want` (the parent across coarse-fine
    // faces, the mirror of `base` across z = 0, 0 on outflow faces), swept in
    // x and y; nothing is written outside shared memory.  Returns the sum and
    // the buffer with the relaxed brick (x or y).
    __device__ double resident_pass(int b, unsigned base, unsigned x, unsigned y, int rpar, unsigned want,
                                    const CT* d1, unsigned* res, bool& ok) {
        constexpr int K = NX * NX * NX / TPB, F = NX * NX;
        unsigned long long tt = (blockIdx.x == 0 && threadIdx.x == 0) ? now() : 0;
#pragma unroll
        for (int r = 0; r < K; r++) {
            const int q = relax_staged<NX>(relax_index<NX, TPB>(threadIdx.x, r));
            smem()[x + q] = smem()[base + q];
        }
        int bad = 0;
        for (int q = threadIdx.x; q < 6 * F; q += TPB) {
            int face, t1, t2, cell, gi;
            relax_ghost<NX>(q, face, t1, t2, cell, gi);
            CT v;
            if (a.bt.ftype[6 * b + face] == FACE_SIB) {
                const int nbr = a.bt.fnbr[6 * b + face];
                if (!tagged_get(tagged_snap(rpar, nbr) + layer_entry<NX>(face ^ 1, t1, t2) * WORDS, want, v)) {
                    bad = 1;
                    v = CT(0);
                }
            } else {
                v = ghost_dphi<NX, CT>(a.g, a.bt, a.st, nullptr, a.stride, b, face, t1, t2, smem() + base);
            }
            smem()[x + gi] = v;
            smem()[y + gi] = v;
        }
        ok = !__syncthreads_or(bad);
        if (!ok) return 0.0;
        split(0, tt);
        int sw;
        const double r = relax_sweeps_in<NX, TPB, CT>(x, y, sm[0], threadIdx.x, d1, res, BlockSync{}, &sw);
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            rsplit[4]++;
            rsplit[5] += sw;
        }
        split(1, tt);
        return r;
    }

    // block 0, thread 0: adds the time since *t to split s and restarts *t
    __device__ void split(int s, unsigned long long& t) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            const unsigned long long u = now();
            rsplit[s] += u - t;
            t = u;
        }
    }

    // The server's part of a pass: takes the bricks' tagged sums of pass word
    // `tag` straight into the shared buffer of the nested sum (or, for a level
    // too large for it, back whole to the pres buffer `done` that the level
    // sum reads), forms the level sum and publishes it as generation lsum_gen.
    // A brick sends its sum of pass k + 1 before it knows the decision on pass
    // k, so the next sum can be formed, and published in the other mailbox,
    // while a slow block still has this one to read; the sum after that needs
    // that block's pass k + 2, which it starts only after it has read this one.
    __device__ bool serve_sum(int l, const double* done, unsigned tag) {
        const int* sl = level(l);
        const int n = a.L.cnt[l];
        const bool in_smem = a.L.max_cnt <= NEST_SMEM;
        int bad = 0;
        for (int q = threadIdx.x; q < n; q += TPB) {
            const int b = sl[q];
            unsigned hi, lo;
            if (!tagged_get2(tagged_sum(done, b), tag, hi, lo)) {
                bad = 1;
                continue;
            }
            if (in_smem)
                nbuf[q] = join_halves(hi, lo);
            else
                const_cast<double*>(done)[b] = join_halves(hi, lo);
        }
        if (__syncthreads_or(bad)) return false;
        const double r = !in_smem ? level_sum(l, done) : l == 0 ? nbuf[0] : nested_sum_smem_in(a.L, done, l, false, nbuf);
        if (threadIdx.x == 0) {
            unsigned long long* w = a.bar->lsum_tag + 2 * (lsum_gen & 1);
            const unsigned long long bits = (unsigned long long)__double_as_longlong(r);
            tagged_put(w, (unsigned)(bits >> 32), lsum_gen);
            tagged_put(w + 1, (unsigned)bits, lsum_gen);
        }
        // the shared buffer is read again by the next pass's sum
        __syncthreads();
        return true;
    }

    // Entries, in the dynamic shared memory, of brick buffer i (0..2) of the
    // shared-memory loop's brick j (0..RESB-1) -- the staged bricks' buffers
    // first, then those behind them -- and of dphi1 of this thread's cells.
    static constexpr int B3 = RelaxSmem<NX, CT>::B3;
    static constexpr unsigned EXT = Lay::NSM * sizeof(RelaxSmem<NX, CT>) / sizeof(CT);
    __device__ static CT* smem() { return reinterpret_cast<CT*>(dyn_smem()); }
    __device__ static unsigned resident_buf(int j, int i) {
        constexpr unsigned SM = sizeof(RelaxSmem<NX, CT>) / sizeof(CT);
        const unsigned q = 3 * j + i;
        return q < 2 * Lay::NSM ? (q / 2) * SM + (q % 2) * B3 : EXT + (q - 2 * Lay::NSM) * B3;
    }
    __device__ static unsigned resident_d1(int j) {
        return EXT + (3 * RESB - 2 * Lay::NSM) * B3 + j * NX * NX * NX + threadIdx.x;
    }

    // Pass 0 of brick j in slot b: the ghost faces are in dphi (filled by the
    // face phase).  Returns its sum, the buffer number of the result in *ri.
    __device__ double first_pass(int j, int b, int* ri) {
        constexpr int K = NX * NX * NX / TPB, P3 = (NX + 2) * (NX + 2) * (NX + 2);
        const unsigned x = resident_buf(j, 0), y = resident_buf(j, 1);
        relax_stage<NX, TPB, CT>(x, y, Corr<CT>::dphi(a.st) + (size_t)b * P3, threadIdx.x);
        CT d1[K];
        relax_load_d1<NX, TPB, CT>(threadIdx.x, Corr<CT>::dphi1(a.st) + (size_t)b * P3, d1);
#pragma unroll
        for (int r = 0; r < K; r++) smem()[resident_d1(j) + r * TPB] = d1[r];
        __syncthreads();
        unsigned res;
        const double rs = relax_sweeps_in<NX, TPB, CT>(x, y, sm[0], threadIdx.x, d1, &res, BlockSync{});
        *ri = res == x ? 0 : 1;
        return rs;
    }

    // A later pass of brick j from its committed buffer i.
    __device__ double next_pass(int j, int b, int i, int rpar, unsigned want, int* ri, bool& ok) {
        constexpr int K = NX * NX * NX / TPB;
        CT d1[K];
#pragma unroll
        for (int r = 0; r < K; r++) d1[r] = smem()[resident_d1(j) + r * TPB];
        const unsigned x = resident_buf(j, (i + 1) % 3);
        unsigned res;
        const double rs = resident_pass(b, resident_buf(j, i), x, resident_buf(j, (i + 2) % 3), rpar, want, d1, &res,
                                        ok);
        *ri = res == x ? (i + 1) % 3 : (i + 2) % 3;
        return rs;
    }

    // A committed brick back to dphi: interior and ghost faces.
    __device__ void write_back(int b, unsigned B) {
        constexpr int K = NX * NX * NX / TPB, P3 = (NX + 2) * (NX + 2) * (NX + 2), F = NX * NX;
        CT* D = Corr<CT>::dphi(a.st) + (size_t)b * P3;
#pragma unroll
        for (int r = 0; r < K; r++) {
            const int t = relax_index<NX, TPB>(threadIdx.x, r);
            D[relax_cell<NX>(t)] = smem()[B + relax_staged<NX>(t)];
        }
        for (int q = threadIdx.x; q < 6 * F; q += TPB) {
            int face, t1, t2, cell, gi;
            relax_ghost<NX>(q, face, t1, t2, cell, gi);
            D[cell] = smem()[B + gi];
        }
    }

    // what every block keeps of a finished loop whose last published pass is k
    __device__ void loop_done(unsigned k) {
        relax_par ^= (1 + k) & 1;
        lsum_gen += 1 + k;
        relax_calls += k + 1;
        // one word more than the passes published: a sum of the pass that was
        // dropped may be out under it
        pass_seq += k + 2;
    }

    // The relaxation loop of a level the blocks can hold in shared memory:
    // one brick per block, the last block (the server) forming the level
    // sums; or, where the level has more bricks than blocks, up to RESB
    // bricks in every worker block and none in the server.  The bricks stay
    // in shared memory for the whole loop.  No grid barrier between passes: a
    // brick waits only for its same-level neighbours' published face layers,
    // computes the next pass from shared memory and sends its sum, while the
    // server forms the last pass's nested sum; that sum decides whether the
    // pass's layers are published, else it is dropped.  A sum goes out as
    // soon as it is known, before the decision on the pass before it, so the
    // decision is there when the next pass is done (the wait for it was 1.7
    // of 7.8 us a pass on the 5-level binary).  A block with several bricks
    // takes them one after the other in every pass; a server with a brick (as
    // many bricks as blocks) forms the sum first, then its pass, so its brick
    // trails the others by the sum's latency -- a smaller delay than a second
    // brick in one block.  A level of one brick (the root) needs no other
    // block: its block decides by itself.  The loop ends with one write of
    // each brick (interior and ghost faces) back to dphi and one grid
    // barrier.  Passes written, their values, the sums and every loop
    // decision are those of the loop in relax_until.
    __device__ bool relax_loop_resident(int l, double ratio, const int* sl, int n) {
        const int W = (int)gridDim.x - 1;
        const bool solo = n == 1;
        const bool server = !solo && (int)blockIdx.x == W;
        const bool many = n > (int)gridDim.x;
        // this block's bricks are sl[blockIdx.x + j W], j < nb
        const int nb = (int)blockIdx.x >= n || (many && server) ? 0 : many ? (n - (int)blockIdx.x + W - 1) / W : 1;
        const unsigned seq0 = pass_seq + 1;  // pass word of pass 0
        if (!nb && !server) {
            // a block without a brick has no part in the loop: it goes to
            // the closing barrier (one polled word instead of the loop's
            // published sums) and takes the loop's length from the block
            // that stores it before it arrives there
            if (!sync(PH_RELAX, 0)) return false;
            loop_done(*(volatile const unsigned*)&a.bar->relax_done_k);
            return true;
        }
        // buffer numbers (two bits a brick) of the bricks' committed values
        // and of the pass being computed
        unsigned ib = 0, inext = 0;
        unsigned k = 0;  // last published pass
        int outer = 1;
        auto par = [&](unsigned pass) { return a.pres + (size_t)((relax_par ^ pass) & 1) * a.L.cap; };
        auto step = [&](unsigned pass) -> bool {  // every brick's pass; its sum sent, its layers not yet
            inext = 0;
#pragma unroll 1
            for (int j = 0; j < nb; j++) {
                const int b = sl[blockIdx.x + j * W];
                bool ok = true;
                int ri;
                const double rs = pass == 0 ? first_pass(j, b, &ri)
                                            : next_pass(j, b, (ib >> (2 * j)) & 3, (pass - 1) & 1, seq0 + pass - 1, &ri,
                                                        ok);
                if (!ok) return false;
                inext |= (unsigned)ri << (2 * j);
                if (solo)
                    solo_sum = rs;
                else
                    put_sum(b, par(pass), rs, seq0 + pass);
            }
            return true;
        };
        auto publish = [&](unsigned pass) {  // the pass just computed becomes the committed one
            ib = inext;
            if (!solo)
#pragma unroll 1
                for (int j = 0; j < nb; j++)
                    put_layers(sl[blockIdx.x + j * W], resident_buf(j, (ib >> (2 * j)) & 3), pass & 1, seq0 + pass);
            if (blockIdx.x == 0 && threadIdx.x == 0) lvl_n[l]++;
        };
        const unsigned gen0 = lsum_gen;
        if (!step(0)) return false;
        publish(0);
        double r0 = solo_sum, r;
        // pass 1 runs whatever the first sum; that sum is formed meanwhile
        lsum_gen = gen0 + 1;
        if (server && !serve_sum(l, par(0), seq0)) return false;
        if (!step(1)) return false;
        publish(1);
        if (!solo && !wait_sum(r0)) return false;
        k = 1;
        for (;;) {
            lsum_gen = gen0 + 1 + k;
            if (solo) {
                r = solo_sum;
            } else {
                if (server && !serve_sum(l, par(k), seq0 + k)) return false;
                unsigned long long tt = 0;
                // the next pass, held until the sum of the last one decides
                // whether it is published
                if (!step(k + 1)) return false;
                if (blockIdx.x == 0 && threadIdx.x == 0) tt = now();
                if (!wait_sum(r)) return false;
                split(2, tt);
            }
            bool again = r / r0 > ratio;
            if (again && outer > max_outer) {
                again = false;
                status = 1;
            }
            if (!again) break;
            if (solo && !step(k + 1)) return false;
            unsigned long long tt = (blockIdx.x == 0 && threadIdx.x == 0) ? now() : 0;
            publish(k + 1);
            split(3, tt);
            ++k;
            ++outer;
        }
#pragma unroll 1
        for (int j = 0; j < nb; j++) write_back(sl[blockIdx.x + j * W], resident_buf(j, (ib >> (2 * j)) & 3));
        // the loop's length for the blocks without a brick
        if ((server || solo) && threadIdx.x == 0) a.bar->relax_done_k = k;
        lsum_gen = gen0;
        loop_done(k);
        return sync(PH_RELAX, n * (k + 1));
    }

    // Poisson::vcycle (poisson.cpp:1069-1074) = vcycle0 (poisson.cpp:53-84)
    // without the two dphi ghost fills that nothing reads (see vcycle0 in
    // poisson_host.cpp)
    __device__ bool vcycle() {
        const int t = threadIdx.x;
        const int maxl = a.nlevels - 1;
        each(a.L.nall, [&](int q) { op_set_source(a.g, a.st, a.L.all[q], t, blockDim.x); });
        if (!sync(PH_SOURCE, a.L.nall)) return false;
        for (int l = maxl - 1; l >= 0; l--) {
            const int* pl = a.parents + a.poff[l];
            constexpr int H3 = (NX / 2) * (NX / 2) * (NX / 2);
            each(a.pcnt[l], [&](int q) {
                for (int u = t; u < 8 * H3; u += TPB) op_phi_from_children(a.g, a.bt, a.st, pl[q], u / H3, u % H3);
            });
            if (!sync(PH_RESTRICT, a.pcnt[l])) return false;
        }
        for (int l = 0; l <= maxl; l++)
            if (!phi_boundaries(l)) return false;
        each(a.L.nall, [&](int q) { op_init_vcycle<CT>(a.g, a.st, a.L.all[q], t, blockDim.x); });
        if (!sync(PH_INIT, a.L.nall)) return false;
        // down sweep (levels maxl .. 0), then up sweep (0 .. maxl), as one
        // loop so that the relaxation loop is expanded once
        for (int step = 0; step < 2 * (maxl + 1); step++) {
            const bool down = step <= maxl;
            const int l = down ? maxl - step : step - (maxl + 1);
            const int* sl = level(l);
            if (down) {
                each(a.L.cnt[l], [&](int q) {
                    op_vdown<CT>(a.g, a.bt, a.st, sl[q], a.vitems, a.vranges + 4 * (a.voff[l] + q));
                    __syncthreads();
                });
                if (!sync(PH_VDOWN, a.L.cnt[l])) return false;
            } else if (l > 0) {
                each(a.L.cnt[l], [&](int q) { op_coarse_correction<CT>(a.g, a.bt, a.st, sl[q], t); });
                if (!sync(PH_CORRECT, a.L.cnt[l])) return false;
            }
            if (!relax_until(l, down ? 1.0 : 0.05)) return false;
            if (!down) {
                each(a.L.cnt[l], [&](int q) { op_retire<CT>(a.g, a.st, sl[q], t, blockDim.x); });
                if (!sync(PH_RETIRE, a.L.cnt[l])) return false;
                if (!phi_boundaries(l)) return false;
            }
        }
        return true;
    }

    // compute_forces + adjust_{x,y,z}_force level by level, finest first
    __device__ bool forces() {
        const int t = threadIdx.x;
        each(a.L.nall, [&](int q) { op_forces(a.g, a.bt, a.st, a.L.all[q], t, blockDim.x); });
        if (!sync(PH_FORCES, a.L.nall)) return false;
        for (int l = a.force_levels - 1; l >= 0; l--) {
            const int n = a.foff[l + 1] - a.foff[l];
            if (n <= 0) continue;
            const RefluxItem* it = a.fitems + a.foff[l];
            each(n, [&](int q) { op_adjust_force(a.g, a.st, it[q], t); });
            if (!sync(PH_ADJUST_FORCE, n)) return false;
        }
        return true;
    }

    // Poisson::solution_error (poisson.cpp:637-669), nested over the tree;
    // the per-brick sums with 256 threads, as the error kernels form them
    __device__ bool error(double* err) {
        const int nl = a.nlevels;
        double* perr = a.pres + 2 * (size_t)a.L.cap;
        each(a.L.nall, [&](int q) {
            op_solution_error<CT>(a.g, a.bt, a.st, a.L.all[q], perr, red, 256);
            __syncthreads();
        });
        if (!sync(PH_ERROR, a.L.nall)) return false;
        if (a.L.max_cnt <= NEST_SMEM) {
            *err = nested_sum_smem(a.L, perr, nl - 1, true, nbuf);
            return true;
        }
        // deepest level: nest = own; then own + children level by level
        const int* sl = a.L.slots + a.L.off[nl - 1];
        for (int q = threadIdx.x; q < a.L.cnt[nl - 1]; q += blockDim.x) nest[sl[q]] = __ldcg(perr + sl[q]);
        __syncthreads();
        *err = nested_sum_block(a.L, a.bt.child, perr, nest, nl - 1, true);
        return true;
    }
};

template <int NX, int TPB, typename CT>
__global__ void __launch_bounds__(TPB, SolveLayout<NX, TPB>::MINB) k_solve_persistent(SolveArgs a) {
    // the staged bricks live in dynamic shared memory, the further brick
    // buffers of the shared-memory relaxation loop and its dphi1 behind them
    RelaxSmem<NX, CT>* sm = reinterpret_cast<RelaxSmem<NX, CT>*>(dyn_smem());
    __shared__ double red[16];
    __shared__ double nbuf[2 * NEST_SMEM];
    __shared__ double s_err;
    // loop limits are read from the control block (set by the host before
    // every launch; a captured graph keeps its arguments)
    const int max_cycles = *(volatile int*)&a.ctl->max_cycles;
    Solver<NX, TPB, CT> s{a, sm, red, nbuf, a.nest + (size_t)blockIdx.x * a.L.cap, 0, 0, 0,
                 *(volatile int*)&a.ctl->max_outer};
    __shared__ unsigned long long s_ph_ns[PH_COUNT];
    __shared__ unsigned s_ph_n[PH_COUNT];
    __shared__ double s_ph_bytes[PH_COUNT];
    __shared__ unsigned long long s_ph_wait[PH_COUNT + 2];
    {
        const int wl = *(volatile int*)&a.ctl->wait_limit;
        if (wl > 0) s.spin_limit = (unsigned long long)wl;
    }
    __shared__ unsigned s_lvl_n[MAX_LEVELS];
    s.lvl_n = s_lvl_n;
    __shared__ unsigned long long s_lvl_ns[MAX_LEVELS];
    s.lvl_ns = s_lvl_ns;
    __shared__ unsigned long long s_rsplit[6];
    s.rsplit = s_rsplit;
    if (threadIdx.x < 6) s_rsplit[threadIdx.x] = 0;
    if (threadIdx.x < MAX_LEVELS) {
        s_lvl_n[threadIdx.x] = 0;
        s_lvl_ns[threadIdx.x] = 0;
    }
    s.ph_ns = s_ph_ns;
    s.ph_n = s_ph_n;
    s.ph_bytes = s_ph_bytes;
    s.ph_wait = s_ph_wait;
    if (threadIdx.x < PH_COUNT + 2) s_ph_wait[threadIdx.x] = 0;
    s.t_last = Solver<NX, TPB, CT>::now();
    if (threadIdx.x < PH_COUNT) {
        s_ph_ns[threadIdx.x] = 0;
        s_ph_n[threadIdx.x] = 0;
        s_ph_bytes[threadIdx.x] = 0.0;
    }
    __syncthreads();
    int cycles = 0;
    bool ok = true;
    double err = 0.0;
    for (;;) {
        if (!(ok = s.vcycle())) break;
        if (!(ok = s.forces())) break;
        if (!(ok = s.error(&err))) break;
        if (threadIdx.x == 0) s_err = err;
        __syncthreads();
        err = s_err;
        cycles++;
        if (!(err > a.tol)) break;
        if (cycles >= max_cycles) {
            s.status = 2;
            break;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        Control* c = a.ctl;
        if (!ok) {
            atomicMax(&c->status, 3);
        } else {
            c->err = err;
            c->cycles = cycles;
            c->cycles_total += cycles;
            c->relax_calls += s.relax_calls;
            if (s.status) atomicMax(&c->status, s.status);
            for (int p = 0; p < PH_COUNT; p++) {
                c->phase_ns[p] += s.ph_ns[p];
                c->phase_n[p] += s.ph_n[p];
                c->phase_bytes[p] += s.ph_bytes[p];
                c->phase_wait_ns[p] += s.ph_wait[p];
            }
            c->level_sum_ns += s.ph_wait[PH_COUNT];
            c->level_sum_n += s.ph_wait[PH_COUNT + 1];
            for (int l = 0; l < MAX_LEVELS; l++) {
                c->relax_level[l] += s.lvl_n[l];
                c->relax_level_ns[l] += s.lvl_ns[l];
            }
            for (int q = 0; q < 4; q++) c->relax_split_ns[q] += s.rsplit[q];
            c->relax_split_passes += s.rsplit[4];
            c->relax_split_sweeps += s.rsplit[5];
        }
    }
}

}  // namespace

template <int NX, int TPB, typename CT>
constexpr size_t solve_smem() {
    using Lay = SolveLayout<NX, TPB>;
    constexpr int B = Lay::template resb<CT>();
    static_assert(3 * B >= 2 * Lay::NSM, "the staged bricks' buffers are the loop's first ones");
    return Lay::NSM * sizeof(RelaxSmem<NX, CT>) +
           sizeof(CT) * ((3 * B - 2 * Lay::NSM) * (size_t)RelaxSmem<NX, CT>::B3 + (size_t)B * NX * NX * NX);
}

namespace {

// The layouts of each brick size, in the order of their layout number.
constexpr int LAYOUTS_8[] = {512, 256};
constexpr int LAYOUTS_12[] = {576, 864, 288};

template <int NX, int TPB, typename CT>
cudaError_t set_attr() {
    return cudaFuncSetAttribute((const void*)k_solve_persistent<NX, TPB, CT>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)solve_smem<NX, TPB, CT>());
}
template <int NX, int TPB, typename CT>
int occupancy() {
    int per = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_solve_persistent<NX, TPB, CT>, TPB,
                                                      solve_smem<NX, TPB, CT>()) != cudaSuccess)
        return -1;
    return per;
}
template <int NX, int TPB, typename CT>
cudaError_t launch(const SolveArgs& a, int blocks, cudaStream_t s) {
    void* args[] = {const_cast<SolveArgs*>(&a)};
    return cudaLaunchCooperativeKernel((const void*)k_solve_persistent<NX, TPB, CT>, dim3(blocks), dim3(TPB), args,
                                       solve_smem<NX, TPB, CT>(), s);
}

// Calls OP<NX, TPB, CT>::run(args...) for the layout (nx, layout, FP32?);
// returns `bad` for an unknown one.
#define AMR_SOLVE_DISPATCH(nx, layout, f32, bad, CALL)                  \
    do {                                                                \
        if ((nx) == 8) {                                                \
            if ((layout) == 0) return (f32) ? CALL(8, 512, float) : CALL(8, 512, double);   \
            if ((layout) == 1) return (f32) ? CALL(8, 256, float) : CALL(8, 256, double);   \
        } else if ((nx) == 12) {                                        \
            if ((layout) == 0) return (f32) ? CALL(12, 576, float) : CALL(12, 576, double); \
            if ((layout) == 1) return (f32) ? CALL(12, 864, float) : CALL(12, 864, double); \
            if ((layout) == 2) return (f32) ? CALL(12, 288, float) : CALL(12, 288, double); \
        }                                                               \
        return (bad);                                                   \
    } while (0)

#define AMR_OCC(NX, TPB, CT) occupancy<NX, TPB, CT>()
#define AMR_LAUNCH(NX, TPB, CT) launch<NX, TPB, CT>(a, blocks, s)

int occupancy_of(int nx, int layout, bool f32) { AMR_SOLVE_DISPATCH(nx, layout, f32, -1, AMR_OCC); }

}  // namespace

int solve_layouts(int nx) {
    return nx == 8 ? (int)(sizeof(LAYOUTS_8) / sizeof(int)) : nx == 12 ? (int)(sizeof(LAYOUTS_12) / sizeof(int)) : 0;
}

int solve_layout_threads(int nx, int layout) {
    if (layout < 0 || layout >= solve_layouts(nx)) return -1;
    return nx == 8 ? LAYOUTS_8[layout] : LAYOUTS_12[layout];
}

int solve_persistent_attributes() {
    cudaError_t e = cudaSuccess;
    auto chk = [&](cudaError_t r) {
        if (e == cudaSuccess) e = r;
    };
    chk(set_attr<8, 512, float>());
    chk(set_attr<8, 512, double>());
    chk(set_attr<8, 256, float>());
    chk(set_attr<8, 256, double>());
    chk(set_attr<12, 576, float>());
    chk(set_attr<12, 576, double>());
    chk(set_attr<12, 864, float>());
    chk(set_attr<12, 864, double>());
    chk(set_attr<12, 288, float>());
    chk(set_attr<12, 288, double>());
    return e == cudaSuccess ? 0 : -1;
}

int solve_persistent_blocks(int nx, int precision, int per_sm_cap, int layout) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return -1;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -1;
    int per = occupancy_of(nx, layout, precision == AMR_PREC_MIXED);
    if (per <= 0) return -1;
    if (per_sm_cap > 0 && per_sm_cap < per) per = per_sm_cap;
    return sms * per;
}

cudaError_t launch_solve_persistent(const SolveArgs& a, int blocks, int layout, cudaStream_t s) {
    ++g_launch_tally;
    AMR_SOLVE_DISPATCH(a.g.nx, layout, a.g.precision == AMR_PREC_MIXED, cudaErrorInvalidValue, AMR_LAUNCH);
}

#undef AMR_OCC
#undef AMR_LAUNCH
#undef AMR_SOLVE_DISPATCH

}  // namespace amr
