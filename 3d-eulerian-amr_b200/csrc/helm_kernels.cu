// Helmholtz EOS kernels (helmholtz/helmeos.cpp), FP64, one thread per point
// (device code of one point in helm_device.cuh).
//
// Table in HBM (L2-resident, 42 MB): node[j][i][12] = f, f_d, f_t, f_dd, f_tt,
// f_dt, f_ddt, f_dtt, f_ddtt, pads -- a node is two 32-byte loads and one
// value; tj[j][4] = t, dt, 1/dt, 1/dt^2 and di[i][4] = d, dd, 1/dd, 1/dd^2
// (computed on the host exactly as read_helm_table does,
// helmeos.cpp:100-129), one 32-byte load each.
#include <cuda_runtime.h>

#include <algorithm>

#include "helm_device.cuh"
#include "launch.cuh"

namespace amr {

namespace {

// S: with entropies (only where s or dsdt is asked for: the logarithm and the
// square roots of the ion entropy are a tenth of a point's operations).  What
// bounds it: FP64 issue (about 900 operations a point, 0.8 ms for 2^24 points
// at 64 a clock and SM, 67% busy), and before the 32-byte table loads the
// first cache's gathers (30 load instructions a point, one line a lane each;
// 14 now).  2^24 points to p, e, cs in cgs: 1.62 -> 1.11-1.16 ms.  Four blocks an
// SM (128 registers) spill: 1.58 ms.
template <bool S>
__global__ void __launch_bounds__(128, 3) k_helm_eos(HelmTable H, long long n, const double* __restrict__ rho,
                                                  const double* __restrict__ T, const double* __restrict__ abar,
                                                  const double* __restrict__ zbar, double* p, double* e, double* cs,
                                                  double* cv, double* s, double* dsdt, int* __restrict__ status) {
    const long long step = (long long)gridDim.x * blockDim.x;
    long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (q >= n) return;
    double nr = rho[q], nt = T[q], na = abar[q], nz = zbar[q];
    for (; q < n; q += step) {
        HelmPoint o;
        const double r = nr, t = nt, ab = na, zb = nz;
        if (q + step < n) {  // the next point's inputs, on their way during this one
            nr = rho[q + step];
            nt = T[q + step];
            na = abar[q + step];
            nz = zbar[q + step];
        }
        helm_point<S>(H, r, t, ab, zb, o);
        status[q] = o.status;
        if (o.status == 1) continue;
        if (p) p[q] = o.p;
        if (e) e[q] = o.e;
        if (cs) cs[q] = o.cs;
        if (cv) cv[q] = o.cv;
        if constexpr (S) {
            if (s) s[q] = o.s;
            if (dsdt) dsdt[q] = o.dsdt;
        }
    }
}

// helmholtz_compute_T (helmeos.cpp:436-486): the steps of helm_invert_point,
// one EOS evaluation a loop pass and lane.  A lane that is done takes the next
// point of its warp's run of points, so a warp does not wait for its slowest
// lane at every point (the iterations of 32 points differ by a factor of two
// and more); the first evaluation (at the temperature floor), the Newton ones
// and the last are the same code, so lanes in different phases stay together.
// 3,000,001 points with 4.7 iterations on average: 3.71 ms with a thread to a
// point, 1.77 ms now.
template <bool S>
__global__ void __launch_bounds__(128, 3) k_helm_invert(HelmTable H, long long n, long long per_warp,
                                                        const double* __restrict__ rho,
                                                        const double* __restrict__ target,
                                                        const double* __restrict__ abar,
                                                        const double* __restrict__ zbar, int from_entropy,
                                                        double* __restrict__ T, double* p, double* e, double* cs,
                                                        double* cv, double* s, int* iters_out,
                                                        int* __restrict__ status) {
    const int lane = threadIdx.x & 31;
    const long long warp = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    long long next = warp * per_warp;  // of the warp's points, the first not taken
    const long long end = min(n, next + per_warp);
    enum { IDLE, FLOOR, NEWTON, LAST };
    int phase = IDLE, st = 0, iters = 0;
    long long q = 0;
    double r = 0.0, e0 = 0.0, ab = 1.0, zb = 0.0, Tq = 0.0, a = 1.0;
    for (;;) {
        const unsigned idle = __ballot_sync(0xffffffffu, phase == IDLE);
        if (phase == IDLE) {
            q = next + __popc(idle & ((1u << lane) - 1u));
            if (q < end) {
                r = rho[q];
                e0 = target[q];
                ab = abar[q];
                zb = zbar[q];
                Tq = T[q];
                phase = FLOOR;
            }
        }
        next += __popc(idle);
        if (__ballot_sync(0xffffffffu, phase != IDLE) == 0u) return;
        if (phase == IDLE) continue;
        HelmPoint o;
        const double T0 = hmax(Tq, HELM_TMIN);
        helm_point<S>(H, r, phase == FLOOR ? HELM_TMIN : Tq, ab, zb, o);
        r = o.rho;
        bool done = false;
        const double got = S && from_entropy ? o.s : o.e;
        if (phase == FLOOR) {
            st = o.status;
            iters = 0;
            a = 1.0;
            if (st == 1) {  // outside the table at the floor temperature
                status[q] = st;
                if (iters_out) iters_out[q] = 0;
                phase = IDLE;
                continue;
            }
            if (got >= e0) {
                Tq = HELM_TMIN;
                done = true;
            } else {
                phase = NEWTON;
            }
        } else {
            Tq = o.T;
            if (!st) st = o.status;
            if (phase == NEWTON) {
                const double f = got - e0;
                const double dT = -f / (S && from_entropy ? o.dsdt : o.cv);
                Tq += a * dT;
                Tq = hmax(Tq, (T0 + HELM_TMIN) / 2.0);
                iters++;
                if (iters % 10 == 0) a *= 0.9;
                if (Tq < HELM_TMIN) {
                    if (!st) st = 5;
                    phase = LAST;
                } else if (!(fabs(f / e0) >= 1.0e-9 && iters < 100)) {
                    phase = LAST;
                }
            } else {
                if (iters >= 100 && !st) st = 4;
                done = true;
            }
        }
        if (!done) continue;
        if (Tq < HELM_TMIN && !st) st = 5;
        status[q] = st;
        if (iters_out) iters_out[q] = iters;
        T[q] = Tq;
        if (st != 1) {
            if (p) p[q] = o.p;
            if (e) e[q] = o.e;
            if (cs) cs[q] = o.cs;
            if (cv) cv[q] = o.cv;
            if constexpr (S)
                if (s) s[q] = o.s;
        }
        phase = IDLE;
    }
}

// helmholtz_ztwd (helmeos.cpp:423-434)
__global__ void k_helm_ztwd(long long n, const double* __restrict__ zbar, const double* __restrict__ rho,
                            double* __restrict__ p, double* __restrict__ e) {
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
         q += (long long)gridDim.x * blockDim.x) {
        const double A = 6.023e+22;
        const double B = 9.7595e+5 * zbar[q];
        const double x = pow(rho[q] / B, 1.0 / 3.0);
        double pv;
        if (x > 0.1) {
            pv = A * (x * (2.0 * x * x - 3.0) * sqrt(x * x + 1.0) + 3.0 * log(x + sqrt(x * x + 1.0)));
        } else {
            pv = A * 1.6 * pow(x, 5);
        }
        p[q] = pv;
        e[q] = A * (8.0 * pow(x, 3) * (sqrt(x * x + 1.0) - 1.0)) - pv / rho[q];
    }
}

int grid_for(long long n) {
    // grid-stride loops over at most 148 SMs x 16 blocks of 128 threads
    const long long want = (n + 127) / 128;
    return (int)(want < 148LL * 16 ? (want > 0 ? want : 1) : 148LL * 16);
}

}  // namespace

void launch_helm_eos(const HelmTable& H, long long n, const double* rho, const double* T, const double* abar,
                     const double* zbar, double* p, double* e, double* cs, double* cv, double* s, double* dsdt,
                     int* status, cudaStream_t st) {
    if (n <= 0) return;
    const auto k = s || dsdt ? k_helm_eos<true> : k_helm_eos<false>;
    launch_k(k, grid_for(n), 128, 0, st, H, n, rho, T, abar, zbar, p, e, cs, cv, s, dsdt, status);
}

void launch_helm_invert(const HelmTable& H, long long n, const double* rho, const double* target,
                        const double* abar, const double* zbar, int from_entropy, double* T, double* p, double* e,
                        double* cs, double* cv, double* s, int* iters, int* status, cudaStream_t st) {
    if (n <= 0) return;
    // the warps that fit at once (148 SMs, three blocks of four warps each)
    // share the points, a whole warp's at least
    const long long warps = 148LL * 3 * 4, per_warp = std::max(32LL, (n + warps - 1) / warps);
    const int blocks = (int)((n + 4 * per_warp - 1) / (4 * per_warp));
    const auto k = s || from_entropy ? k_helm_invert<true> : k_helm_invert<false>;
    launch_k(k, blocks, 128, 0, st, H, n, per_warp, rho, target, abar, zbar, from_entropy, T, p, e, cs, cv, s, iters,
             status);
}

void launch_helm_ztwd(long long n, const double* zbar, const double* rho, double* p, double* e, cudaStream_t st) {
    if (n <= 0) return;
    launch_k(k_helm_ztwd, grid_for(n), 128, 0, st, n, zbar, rho, p, e);
}

}  // namespace amr
