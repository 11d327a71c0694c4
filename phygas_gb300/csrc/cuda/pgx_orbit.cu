// pgx_orbit.cu -- FP64 orbit kernels of libphygas_gb300: the state-transition tracks of the linear screen and the
// clone Monte Carlo of ph_pair with its quantile reduction.
//
//   k_stm_orbits   one thread per orbit: an object's nominal orbit and its 6 neighbours (+1e-5 on one phase-space
//                  axis) are 7 independent threads, so a warp is 32 orbits with identical work and no barrier
//                  (reference lin_integrate, src/phygas.c:286-323); k_stm_orbits_quad: four lanes per orbit, for few
//                  objects
//   k_stm_cov      one thread per (object, point): A = (neighbour - nominal) / eps, S = A Sigma0 A^T, and the
//                  track layouts the screen reads (FP64 for the exact stages, split FP32 for the filter, and a
//                  lower bound on the smallest eigenvalue of S for the filter's error bounds)
//   k_mc_prep, k_pair_mc_t, k_pair_reduce_dev  the clone Monte Carlo as one captured CUDA graph, its parameters read
//                  from device memory.  k_pair_mc_t is persistent: warps take items of clones of one pair from a device
//                  queue (longest first) and trace them back with KDK leapfrog and the segment closest approach
//                  (reference ph_pair_clone, src/phygas.c:200-216), on the FP32 and integer units where they are as
//                  accurate; its launch shape (warps per block, clones per lane) is a template the autotuner picks.
//                  k_pair_mc_quad: eight lanes per clone, for batches of few clones.  k_pair_reduce_dev: a warp per
//                  pair reduces it in registers with warp shuffles (reference ph_pair_reduce, src/phygas.c:218-238)
//   k_pair_reduce_big  the same reduction for pairs of more than 1024 clones, one CTA per pair
//
// Built with --fmad=false: every fused multiply-add is an explicit fma(), so the rounding does not depend on how the
// compiler arranges a kernel, and every launch shape gives the same bits.
#include <algorithm>
#include <cstdio>
#include <mutex>

#include "phygas_gb300.h"
#include "pgx_force.cuh"
#include "pgx_kernels.h"

namespace pgx {

// npts == nullptr: every object has nmax points.  Orbit t of the 7 N (object i = t % N, axis j = t / N) per
// thread, grid-stride, so a small grid can trace a chunk beside other work (one orbit per thread with a full grid).
// The start of orbit j of an object: its nominal state, +1e-5 on phase-space axis j - 1.
__device__ __forceinline__ double stm_start(const double *__restrict__ ps0, size_t NN, int i, int axis, int j) {
    const double v = ps0[(size_t)axis * NN + i];
    return axis == j - 1 ? v + kEps : v;
}

static __global__ void __launch_bounds__(128) k_stm_orbits(int N, const double *__restrict__ ps0, const int *__restrict__ npts,
                                                    int nmax, double *__restrict__ opos, double *__restrict__ ovel) {
    const size_t NN = N;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < 7 * NN; t += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(t % NN), j = (int)(t / NN);
        Orbit o;
        o.x = stm_start(ps0, NN, i, 0, j); o.y = stm_start(ps0, NN, i, 1, j); o.z = stm_start(ps0, NN, i, 2, j);
        o.vx = stm_start(ps0, NN, i, 3, j); o.vy = stm_start(ps0, NN, i, 4, j); o.vz = stm_start(ps0, NN, i, 5, j);
        o.init();
        const int n = npts ? npts[i] : nmax;
        constexpr double dt = -kStepMyr / kSub, h = 0.5 * dt;
        for (int k = 0; k < n; k++) {
            if (k > 0) {
#pragma unroll 1
                for (int s = 0; s < kSub; s++) o.kdk(dt, h);
            }
            double *p = opos + (size_t)(k * 7 + j) * 3 * NN + i;
            p[0] = o.x; p[NN] = o.y; p[2 * NN] = o.z;
            if (j == 0) {
                double *v = ovel + (size_t)k * 3 * NN + i;
                v[0] = o.vx; v[NN] = o.vy; v[2 * NN] = o.vz;
            }
        }
    }
}

// The same orbits on four lanes each (quad_accel: the same bits), 8 orbits per warp, one warp per block.  For objects few
// enough that every warp has a scheduler to itself: a step is then 34 FP64 warp instructions in a row where one lane
// per orbit takes 68, at 64 cycles each with the SM's other schedulers idle.
static __global__ void __launch_bounds__(32) k_stm_orbits_quad(int N, const double *__restrict__ ps0,
                                                               const int *__restrict__ npts, int nmax,
                                                               double *__restrict__ opos, double *__restrict__ ovel) {
    const size_t NN = N, t = (size_t)blockIdx.x * 8 + (threadIdx.x >> 2);
    const int role = threadIdx.x & 3, c = role < 3 ? role : 2;
    const bool mine = t < 7 * NN;
    const size_t u = mine ? t : 7 * NN - 1;                   // lanes past the end repeat the last orbit
    const int i = (int)(u % NN), j = (int)(u / NN);
    QuadOrbit o;
    o.q = role < 3 ? stm_start(ps0, NN, i, c, j) : 0.0;
    o.v = role < 3 ? stm_start(ps0, NN, i, 3 + c, j) : 0.0;
    o.init(role);
    const int n = npts ? npts[i] : nmax, nw = __reduce_max_sync(0xffffffffu, n);
    constexpr double dt = -kStepMyr / kSub, h = 0.5 * dt;
    for (int k = 0; k < nw; k++) {
        if (k > 0) {
#pragma unroll 1
            for (int s = 0; s < kSub; s++) o.kdk(dt, h, role);
        }
        if (mine && role < 3 && k < n) {
            opos[((size_t)(k * 7 + j) * 3 + c) * NN + i] = o.q;
            if (j == 0) ovel[((size_t)k * 3 + c) * NN + i] = o.v;
        }
    }
}

// Four lanes per orbit while 7 N orbits at 8 a warp leave each scheduler at most one warp (694 objects on 152 SMs): 1 star
// 4.7 -> 2.96 ms, 301 stars 4.8 -> 3.01 ms.  Beyond, a scheduler would issue 2 x 34 instructions a step for 16 orbits where
// one lane per orbit issues 68 for 32.  There, blocks of one warp while the warps are fewer than the schedulers, so that
// they spread over the SMs (four schedulers share a pipe that serves each at 76 cycles an instruction, three at 64):
// 2,000 stars 5.3 -> 4.8 ms.  max_blocks > 0: a grid of that many blocks of 128 at most, to run beside other work.
cudaError_t launch_stm_orbits(cudaStream_t st, int sms, int N, const double *ps0, const int *npts, int nmax, double *opos,
                              double *ovel, int max_blocks) {
    const long orbits = 7L * N, warps = (orbits + 31) / 32;
    if (max_blocks <= 0 && orbits <= 8L * 4 * sms) {
        k_stm_orbits_quad<<<(unsigned)((orbits + 7) / 8), 32, 0, st>>>(N, ps0, npts, nmax, opos, ovel);
    } else {
        const int threads = max_blocks <= 0 && warps <= 4L * sms ? 32 : 128;
        long g = (orbits + threads - 1) / threads;
        if (max_blocks > 0) g = std::min(g, (long)max_blocks);
        k_stm_orbits<<<(unsigned)g, threads, 0, st>>>(N, ps0, npts, nmax, opos, ovel);
    }
    return cudaGetLastError();
}

// sig21: the 21 distinct entries of the symmetric 6x6 Sigma0, [21][N], upper triangle row by row
__global__ void __launch_bounds__(256) k_stm_cov(int N, int nmax, const int *__restrict__ npts,
                                                 const double *__restrict__ opos, const double *__restrict__ ovel,
                                                 const double *__restrict__ sig21, double *__restrict__ t64,
                                                 float4 *__restrict__ t32, float *__restrict__ lm) {
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t NN = N;
    if (idx >= NN * nmax) return;
    const int i = (int)(idx % NN), k = (int)(idx / NN);
    if (npts && k >= npts[i]) return;
    const double *P = opos + (size_t)k * 21 * NN + i;
    const double x0 = P[0], y0 = P[NN], z0 = P[2 * NN];
    double A[3][6];
#pragma unroll
    for (int j = 0; j < 6; j++) {
        const double *Q = P + (size_t)(j + 1) * 3 * NN;
        A[0][j] = (Q[0] - x0) * 1e5;
        A[1][j] = (Q[NN] - y0) * 1e5;
        A[2][j] = (Q[2 * NN] - z0) * 1e5;
    }
    double sg[6][6];
    {
        int q = 0;
#pragma unroll
        for (int a = 0; a < 6; a++)
#pragma unroll
            for (int b = a; b < 6; b++) { sg[a][b] = sg[b][a] = sig21[(size_t)q * NN + i]; q++; }
    }
    double AS[3][6];
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int b = 0; b < 6; b++) {
            double acc = 0.0;
#pragma unroll
            for (int a = 0; a < 6; a++) acc = fma(A[r][a], sg[a][b], acc);
            AS[r][b] = acc;
        }
    double S[6];
    const int rr[6] = {0, 0, 0, 1, 1, 2}, ss[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
    for (int q = 0; q < 6; q++) {
        double acc = 0.0;
#pragma unroll
        for (int b = 0; b < 6; b++) acc = fma(AS[rr[q]][b], A[ss[q]][b], acc);
        S[q] = acc;
    }
    const double *V = ovel + (size_t)k * 3 * NN + i;
    double *T = t64 + (size_t)k * 12 * NN + i;
    const double vals[12] = {x0, y0, z0, V[0], V[NN], V[2 * NN], S[0], S[1], S[2], S[3], S[4], S[5]};
#pragma unroll
    for (int f = 0; f < 12; f++) T[(size_t)f * NN] = vals[f];
    const float hx = (float)x0, hy = (float)y0, hz = (float)z0;
    float4 *o = t32 + ((size_t)k * NN + i) * 3;
    o[0] = make_float4(hx, hy, hz, (float)(x0 - (double)hx));
    o[1] = make_float4((float)(y0 - (double)hy), (float)(z0 - (double)hz), (float)S[0], (float)S[1]);
    o[2] = make_float4((float)S[2], (float)S[3], (float)S[4], (float)S[5]);
    // lower bound on lambda_min(S), rounded down to FP32, for the mixed-precision filter's error bounds
    const double l = sym3_min_eig_lb(S[0], S[1], S[2], S[3], S[4], S[5]);
    lm[(size_t)k * NN + i] = __double2float_rd(l - 1e-12 * fabs(l));
}

// ---------------------------------------------------------------------------------------------------------------
// clone Monte Carlo

// |v| in FP32 (components already in FP32), bounded from below (lo) or above (hi): the approximate square root is
// within a few ulp, and the 1e-6 margins cover it; outside 1e-18 <= |v| <= 1e18 the bounds are 0 and +inf
__device__ __forceinline__ float norm32_rsqrt(float q) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(q));
    return r;
}
__device__ __forceinline__ float norm32_lo(float x, float y, float z) {
    const float q = fmaf(x, x, fmaf(y, y, z * z));
    return q >= 1e-36f && q <= 1e36f ? q * norm32_rsqrt(q) * (1.f - 1e-6f) : 0.f;
}
__device__ __forceinline__ float norm32_hi(float x, float y, float z) {
    const float q = fmaf(x, x, fmaf(y, y, z * z));
    return q >= 1e-36f && q <= 1e36f ? q * norm32_rsqrt(q) * (1.f + 1e-6f) : __int_as_float(0x7f800000);
}

// One clone traced back: the target's and the cluster's orbit, the closest approach so far (reference
// ph_pair_clone and seg_min, src/phygas.c:147-156, 200-216).  Results in kpc, Myr, kpc/Myr.
//
// Each step's segment r0 -> r1 first gets an FP32 lower bound on its distance from the origin: every point of it is
// within |r1 - r0| / 2 of r0 or of r1, so none is nearer than min(|r0|, |r1|) - |r1 - r0| / 2.  The separations in
// FP32 are truncated (never above |r|) and the FP32 norms carry 1e-6 margins; when the bound exceeds the closest
// approach so far (an upper bound of it in FP32, with an absolute margin for the FP64 path's own rounding), the
// segment cannot improve it and the FP64 segment test is skipped.  Otherwise the reference's test runs as before,
// so the results are the same bits -- and the FP64 pipe does that work only near the closest approach.
struct Nearest {
    double r0x, r0y, r0z, best, tbest, vbest;
    float f0x, f0y, f0z, n0, best_up;          // r0 truncated to FP32, |r0| from below, best from above
    __device__ __forceinline__ void set_best_up() { best_up = fmaf(f32_trunc(best), 1.f + 2.4e-7f, 1e-37f); }
    // r0 = the separation, (ux, uy, uz) the relative velocity at the start
    __device__ __forceinline__ void start(double rx, double ry, double rz, double ux, double uy, double uz) {
        r0x = rx; r0y = ry; r0z = rz;
        best = sqrt(fma(r0x, r0x, fma(r0y, r0y, r0z * r0z)));
        tbest = 0.0;
        vbest = sqrt(fma(ux, ux, fma(uy, uy, uz * uz)));
        f0x = f32_trunc(r0x); f0y = f32_trunc(r0y); f0z = f32_trunc(r0z);
        n0 = norm32_lo(f0x, f0y, f0z);
        set_best_up();
    }
    // step i (1-based) of length dt (negative) has ended at separation r1; vel() = the relative speed there
    template <class Vel>
    __device__ __forceinline__ void segment(int i, double dt, double r1x, double r1y, double r1z, const Vel &vel) {
        const float f1x = f32_trunc(r1x), f1y = f32_trunc(r1y), f1z = f32_trunc(r1z);
        const float n1 = norm32_lo(f1x, f1y, f1z);
        const float dn = fmaf(2.2e-7f, n0 + n1, norm32_hi(f1x - f0x, f1y - f0y, f1z - f0z));
        const float lb = (fminf(n0, n1) - 0.5f * dn) * (1.f - 1e-6f) - 1e-12f * (n0 + n1);
        if (!(lb > best_up)) {
            // the reference's segment test (seg_min and its strict comparison), with its own cheap pre-test
            const double dx = r1x - r0x, dy = r1y - r0y, dz = r1z - r0z;
            const double dd = fma(dx, dx, fma(dy, dy, dz * dz));
            const double an = fma(r0x, dx, fma(r0y, dy, r0z * dz));
            const double r0s = fma(r0x, r0x, fma(r0y, r0y, r0z * r0z));
            const double r1s = fma(r1x, r1x, fma(r1y, r1y, r1z * r1z));
            const double best2 = best * best;
            double near2dd;
            if (!(dd > 0) || an >= 0) near2dd = r0s * dd;
            else if (-an >= dd) near2dd = r1s * dd;
            else near2dd = fma(r0s, dd, -an * an);
            if (near2dd < best2 * dd * (1.0 + 1e-12) || (!(dd > 0) && r0s < best2 * (1.0 + 1e-12))) {
                double s = 0.0;
                if (dd > 0) {
                    s = -an / dd;
                    s = s < 0.0 ? 0.0 : (s > 1.0 ? 1.0 : s);
                }
                const double mx = fma(dx, s, r0x), my = fma(dy, s, r0y), mz = fma(dz, s, r0z);
                const double dm = sqrt(fma(mx, mx, fma(my, my, mz * mz)));
                if (dm < best) {
                    best = dm;
                    tbest = ((double)(i - 1) + s) * -dt;
                    vbest = vel();
                    set_best_up();
                }
            }
        }
        r0x = r1x; r0y = r1y; r0z = r1z;
        f0x = f1x; f0y = f1y; f0z = f1z;
        n0 = n1;
    }
};

// A clone's closest approach: distance (kpc), time (Myr), speed (kpc/Myr)
struct Approach {
    double best, tbest, vbest;
};

// One clone per lane in FP64, one orbit after the other.
__device__ __noinline__ Approach trace_clone64(const double *__restrict__ ps, int steps, double dt) {
    Orbit a, b;
    a.x = ps[0]; a.y = ps[1]; a.z = ps[2]; a.vx = ps[3]; a.vy = ps[4]; a.vz = ps[5];
    b.x = ps[6]; b.y = ps[7]; b.z = ps[8]; b.vx = ps[9]; b.vy = ps[10]; b.vz = ps[11];
    a.init();
    b.init();
    Nearest n;
    n.start(a.x - b.x, a.y - b.y, a.z - b.z, a.vx - b.vx, a.vy - b.vy, a.vz - b.vz);
    const double h = 0.5 * dt;
#pragma unroll 1
    for (int i = 1; i <= steps; i++) {
        a.kdk(dt, h);
        b.kdk(dt, h);
        n.segment(i, dt, a.x - b.x, a.y - b.y, a.z - b.z, [&]() {
            const double wx = a.vx - b.vx, wy = a.vy - b.vy, wz = a.vz - b.vz;
            return sqrt(fma(wx, wx, fma(wy, wy, wz * wz)));
        });
    }
    return Approach{n.best, n.tbest, n.vbest};
}

// Four clones by a warp in FP64, eight lanes each (the same bits): lanes 0-3 of the eight trace the target, 4-7 the cluster
// (quad_accel).  ps, steps and dt are the eight's clone's; every lane of the warp calls.  A step takes 34 FP64 instructions
// where trace_clone64 takes 136, so up to three such passes end sooner.
__device__ __noinline__ Approach trace_clone64_eights(const double *__restrict__ ps, int steps, double dt) {
    const unsigned all = 0xffffffffu, eight = 0xffu << (threadIdx.x & 24u);
    const int role = threadIdx.x & 3, c = role < 3 ? role : 2;
    const double *p = ps + (threadIdx.x & 4 ? 6 : 0);
    QuadOrbit o;
    o.q = role < 3 ? p[c] : 0.0;
    o.v = role < 3 ? p[3 + c] : 0.0;
    o.init(role);
    Nearest n;
    // component k of the target's orbit less the cluster's, on each of the lanes m (the warp's, or one eight's)
    auto diff = [&](unsigned m, double v, int k) { return __shfl_sync(m, v, k, 8) - __shfl_sync(m, v, 4 + k, 8); };
    n.start(diff(all, o.q, 0), diff(all, o.q, 1), diff(all, o.q, 2), diff(all, o.v, 0), diff(all, o.v, 1),
            diff(all, o.v, 2));
    const double h = 0.5 * dt;
    const int most = __reduce_max_sync(all, steps);
#pragma unroll 1
    for (int i = 1; i <= most; i++) {
        o.kdk(dt, h, role);
        const double x = diff(all, o.q, 0), y = diff(all, o.q, 1), z = diff(all, o.q, 2);
        if (i <= steps)
            n.segment(i, dt, x, y, z, [&]() {
                const double wx = diff(eight, o.v, 0), wy = diff(eight, o.v, 1), wz = diff(eight, o.v, 2);
                return sqrt(fma(wx, wx, fma(wy, wy, wz * wz)));
            });
    }
    return Approach{n.best, n.tbest, n.vbest};
}

// ---- the clone on the FP32 and integer units (pgx_orbit32.cuh) -----------------------------------------------------
// Two orbits of about 340 instructions a step and 50 for the closest approach: bound by the issue rate, where the FP64
// clone above is bound by the FP64 pipe at 141.6 instructions x 19 cycles per SM a clone-step.  1,024 pulsar pairs x
// 1,000 clones: 3.55e10 clone-steps/s against 3.5e9; 64 pairs x 200 clones x 400 steps, where a warp's latency counts,
// 1.1 against 8.4 ms.  FP64 stays for orbits outside its range and for ties (segment64).
//
// The closest approach over the steps' segments r0 -> r1 = r0 + d (exact integer differences of the positions) is the
// reference's, with most segments decided from float estimates of r1.d and r1.r1:
//   receding   r0.d > 0 for certain: the segment's nearest point is r0, which the segment before has counted;
//   approaching r1.d < 0 for certain: the nearest point is r1.  When it improves on the best for certain it becomes the
//              record without being evaluated ("pending"): while the pair keeps approaching, each next r1 is nearer
//              still.  It is evaluated when the approach ends there;
//   otherwise  (a minimum inside the step, a few per clone, or an undecided sign) the reference's test in FP64.
// The float errors, in units of a position's high word (2^-23 kpc): each component of r1 and d is within 2^-23 relative
// or 2^-24 absolute, so with |r1|, |d| > 8 r1.d is within 2^-21.3 |r1||d| and r0.d = r1.d - d.d within 2^-21.3 (|r1||d| +
// d.d); both signs are certain where the square exceeds 2^-40 d.d (r1.r1 + d.d).  Squared distances are compared with a
// relative margin of 2^-19.  Shorter vectors (10^-6 kpc) take the FP64 test.
constexpr float kSure2 = 0x1p-40f, kSureUp = 1.f + 0x1p-19f, kSureDown = 1.f - 0x1p-19f, kSureMin = 64.f;

struct I3 {
    long long x, y, z;
};
__device__ __forceinline__ I3 operator-(const I3 &a, const I3 &b) { return I3{a.x - b.x, a.y - b.y, a.z - b.z}; }
// in units of the high word, within 2^-23 relative
__device__ __forceinline__ float fixed_to_f32(long long v) {
    return fmaf((float)(unsigned)v, 0x1p-32f, (float)(int)(v >> 32));
}
__device__ __forceinline__ double norm64(const I3 &v) {
    const double x = (double)v.x, y = (double)v.y, z = (double)v.z;
    return sqrt(fma(x, x, fma(y, y, z * z)));
}

// The segment test of step i (1-based) in FP64: r1, d = r1 - r0 in position units of u kpc, v2 = twice the relative
// displacement at the step's end in units of 2 uv kpc.  at_r0: the best is at r0 and unevaluated.  r0's distance is
// counted already: only a point beyond it can improve (s > 0).
//
// A minimum within a hair of an end of its step: the reference compares the two steps' distances, which differ by less
// than FP64 resolves, and which of them is the record (the time is the same, the speed is that at the end of the
// record's step) is decided by the rounding of its FP64 orbits.  *tie = the step after which the FP64 trace decides it
// (kTie: seven roundings of 2^-53, as a relative difference of the distances, doubled for squares).
constexpr double kTie = 0x1p-50;
enum { kSegNone, kSegBest, kSegAtR0 };

__device__ __noinline__ int segment64(const I3 r1, const I3 d, const I3 v2, int i, double dt, double u, double uv,
                                      bool at_r0, Approach &b, int *tie) {
    const double dx = (double)d.x, dy = (double)d.y, dz = (double)d.z;
    const I3 r0 = r1 - d;
    const double rx = (double)r0.x, ry = (double)r0.y, rz = (double)r0.z;
    const double dd = fma(dx, dx, fma(dy, dy, dz * dz)), an = fma(rx, dx, fma(ry, dy, rz * dz));
    const int none = at_r0 ? kSegAtR0 : kSegNone;
    if (!(dd > 0) || !(an < 0)) return none;
    const double s = fmin(-an / dd, 1.0);
    const double mx = fma(dx, s, rx), my = fma(dy, s, ry), mz = fma(dz, s, rz);
    const double m2 = fma(mx, mx, fma(my, my, mz * mz)), dm = sqrt(m2) * u;
    const bool hair = at_r0 ? s < 1.0 && an * an < kTie * dd * m2 : fabs(dm - b.best) < kTie * dm;
    if (!at_r0 && !hair && !(dm < b.best)) return none;
    *tie = s < 1.0 && (an + dd) * (an + dd) < kTie * dd * m2 ? i + 1 : (hair ? i : 0);
    b.best = dm;
    b.tbest = ((double)(i - 1) + s) * -dt;
    b.vbest = norm64(v2) * uv / fabs(dt);
    return kSegBest;
}

// 2^-55 and 2^-62 kpc in the scale's units: of positions, and half that of displacements
__device__ __forceinline__ double unit64(const OrbitScale &s) { return pow2(s.e - 55); }
__device__ __forceinline__ double half_unit64(const OrbitScale &s) { return pow2(s.e - s.k - 62); }
__device__ __forceinline__ Acc64i mw_accel32(const Force32 &K, const OrbitScale &s, double dt, float near2, long long x,
                                             long long y, long long z, float &r2) {
    return orbit32_accel<MwModel32>(K, HaloTable32(), MwNear(), s, dt, near2, x, y, z, r2);
}

// The record at the end of step i: both orbits there, their displacements those of the next drift
__device__ __noinline__ Approach vertex64(const Orbit32 a, const Orbit32 b, const Force32 K, const OrbitScale s, int i,
                                          double dt) {
    float r2;
    const float near2 = orbit32_near2(dt);
    const Acc64i A = mw_accel32(K, s, dt, near2, a.x, a.y, a.z, r2), B = mw_accel32(K, s, dt, near2, b.x, b.y, b.z, r2);
    const I3 v2 = {2 * (a.wx - b.wx) - (A.x - B.x), 2 * (a.wy - b.wy) - (A.y - B.y),
                   2 * (a.wz - b.wz) - (A.z - B.z)};                 // 2 v dt = 2 w - a dt^2
    return Approach{norm64(I3{a.x - b.x, a.y - b.y, a.z - b.z}) * unit64(s), (double)i * -dt,
                    norm64(v2) * half_unit64(s) / fabs(dt)};
}

// The closest approach so far, from the float estimates of each step
struct Near32 {
    Approach r;
    float q;                 // r.best^2 in squared high-word units
    int tie;                 // > 0: the record is a tie that the FP64 trace of this many steps decides
    bool pend;
    __device__ __forceinline__ void set_q(const OrbitScale &s) {
        const float f = (float)(r.best * __hiloint2double((1023 + 23 - s.e) << 20, 0));
        q = f * f;
    }
    __device__ __forceinline__ void start(const double *p, const OrbitScale &s) {
        const double rx = p[0] - p[6], ry = p[1] - p[7], rz = p[2] - p[8];
        const double ux = p[3] - p[9], uy = p[4] - p[10], uz = p[5] - p[11];
        r = Approach{sqrt(fma(rx, rx, fma(ry, ry, rz * rz))), 0.0, sqrt(fma(ux, ux, fma(uy, uy, uz * uz)))};
        pend = false;
        tie = 0;
        set_q(s);
    }
    // a step's dd = d.d, q1 = r1.r1, b1 = r1.d, where nothing has to be evaluated: receding with nothing pending, approaching
    // outside the best, or approaching with a pending record.  false: step() on the same
    __device__ __forceinline__ bool quick(float dd, float q1, float b1) {
        const float a0 = b1 - dd;
        const float t = fminf(dd, q1) > kSureMin ? kSure2 * dd * (q1 + dd) : __int_as_float(0x7f800000);
        const bool away = a0 > 0.f && a0 * a0 > t, in = !away && b1 < 0.f && b1 * b1 > t;
        const bool go = in && (pend || q1 * kSureUp < q);
        if (go) {
            pend = true;
            tie = 0;
            q = q1;
        }
        return go || (!pend && (away || (in && !(q1 * kSureDown <= q))));
    }
    // segment(at_r0) runs segment64 on it, vertex() the record at its start
    template <class Segment, class Vertex>
    __device__ __forceinline__ void step(float dd, float q1, float b1, const OrbitScale &s, const Segment &segment,
                                         const Vertex &vertex) {
        const float a0 = b1 - dd;
        const float t = fminf(dd, q1) > kSureMin ? kSure2 * dd * (q1 + dd) : __int_as_float(0x7f800000);
        if (a0 > 0.f && a0 * a0 > t) {
            if (!pend) return;
            r = vertex();                                     // the approach ended at r0
        } else {
            const bool in = b1 < 0.f && b1 * b1 > t;
            if (in && (pend || q1 * kSureUp < q)) {
                pend = true;
                tie = 0;
                q = q1;
                return;
            }
            if (!(in ? q1 * kSureDown <= q : (pend || could_improve(q1, fmaf(-2.f, b1, q1 + dd), dd)))) return;
            if (segment(pend, r, &tie) == kSegAtR0) r = vertex();
        }
        pend = false;
        set_q(s);
    }
    // whether a segment between squared distances q0 and q1 can come nearer than the best: no point of it is nearer
    // than the nearer end less its length
    __device__ __forceinline__ bool could_improve(float q1, float q0, float dd) const {
        const float m = fmaxf(fminf(fmaf(-0x1p-18f, q1 + dd, q0), q1), 0.f);
        const float lb = sqrtf(m) * kSureDown - sqrtf(dd) * kSureUp;
        return !(fminf(dd, q1) > kSureMin && lb > 0.f && lb * lb * kSureDown > q);
    }
};

__device__ __forceinline__ bool in_range32(float ra, float rb, float rmax) {
    return fmaxf(ra, rb) < rmax && fminf(ra, rb) > kOrbit32MinR2;
}

// the scale of a clone's two orbits (false: none, NaN and infinities included)
__device__ __forceinline__ bool clone_scale(const double *p, int steps, double dt, OrbitScale &s) {
    double va, vb, sum = 0.0;
    const double ra = orbit32_reach(p, p + 3, steps, dt, va), rb = orbit32_reach(p + 6, p + 9, steps, dt, vb);
#pragma unroll
    for (int j = 0; j < 12; j++) sum += p[j];                 // fmax passes over NaN
    return fabs(sum) < 1e300 && orbit32_start_ok(p) && orbit32_start_ok(p + 6) &&
           orbit32_units(fmax(ra, rb), fmax(va, vb), dt, s);
}

// A step that floats alone do not settle: near the centre, or one whose segment or record is evaluated.  Out of line, its data
// through memory, so that the loop's registers are the common step's (1 x 20,000 clones 2.72 -> 2.53 ms, 300 x 1,000 17.5 -> 16.7).
struct SlowStep {
    Orbit32 a, b;            // drifted, not yet kicked
    I3 sa, sb;               // their drifts
    Acc64i A, B;             // their accelerations
    Force32 K;
    OrbitScale s;
    Near32 n;
    float ra, rb, near2, dd, q1, b1;
    bool done;               // the closest approach needs nothing
};
// false: an orbit too close to the centre
__device__ __noinline__ bool slow_step(SlowStep &t, int i, double dt) {
    if (t.ra < t.near2) t.A = mw_accel_near(t.K, t.s, dt, t.a.x, t.a.y, t.a.z);            // (as orbit32_accel)
    if (t.rb < t.near2) t.B = mw_accel_near(t.K, t.s, dt, t.b.x, t.b.y, t.b.z);
    if (!(fminf(t.ra, t.rb) > kOrbit32MinR2)) return false;
    if (t.done) return true;
    t.n.step(t.dd, t.q1, t.b1, t.s,
             [&](bool at_r0, Approach &r, int *tie) {
                 const Orbit32 &a = t.a, &b = t.b;
                 const I3 v2 = {2 * (a.wx - b.wx) + (t.A.x - t.B.x), 2 * (a.wy - b.wy) + (t.A.y - t.B.y),
                                2 * (a.wz - b.wz) + (t.A.z - t.B.z)};
                 return segment64(I3{a.x - b.x, a.y - b.y, a.z - b.z}, t.sa - t.sb, v2, i, dt, unit64(t.s),
                                  half_unit64(t.s), at_r0, r, tie);
             },
             [&]() {
                 Orbit32 a0 = t.a, b0 = t.b;
                 a0.x -= t.sa.x; a0.y -= t.sa.y; a0.z -= t.sa.z;
                 b0.x -= t.sb.x; b0.y -= t.sb.y; b0.z -= t.sb.z;
                 return vertex64(a0, b0, t.K, t.s, i - 1, dt);
             });
    return true;
}

struct Clone32 {
    Orbit32 a, b;
    Force32 K;
    OrbitScale s;
    Near32 n;
    float rmax, near2;       // r2 limits
    bool ok;
    // false: not an orbit for these units, or FP64 asked for (traced in FP64)
    __device__ __forceinline__ bool start(const double *__restrict__ ps, int steps, double dt, bool fp64) {
        double p[12];
#pragma unroll
        for (int j = 0; j < 12; j++) p[j] = ps[j];
        n.pend = false;
        n.tie = 0;
        near2 = orbit32_near2(dt);
        ok = !fp64 && clone_scale(p, steps, dt, s);
        if (!ok) {                                            // (stepped along where its lane has another clone)
            a = b = Orbit32{};
            K = Force32{};
            s = OrbitScale{0x1p-23f, 0};
            rmax = near2 = 0.f;
            return false;
        }
        K = force32_constants<MwModel32>(dt, s);
        rmax = orbit32_max_r2(s);
        float ra, rb;
        auto accel = [&](long long x, long long y, long long z, float &r2) {
            return mw_accel32(K, s, dt, near2, x, y, z, r2);
        };
        orbit32_start(a, accel, s, p, p + 3, dt, ra);
        orbit32_start(b, accel, s, p + 6, p + 9, dt, rb);
        ok = in_range32(ra, rb, rmax);
        n.start(p, s);
        return true;
    }
    __device__ __forceinline__ void step(int i, double dt) {
        const int sh = 6 + s.k;
        const I3 sa = {orbit32_drift(a.wx, sh), orbit32_drift(a.wy, sh), orbit32_drift(a.wz, sh)};
        const I3 sb = {orbit32_drift(b.wx, sh), orbit32_drift(b.wy, sh), orbit32_drift(b.wz, sh)};
        a.x += sa.x; a.y += sa.y; a.z += sa.z;
        b.x += sb.x; b.y += sb.y; b.z += sb.z;
        float ra, rb;
        const HaloTable32 T;
        Acc64i A = accel32<MwModel32>(K, T, s.c, a.x, a.y, a.z, ra), B = accel32<MwModel32>(K, T, s.c, b.x, b.y, b.z, rb);
        const I3 d = sa - sb, r1 = {a.x - b.x, a.y - b.y, a.z - b.z};
        const float dx = fixed_to_f32(d.x), dy = fixed_to_f32(d.y), dz = fixed_to_f32(d.z);
        const float rx = fixed_to_f32(r1.x), ry = fixed_to_f32(r1.y), rz = fixed_to_f32(r1.z);
        const float dd = fmaf(dx, dx, fmaf(dy, dy, dz * dz)), q1 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
        const float b1 = fmaf(rx, dx, fmaf(ry, dy, rz * dz));
        ok = ok && fmaxf(ra, rb) < rmax;
        const bool near = fminf(ra, rb) < near2, done = n.quick(dd, q1, b1);
        if (ok && (near || !done)) {
            SlowStep t = {a, b, sa, sb, A, B, K, s, n, ra, rb, near2, dd, q1, b1, done};
            ok = slow_step(t, i, dt);
            A = t.A;
            B = t.B;
            n = t.n;
        }
        a.wx += A.x; a.wy += A.y; a.wz += A.z;
        b.wx += B.x; b.wy += B.y; b.wz += B.z;
    }
    // after the last step: the approach may still be on
    __device__ __forceinline__ void finish(int steps, double dt) {
        if (n.pend) n.r = vertex64(a, b, K, s, steps, dt);
    }
    // the steps the FP64 trace takes for this clone's record (0: none, the record stands)
    __device__ __forceinline__ int fp64_steps(int steps) const { return ok ? min(n.tie, steps) : max(steps, 1); }
};

// orbit32_accel on four lanes (every lane of the warp calls)
__device__ __forceinline__ long long quad_step_accel(const F3 &k, const OrbitScale &s, double dt, float near2, long long x,
                                                     int role, float &r2) {
    long long a = quad_accel32(k, s.c, x, role, r2);
    if (__any_sync(0xffffffffu, r2 < near2)) {
        const long long f = quad_accel_near(k, s, dt, x, role);
        if (r2 < near2) a = f;
    }
    return a;
}

// The same clone on eight lanes (quad_accel32: target on lanes 0-3 of the eight, cluster on 4-7): the same bits.
struct QuadClone32 {
    long long x, w;          // the lane's coordinate and displacement
    F3 k;
    OrbitScale s;
    Near32 n;                // alike on the eight lanes
    float rmax, near2;
    bool ok;
    __device__ __forceinline__ static unsigned group() { return 0xffu << (threadIdx.x & 24u); }
    // lanes 0, 1, 2 of the eight hold the target's v, lanes 4, 5, 6 the cluster's: the differences, on every lane
    __device__ __forceinline__ static I3 diff3(long long v) {
        const unsigned m = group();
        const long long d = v - __shfl_xor_sync(m, v, 4);
        return I3{__shfl_sync(m, d, 0, 8), __shfl_sync(m, d, 1, 8), __shfl_sync(m, d, 2, 8)};
    }
    __device__ __forceinline__ static Orbit32 gather(long long x, long long w, int o) {
        const unsigned m = group();
        return Orbit32{__shfl_sync(m, x, o, 8), __shfl_sync(m, x, o + 1, 8), __shfl_sync(m, x, o + 2, 8),
                       __shfl_sync(m, w, o, 8), __shfl_sync(m, w, o + 1, 8), __shfl_sync(m, w, o + 2, 8)};
    }
    __device__ __forceinline__ Approach vertex(long long x0, int i, double dt) const {
        const Orbit32 a = gather(x0, w, 0), b = gather(x0, w, 4);
        return vertex64(a, b, force32_constants<MwModel32>(dt, s), s, i, dt);
    }
    __device__ __forceinline__ void start(const double *__restrict__ ps, int steps, double dt, int role, bool fp64) {
        double p[12];
#pragma unroll
        for (int j = 0; j < 12; j++) p[j] = ps[j];
        near2 = orbit32_near2(dt);
        ok = !fp64 && clone_scale(p, steps, dt, s);
        if (!ok) {                                            // (traced along with its warp, and again in FP64)
            s = OrbitScale{0x1p-23f, 0};
            near2 = 0.f;
        }
        k = quad_constant(force32_constants<MwModel32>(ok ? dt : 0.05, s), role);
        rmax = orbit32_max_r2(s);
        const int o = threadIdx.x & 4 ? 6 : 0;
        const double q = role == 0 ? ps[o] : (role == 1 ? ps[o + 1] : ps[o + 2]);
        const double v = role == 0 ? ps[o + 3] : (role == 1 ? ps[o + 4] : ps[o + 5]);
        x = ok && role < 3 ? f64_to_i64(q * pow2(55 - s.e)) : 0;
        float r2;
        const long long a = quad_step_accel(k, s, dt, near2, x, role, r2);
        w = (ok && role < 3 ? displacement(v, dt, pow2(61 - s.e + s.k)) + a / 2 : 0) + (1LL << (5 + s.k));
        const float rb = __shfl_xor_sync(0xffffffffu, r2, 4);        // (every lane, whatever its ok)
        ok = ok && in_range32(r2, rb, rmax);
        n.start(p, s);
    }
    __device__ __forceinline__ void step(int i, double dt, int role) {
        const unsigned all = 0xffffffffu;
        const long long sw = orbit32_drift(w, 6 + s.k);
        x += sw;
        float r2;
        long long a = quad_accel32(k, s.c, x, role, r2);
        const float rb = __shfl_xor_sync(all, r2, 4);                 // (every lane, whatever its ok)
        const float fd = fixed_to_f32(sw - __shfl_xor_sync(all, sw, 4)), fr = fixed_to_f32(x - __shfl_xor_sync(all, x, 4));
        const float dx = __shfl_sync(all, fd, 0, 8), dy = __shfl_sync(all, fd, 1, 8), dz = __shfl_sync(all, fd, 2, 8);
        const float rx = __shfl_sync(all, fr, 0, 8), ry = __shfl_sync(all, fr, 1, 8), rz = __shfl_sync(all, fr, 2, 8);
        const float dd = fmaf(dx, dx, fmaf(dy, dy, dz * dz)), q1 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
        const float b1 = fmaf(rx, dx, fmaf(ry, dy, rz * dz));
        ok = ok && fmaxf(r2, rb) < rmax;
        const bool near = fminf(r2, rb) < near2, done = n.quick(dd, q1, b1);
        if (__any_sync(all, ok && (near || !done))) {
            if (__any_sync(all, ok && near)) {                        // (as orbit32_accel)
                const long long m = quad_accel_near(k, s, dt, x, role);
                if (ok && r2 < near2) a = m;
                ok = ok && fminf(r2, rb) > kOrbit32MinR2;
            }
            if (ok && !done)
                n.step(dd, q1, b1, s,
                       [&](bool at_r0, Approach &r, int *tie) {
                           return segment64(diff3(x), diff3(sw), diff3(2 * w + a), i, dt, unit64(s), half_unit64(s), at_r0,
                                            r, tie);
                       },
                       [&]() { return vertex(x - sw, i - 1, dt); });
        }
        w += a;
    }
    __device__ __forceinline__ void finish(int steps, double dt) {
        if (n.pend) n.r = vertex(x, steps, dt);
    }
    __device__ __forceinline__ int fp64_steps(int steps) const { return ok ? min(n.tie, steps) : max(steps, 1); }
};

// Coarse tracks of the prefilter (reference track, src/phygas.c:98-111): the nominal orbit of each object from ps
// (6 doubles per object); pos[k][3][N] = the position after 10 k KDK steps of -0.05 Myr, for k < npts[i].  On the FP32
// and integer units, four lanes per orbit (quad_accel32), one warp per block: a few to a few thousand orbits, whose steps'
// latency is the time.  Orbits outside the units' range are traced again in FP64 (quad_accel).  The tracks of 3 pulsars and
// their pair tests: 4.7 -> 0.8 ms.
static __global__ void __launch_bounds__(32) k_coarse_tracks(int N, const double *__restrict__ ps,
                                                             const int *__restrict__ npts, double *__restrict__ pos) {
    const unsigned all = 0xffffffffu;
    const size_t NN = N;
    const int t = blockIdx.x * 8 + (threadIdx.x >> 2), role = threadIdx.x & 3, c = role < 3 ? role : 2;
    const int i = min(t, N - 1);                              // lanes past the end repeat the last orbit
    const bool mine = t < N && role < 3;
    const double *q = ps + 6 * (size_t)i;
    const int n = npts[i], nw = __reduce_max_sync(all, n);
    constexpr double dt = -kStepMyr / kSub, h = 0.5 * dt;
    double p12[12];
#pragma unroll
    for (int j = 0; j < 6; j++) p12[j] = p12[6 + j] = q[j];
    OrbitScale s;
    float near2 = orbit32_near2(dt);
    bool ok = clone_scale(p12, (n - 1) * kSub, dt, s);
    if (!ok) {
        s = OrbitScale{0x1p-23f, 0};
        near2 = 0.f;
    }
    const F3 k = quad_constant(force32_constants<MwModel32>(dt, s), role);
    const float rmax = orbit32_max_r2(s);
    const double unit = unit64(s);
    long long x = ok && role < 3 ? f64_to_i64(q[c] * pow2(55 - s.e)) : 0;
    float r2;
    const long long a0 = quad_step_accel(k, s, dt, near2, x, role, r2);
    ok = ok && in_range32(r2, r2, rmax);
    long long w = (ok && role < 3 ? displacement(q[3 + c], dt, pow2(61 - s.e + s.k)) + a0 / 2 : 0) + (1LL << (5 + s.k));
    for (int j = 0; j < nw; j++) {
        if (j > 0) {
#pragma unroll 1
            for (int m = 0; m < kSub; m++) {
                x += orbit32_drift(w, 6 + s.k);
                w += quad_step_accel(k, s, dt, near2, x, role, r2);
                ok = ok && (j >= n || in_range32(r2, r2, rmax));
            }
        }
        if (mine && j < n) pos[((size_t)j * 3 + c) * NN + i] = j ? (double)x * unit : q[c];
    }
    if (!__any_sync(all, !ok)) return;
    QuadOrbit o;
    o.q = role < 3 ? q[c] : 0.0;
    o.v = role < 3 ? q[3 + c] : 0.0;
    o.init(role);
    for (int j = 0; j < nw; j++) {
        if (j > 0) {
#pragma unroll 1
            for (int m = 0; m < kSub; m++) o.kdk(dt, h, role);
        }
        if (mine && !ok && j < n) pos[((size_t)j * 3 + c) * NN + i] = o.q;
    }
}

cudaError_t launch_coarse_tracks(cudaStream_t st, int N, const double *ps, const int *npts, double *pos) {
    if (N <= 0) return cudaSuccess;
    k_coarse_tracks<<<(N + 7) / 8, 32, 0, st>>>(N, ps, npts, pos);
    return cudaGetLastError();
}

// The clones of a warp that take the FP64 trace: n steps of each lane's clone (0: none; every lane calls).  Up to twelve are
// traced four at a time (3 x 34 FP64 instructions a step at most), more lane by lane (136).  One after the other, as it was,
// 10 pairs x 400 clones at steps of 0.2 Myr took 8.5 ms, four at a time 2.3.
__device__ __forceinline__ void trace_fp64(const double *ps, int n, int steps, double dt, Approach &r) {
    const unsigned all = 0xffffffffu;
    unsigned m = __ballot_sync(all, n > 0);
    if (__popc(m) > 12) {
        if (n > 0) r = trace_clone64(ps, min(n, steps), dt);
        return;
    }
    const int lane = threadIdx.x & 31;
    while (m) {
        // the eights take the next four set lanes' clones (with fewer left, the others repeat the first)
        int src = __ffs(m) - 1;
        unsigned left = m;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (k == lane >> 3 && left) src = __ffs(left) - 1;
            left &= left - 1u;
        }
        const unsigned long long p = __shfl_sync(all, (unsigned long long)ps, src);
        const Approach x = trace_clone64_eights((const double *)p, __shfl_sync(all, min(n, steps), src),
                                                __shfl_sync(all, dt, src));
        const int k = __popc(m & ((1u << lane) - 1u)), from = 8 * min(k, 3);
        const Approach y = {__shfl_sync(all, x.best, from), __shfl_sync(all, x.tbest, from), __shfl_sync(all, x.vbest, from)};
        if ((m >> lane & 1u) && k < 4) r = y;
        m = left;
    }
}

// a lane's clone (every lane of the warp calls; active: it has one)
__device__ __forceinline__ Approach trace_clone(bool active, const double *__restrict__ ps, int steps, double dt) {
    Clone32 c;
    c.ok = c.n.pend = false;
    c.n.tie = 0;
    if (active && c.start(ps, steps, dt, false)) {
#pragma unroll 1
        for (int i = 1; i <= steps; i++) c.step(i, dt);
    }
    if (active && c.ok) c.finish(steps, dt);
    __syncwarp();
    trace_fp64(ps, active ? c.fp64_steps(steps) : 0, steps, dt, c.n.r);
    return c.n.r;
}

// ---- reduction of one pair (m clones) ---------------------------------------------------------------------------
// All sorted quantities are non-negative doubles, whose IEEE bit patterns order like their values, so the sort
// runs on 64-bit integer keys (the integer pipe; a double compare would occupy the scarce FP64 pipe).
__device__ __forceinline__ unsigned long long kmin(unsigned long long a, unsigned long long b) { return a < b ? a : b; }
__device__ __forceinline__ unsigned long long kmax(unsigned long long a, unsigned long long b) { return a < b ? b : a; }

// bitonic sort of 32*R keys held by one warp, element e = 32*r + lane in register r: stages whose partner distance
// j is below 32 exchange across lanes with shuffles, the others swap registers within a lane
template <int R>
__device__ __forceinline__ void warp_bitonic(unsigned long long (&a)[R], int lane) {
#pragma unroll
    for (int k = 2; k <= 32 * R; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= 32) {
                const int jr = j >> 5;
#pragma unroll
                for (int r = 0; r < R; r++) {
                    if (r & jr) continue;
                    const bool asc = ((32 * r) & k) == 0;
                    const unsigned long long lo = kmin(a[r], a[r | jr]), hi = kmax(a[r], a[r | jr]);
                    a[r] = asc ? lo : hi;
                    a[r | jr] = asc ? hi : lo;
                }
            } else {
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const unsigned long long p = __shfl_xor_sync(0xffffffffu, a[r], j);
                    const bool asc = ((32 * r + lane) & k) == 0, lower = (lane & j) == 0;
                    a[r] = (asc == lower) ? kmin(a[r], p) : kmax(a[r], p);
                }
            }
        }
    }
}

// linear-interpolated quantile of a sorted array (reference quantile, src/phygas.c:175-180), without contraction
__device__ __forceinline__ double interp_q(const double *v, int n, double q) {
    const double pos = __dmul_rn(q, (double)(n - 1));
    const int i = (int)pos;
    if (i >= n - 1) return v[n - 1];
    return __dadd_rn(v[i], __dmul_rn(__dsub_rn(pos, (double)i), __dsub_rn(v[i + 1], v[i])));
}

// one warp reduces one pair: cres holds best/tbest/vbest of its m clones (m <= 32*R)
template <int R>
__device__ void warp_reduce_pair(const double *__restrict__ best, const double *__restrict__ tbest,
                                 const double *__restrict__ vbest, int m, double r50_pc, double rtot_pc,
                                 double *smem_w, PhResultDev *out, int lane) {
    unsigned long long a[R];
    int in50 = 0, intot = 0;
    double res[9];
#pragma unroll 1
    for (int which = 0; which < 3; which++) {
        const double *src = which == 0 ? best : (which == 1 ? tbest : vbest);
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int e = 32 * r + lane;
            double v = 0.0;
            if (e < m) {
                v = __ldcg(src + e);
                if (which == 0) {
                    v = __dmul_rn(v, 1000.0);
                    in50 += v < r50_pc;
                    intot += v < rtot_pc;
                } else if (which == 2) {
                    v = __dmul_rn(v, kKms);
                }
            }
            a[r] = e < m ? (unsigned long long)__double_as_longlong(v) : 0x7ff0000000000000ULL;
        }
        warp_bitonic<R>(a, lane);
#pragma unroll
        for (int r = 0; r < R; r++) smem_w[32 * r + lane] = __longlong_as_double((long long)a[r]);
        __syncwarp();
        if (lane == 0) {
            res[3 * which + 0] = interp_q(smem_w, m, 0.05);
            res[3 * which + 1] = interp_q(smem_w, m, 0.5);
            res[3 * which + 2] = interp_q(smem_w, m, 0.95);
        }
        __syncwarp();
    }
    in50 = __reduce_add_sync(0xffffffffu, in50);
    intot = __reduce_add_sync(0xffffffffu, intot);
    if (lane == 0) {
        PhResultDev o;
        o.n = m;
        o.pad = 0;
        o.d05 = res[0]; o.d50 = res[1]; o.d95 = res[2];
        o.t05 = res[3]; o.t50 = res[4]; o.t95 = res[5];
        o.v05 = res[6]; o.v50 = res[7]; o.v95 = res[8];
        o.f_r50 = m > 0 ? __ddiv_rn((double)in50, (double)m) : 0.0;
        o.f_rtot = m > 0 ? __ddiv_rn((double)intot, (double)m) : 0.0;
        if (m <= 0) { o.d05 = o.d50 = o.d95 = o.t05 = o.t50 = o.t95 = o.v05 = o.v50 = o.v95 = 0.0; }
        *out = o;
    }
}

__device__ void reduce_dispatch(const McPairs &P, int p, double *smem_w, int lane) {
    const int m = P.clone_off[p + 1] - P.clone_off[p];
    const size_t o = P.clone_off[p];
    const double *b = P.cres + o, *t = P.cres + P.n_clones + o, *v = P.cres + 2 * (size_t)P.n_clones + o;
    PhResultDev *out = P.res + p;
    const double r50 = P.r50_pc[p], rt = P.rtot_pc[p];
    if (m <= 32) warp_reduce_pair<1>(b, t, v, m, r50, rt, smem_w, out, lane);
    else if (m <= 64) warp_reduce_pair<2>(b, t, v, m, r50, rt, smem_w, out, lane);
    else if (m <= 128) warp_reduce_pair<4>(b, t, v, m, r50, rt, smem_w, out, lane);
    else if (m <= 256) warp_reduce_pair<8>(b, t, v, m, r50, rt, smem_w, out, lane);
    else if (m <= 512) warp_reduce_pair<16>(b, t, v, m, r50, rt, smem_w, out, lane);
    else warp_reduce_pair<32>(b, t, v, m, r50, rt, smem_w, out, lane);
}

// A warp's first item goes by its place in the grid, the next ones by the queue (k_mc_prep sets its head past the first
// ones).  With all of them from the queue, the SMs whose warps came first took a small batch's items for themselves, 16
// warps where others had none: 1 pair x 20,000 clones took 3.4 to 4.4 ms, spread out 2.2 ms.
__device__ __forceinline__ int first_item() { return blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); }
__device__ __forceinline__ int next_item(const McPairs &P) {
    int q = 0;
    if ((threadIdx.x & 31) == 0) q = atomicAdd(P.qhead, 1);
    return __shfl_sync(0xffffffffu, q, 0);
}

// Persistent clone tracing for batches replayed from a captured graph: parameters read from device memory, and the
// launch shape a template: WARPS warps per block, CPL clones per lane traced in lockstep (items of up to 32 * CPL
// clones; a lane past its item's end repeats another clone and discards the copy), and MINB resident blocks per SM
// asked of the compiler (fewer registers per thread, more warps to hide the FP64 pipe's latency).  Tracing only -- the pairs are
// reduced by k_pair_reduce_dev afterwards, which keeps this kernel's registers to the orbits'.  The clones'
// arithmetic is the same in every variant, so every variant gives the same bits.
template <int WARPS, int CPL, int MINB>
__global__ void __launch_bounds__(WARPS * 32, MINB > 1 ? MINB : 16 / (WARPS * CPL)) k_pair_mc_t(const McPairs *__restrict__ Pd) {
    const McPairs P = *Pd;
    const int lane = threadIdx.x & 31;
    for (int q = first_item(); q < P.n_items; q = next_item(P)) {
        const int4 it = P.items[q];   // x = pair, y = first clone, z = count
        const int p = it.x;
        const int steps = P.steps[p];
        const double dt = P.dt[p];
        Clone32 c[CPL];
        bool any = false;
#pragma unroll
        for (int j = 0; j < CPL; j++) {
            const int e = lane + 32 * j < it.z ? lane + 32 * j : min(lane, it.z - 1);
            any |= c[j].start(P.ps + (size_t)(it.y + e) * 12, steps, dt, P.fp64 != 0);
        }
        if (any) {
#pragma unroll 1
            for (int i = 1; i <= steps; i++) {
#pragma unroll
                for (int j = 0; j < CPL; j++) c[j].step(i, dt);
            }
        }
#pragma unroll
        for (int j = 0; j < CPL; j++) {
            const bool mine = lane + 32 * j < it.z;
            const int cc = it.y + (mine ? lane + 32 * j : 0);
            if (c[j].ok) c[j].finish(steps, dt);
            __syncwarp();
            trace_fp64(P.ps + (size_t)cc * 12, mine ? c[j].fp64_steps(steps) : 0, steps, dt, c[j].n.r);
            if (!mine) continue;
            P.cres[cc] = c[j].n.r.best;
            P.cres[P.n_clones + cc] = c[j].n.r.tbest;
            P.cres[2 * (size_t)P.n_clones + cc] = c[j].n.r.vbest;
        }
    }
}

// The same with eight lanes per clone, items of up to four clones: for batches of few clones, where a step's latency
// counts (kMcQuadClones).
__global__ void __launch_bounds__(kMcQuadWarps * 32) k_pair_mc_quad(const McPairs *__restrict__ Pd) {
    const McPairs P = *Pd;
    const int lane = threadIdx.x & 31, role = threadIdx.x & 3, e = lane >> 3;
    for (int q = first_item(); q < P.n_items; q = next_item(P)) {
        const int4 it = P.items[q];   // x = pair, y = first clone, z = count
        const int p = it.x, steps = P.steps[p], cc = it.y + min(e, it.z - 1);
        const double dt = P.dt[p];
        QuadClone32 c;
        c.start(P.ps + (size_t)cc * 12, steps, dt, role, P.fp64 != 0);
        if (__any_sync(0xffffffffu, c.ok)) {
#pragma unroll 1
            for (int i = 1; i <= steps; i++) c.step(i, dt, role);
        }
        if (c.ok) c.finish(steps, dt);
        __syncwarp();
        const bool mine = (lane & 7) == 0 && e < it.z;
        trace_fp64(P.ps + (size_t)cc * 12, mine ? c.fp64_steps(steps) : 0, steps, dt, c.n.r);
        if (!mine) continue;
        P.cres[cc] = c.n.r.best;
        P.cres[P.n_clones + cc] = c.n.r.tbest;
        P.cres[2 * (size_t)P.n_clones + cc] = c.n.r.vbest;
    }
}

// before k_pair_mc_t: queue head past the first items of its warps, empty results for pairs without clones
__global__ void k_mc_prep(const McPairs *__restrict__ Pd, int warps) {
    const McPairs P = *Pd;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t == 0) *P.qhead = warps;
    for (int p = t; p < P.n_pairs; p += gridDim.x * blockDim.x) {
        if (P.clone_off[p + 1] - P.clone_off[p] > 0) continue;
        PhResultDev o;
        o.n = 0;
        o.pad = 0;
        o.d05 = o.d50 = o.d95 = o.t05 = o.t50 = o.t95 = o.v05 = o.v50 = o.v95 = o.f_r50 = o.f_rtot = 0.0;
        P.res[p] = o;
    }
}

// after k_pair_mc_t: one warp per pair of 1 .. 1024 clones, over a fixed grid
__global__ void __launch_bounds__(kMcThreads) k_pair_reduce_dev(const McPairs *__restrict__ Pd) {
    __shared__ double smem[kMcThreads / 32][1024];
    const McPairs P = *Pd;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int p = blockIdx.x * (kMcThreads / 32) + w; p < P.n_pairs; p += gridDim.x * (kMcThreads / 32)) {
        const int m = P.clone_off[p + 1] - P.clone_off[p];
        if (m > 0 && m <= 1024) reduce_dispatch(P, p, smem[w], lane);
    }
}

namespace {
struct McVariant {
    int warps, cpl, min_blocks;
    void (*fn)(const McPairs *);
};
// the last entry: eight lanes per clone (not one of the tuner's shapes)
const McVariant kMcVariants[] = {
    {4, 1, 1, k_pair_mc_t<4, 1, 1>}, {2, 1, 1, k_pair_mc_t<2, 1, 1>}, {8, 1, 1, k_pair_mc_t<8, 1, 1>},
    {4, 2, 1, k_pair_mc_t<4, 2, 1>}, {2, 2, 1, k_pair_mc_t<2, 2, 1>}, {8, 2, 1, k_pair_mc_t<8, 2, 1>},
    {4, 1, 5, k_pair_mc_t<4, 1, 5>}, {4, 1, 6, k_pair_mc_t<4, 1, 6>}, {8, 1, 3, k_pair_mc_t<8, 1, 3>},
    {kMcQuadWarps, 0, 1, k_pair_mc_quad},
};
}  // namespace

int mc_variants() { return (int)(sizeof kMcVariants / sizeof kMcVariants[0]) - 1; }
int mc_quad_variant() { return mc_variants(); }

void mc_variant_shape(int v, int &warps, int &cpl, int &min_blocks) {
    warps = kMcVariants[v].warps;
    cpl = kMcVariants[v].cpl;
    min_blocks = kMcVariants[v].min_blocks;
}

// resident blocks of variant v for a full persistent grid (blocks per SM x SMs)
cudaError_t mc_variant_grid(int v, int sms, int &grid) {
    int per_sm = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &per_sm, reinterpret_cast<const void *>(kMcVariants[v].fn), kMcVariants[v].warps * 32, 0);
    grid = sms * (per_sm > 0 ? per_sm : 1);
    return e;
}

// prep, trace (variant v on a persistent grid) and reduce on one stream; reduce_grid blocks of kMcThreads
cudaError_t launch_mc(int v, int grid, int prep_grid, int reduce_grid, cudaStream_t st, const McPairs *Pd) {
    k_mc_prep<<<prep_grid, 256, 0, st>>>(Pd, grid * kMcVariants[v].warps);
    kMcVariants[v].fn<<<grid, kMcVariants[v].warps * 32, 0, st>>>(Pd);
    k_pair_reduce_dev<<<reduce_grid, kMcThreads, 0, st>>>(Pd);
    return cudaGetLastError();
}

// reduction alone, one warp per pair, for results traced elsewhere (the drop-in ph_pair_reduce)
__global__ void __launch_bounds__(kMcThreads) k_pair_reduce_only(McPairs P) {
    __shared__ double smem[kMcThreads / 32][1024];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int p = blockIdx.x * (kMcThreads / 32) + w;
    if (p >= P.n_pairs) return;
    const int m = P.clone_off[p + 1] - P.clone_off[p];
    if (m > 0 && m <= 1024) reduce_dispatch(P, p, smem[w], lane);
}

// A pair's clone value e of array `which` (0 best, 1 tbest, 2 vbest) in the units of the reduction, as the bit
// pattern that orders it: the values are non-negative, so their IEEE patterns sort as unsigned integers.
__device__ __forceinline__ unsigned long long reduce_key(const double *src, int which, int e) {
    double v = src[e];
    if (which == 0) v = __dmul_rn(v, 1000.0);
    else if (which == 2) v = __dmul_rn(v, kKms);
    return (unsigned long long)__double_as_longlong(v);
}

// Order statistics of a pair's m values of array `which`, read from global memory by the whole block: an MSB radix
// selection of all kRanks ranks (rank[r], 0-based) at once, 8 bits a pass, starting below the bits that all values share.
// A pass counts the values under each prefix that some rank still follows; a warp per rank then finds its digit.  Exact:
// the elements that a sort would put there.  For pairs too large to sort in shared memory: 20,000 values in about 9
// passes, where a selection per rank and array in turn, a digit found by one thread, read them 144 times (1.86 ms).
constexpr int kRanks = 6, kReduceThreads = 1024;
__device__ void radix_select(const double *src, int which, int m, const int *rank, double *value) {
    __shared__ unsigned hist[kRanks][256];
    __shared__ unsigned long long s_prefix[kRanks], s_min, s_max;
    __shared__ int s_left[kRanks], s_group[kRanks];             // rank within its prefix; the first rank of its prefix
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (tid == 0) { s_min = ~0ull; s_max = 0; }
    __syncthreads();
    unsigned long long lo = ~0ull, hi = 0;
    for (int e = tid; e < m; e += blockDim.x) {
        const unsigned long long key = reduce_key(src, which, e);
        lo = kmin(lo, key);
        hi = kmax(hi, key);
    }
    for (int o = 16; o > 0; o >>= 1) {
        lo = kmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = kmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if (lane == 0) { atomicMin(&s_min, lo); atomicMax(&s_max, hi); }
    __syncthreads();
    const int top = s_min == s_max ? 0 : 64 - __clzll((long long)(s_min ^ s_max));      // bits that differ
    unsigned long long mask = top == 64 ? 0ull : ~0ull << top;
    if (tid < kRanks) { s_prefix[tid] = s_min & mask; s_left[tid] = rank[tid]; }
    __syncthreads();
    for (int shift = top - 8; mask != ~0ull; shift -= 8) {
        const int sh = shift > 0 ? shift : 0;                    // the last pass takes the bits that are left
        const unsigned long long digits = ~mask & (~0ull << sh);
        if (tid < kRanks) {
            int g = 0;
            while (s_prefix[g] != s_prefix[tid]) g++;
            s_group[tid] = g;
        }
        for (int b = tid; b < kRanks * 256; b += blockDim.x) (&hist[0][0])[b] = 0;
        __syncthreads();
        for (int e = tid; e < m; e += blockDim.x) {
            const unsigned long long key = reduce_key(src, which, e), pre = key & mask;
            const unsigned d = (unsigned)((key & digits) >> sh);
#pragma unroll
            for (int g = 0; g < kRanks; g++)
                if (s_group[g] == g && pre == s_prefix[g]) atomicAdd(&hist[g][d], 1u);
        }
        __syncthreads();
        if (w < kRanks) {                                        // warp w: rank w's digit, 8 bins a lane
            const unsigned *h = hist[s_group[w]] + 8 * lane;
            int c[8], sum = 0;
#pragma unroll
            for (int b = 0; b < 8; b++) { c[b] = (int)h[b]; sum += c[b]; }
            int before = sum;
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, before, o);
                if (lane >= o) before += t;
            }
            before -= sum;
            const int k = s_left[w];
            const unsigned long long prefix = s_prefix[w];
            __syncwarp();
            if (k >= before && k < before + sum) {
                int b = 0;
                for (int left = k - before; left >= c[b]; b++) left -= c[b];
                for (int q = 0; q < b; q++) before += c[q];
                s_left[w] = k - before;
                s_prefix[w] = prefix | (unsigned long long)(8 * lane + b) << sh;
            }
        }
        mask |= digits;
        __syncthreads();
    }
    if (tid < kRanks) value[tid] = __longlong_as_double((long long)s_prefix[tid]);
    __syncthreads();
}

// Pairs of more than 1024 clones (and the empty result of pairs without clones), a block per pair and array: sorted in
// shared memory up to kSortMax clones (launched with room for the batch's largest such pair), beyond that by radix
// selection from global memory.
__global__ void __launch_bounds__(kReduceThreads) k_pair_reduce_big(McPairs P) {
    extern __shared__ double sm[];
    const int p = blockIdx.x / 3, which = blockIdx.x % 3;
    const int m = P.clone_off[p + 1] - P.clone_off[p];
    if (m > 0 && m <= 1024) return;
    PhResultDev *out = P.res + p;
    double *quant = which == 0 ? &out->d05 : (which == 1 ? &out->t05 : &out->v05);
    if (m <= 0) {
        if (threadIdx.x == 0) {
            quant[0] = quant[1] = quant[2] = 0.0;
            if (which == 0) { out->n = 0; out->pad = 0; out->f_r50 = out->f_rtot = 0.0; }
        }
        return;
    }
    const size_t o = P.clone_off[p];
    const double *src = P.cres + (size_t)which * P.n_clones + o;
    if (which == 0) {
        __shared__ int c50, ctot;
        if (threadIdx.x == 0) { c50 = 0; ctot = 0; }
        __syncthreads();
        const double r50 = P.r50_pc[p], rtot = P.rtot_pc[p];
        int l50 = 0, ltot = 0;
        for (int e = threadIdx.x; e < m; e += blockDim.x) {
            const double v = __dmul_rn(src[e], 1000.0);
            l50 += v < r50;
            ltot += v < rtot;
        }
        l50 = __reduce_add_sync(0xffffffffu, l50);
        ltot = __reduce_add_sync(0xffffffffu, ltot);
        if ((threadIdx.x & 31) == 0) { atomicAdd(&c50, l50); atomicAdd(&ctot, ltot); }
        __syncthreads();
        if (threadIdx.x == 0) {
            out->n = m;
            out->pad = 0;
            out->f_r50 = __ddiv_rn((double)c50, (double)m);
            out->f_rtot = __ddiv_rn((double)ctot, (double)m);
        }
    }
    if (m > kSortMax) {
        __shared__ int rank[kRanks];
        __shared__ double value[kRanks];
        if (threadIdx.x < 3) {
            const double pos = __dmul_rn(threadIdx.x == 0 ? 0.05 : (threadIdx.x == 1 ? 0.5 : 0.95), (double)(m - 1));
            const int i = min((int)pos, m - 1);
            rank[2 * threadIdx.x] = i;
            rank[2 * threadIdx.x + 1] = min(i + 1, m - 1);
        }
        __syncthreads();
        radix_select(src, which, m, rank, value);
        if (threadIdx.x < 3) {
            const double pos = __dmul_rn(threadIdx.x == 0 ? 0.05 : (threadIdx.x == 1 ? 0.5 : 0.95), (double)(m - 1));
            const int i = (int)pos;
            const double a = value[2 * threadIdx.x], b = value[2 * threadIdx.x + 1];
            quant[threadIdx.x] = i >= m - 1 ? a : __dadd_rn(a, __dmul_rn(__dsub_rn(pos, (double)i), __dsub_rn(b, a)));
        }
        return;
    }
    int n2 = 1;
    while (n2 < m) n2 <<= 1;
    unsigned long long *key = reinterpret_cast<unsigned long long *>(sm);
    for (int e = threadIdx.x; e < n2; e += blockDim.x) key[e] = e < m ? reduce_key(src, which, e) : 0x7ff0000000000000ULL;
    __syncthreads();
    for (int k = 2; k <= n2; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int h = threadIdx.x; h < n2 / 2; h += blockDim.x) {
                const int e = ((h & ~(j - 1)) << 1) | (h & (j - 1)), f = e | j;      // the pair of h in this stage
                const unsigned long long x = key[e], y = key[f];
                const bool asc = (e & k) == 0;
                if ((x > y) == asc) { key[e] = y; key[f] = x; }
            }
            __syncthreads();
        }
    if (threadIdx.x < 3)
        quant[threadIdx.x] = interp_q(reinterpret_cast<const double *>(key), m,
                                      threadIdx.x == 0 ? 0.05 : (threadIdx.x == 1 ? 0.5 : 0.95));
}

// sort_max: the most clones of a pair of the batch that is sorted (at most kSortMax)
cudaError_t launch_pair_reduce_big(cudaStream_t st, const McPairs &P, int sort_max) {
    size_t n2 = 1;
    while (n2 < (size_t)sort_max) n2 <<= 1;
    const size_t smem = sort_max > 1024 ? n2 * 8 : 0;         // (allowed for up to kSortMax clones by orbit_setup)
    k_pair_reduce_big<<<3 * P.n_pairs, kReduceThreads, smem, st>>>(P);
    return cudaGetLastError();
}

}  // namespace pgx

namespace pgx {
// Peak-rate probes for the roofline denominators (FP64 and FP32 are not in the driver's measured peaks): long
// independent FMA chains, 8 per thread; the result is stored so nothing is eliminated.
__global__ void k_peak_dfma(double *out, int iters, double a, double b) {
    double x[8];
#pragma unroll
    for (int i = 0; i < 8; i++) x[i] = threadIdx.x * 1e-3 + i;
    for (int it = 0; it < iters; it++)
#pragma unroll
        for (int i = 0; i < 8; i++) x[i] = fma(x[i], a, b);
    double s = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) s += x[i];
    out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}
__global__ void k_peak_ffma(float *out, int iters, float a, float b) {
    float x[8];
#pragma unroll
    for (int i = 0; i < 8; i++) x[i] = threadIdx.x * 1e-3f + i;
    for (int it = 0; it < iters; it++)
#pragma unroll
        for (int i = 0; i < 8; i++) x[i] = fmaf(x[i], a, b);
    float s = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) s += x[i];
    out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}
}  // namespace pgx

// ---------------------------------------------------------------------------------------------------------------
// pgx_pair_noalloc: the pair Monte Carlo for callers that cannot allocate GPU memory.
//
// Some callers may not call cudaMalloc at all: code that runs inside another framework's memory pool (the pool
// owns the device memory and a stray allocation fragments it or fails), real-time loops that must not stall on the
// allocator, and host code that hands this library only the device buffers it already has.  This entry point takes
// the caller's device buffers for inputs and outputs and keeps its own scratch -- the per-clone closest approaches
// and the work-queue head -- in a fixed array compiled into the library (static __device__ storage, held by every
// GPU that loads the library until the process exits).  It calls no allocating routine.
//
// Limits: at most kNoAllocMaxClones clones per call (24 MiB of scratch); pairs of more than 1024 clones get a result
// with n = -1 (pgx_pair handles them), and so does a pair whose offsets leave [0, n_clones).  Every call shares the
// one scratch array and leaves its contents behind; two calls whose work overlaps on the GPU (different streams, or
// different host threads) race on it and must be serialised by the caller.  The first call on a device runs the
// set-up below, which fills the force tables with a kernel on the legacy default stream and synchronizes the whole
// device: make it before any stream capture, and outside latency-critical work.
namespace pgx {

constexpr int kNoAllocMaxClones = 1 << 20;

// per-clone results: best (kpc), tbest (Myr), vbest (kpc/Myr), each kNoAllocMaxClones long
static __device__ __align__(256) double g_noalloc_cres[3 * kNoAllocMaxClones];
// work-queue head (cleared at the start of every call)
static __device__ __align__(256) int g_noalloc_qhead[64];

// persistent: warps take chunks of 32 consecutive clones; a lane finds its clone's pair by binary search
__global__ void __launch_bounds__(kMcThreads) k_pair_mc_noalloc(int n_pairs, int n_clones,
                                                                const int *__restrict__ clone_off,
                                                                const double *__restrict__ ps,
                                                                const int *__restrict__ steps,
                                                                const double *__restrict__ dt, double *cres, int *qhead) {
    const int lane = threadIdx.x & 31;
    const int n_chunks = (n_clones + 31) / 32;
    for (;;) {
        int q = 0;
        if (lane == 0) q = atomicAdd(qhead, 1);
        q = __shfl_sync(0xffffffffu, q, 0);
        if (q >= n_chunks) break;
        const int c = q * 32 + lane;
        int lo = 0, hi = n_pairs;              // clone_off[lo] <= c < clone_off[hi]
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (clone_off[mid] <= c) lo = mid; else hi = mid;
        }
        const Approach r = trace_clone(c < n_clones, ps + (size_t)c * 12, steps[lo], dt[lo]);
        if (c < n_clones) {
            cres[c] = r.best;
            cres[kNoAllocMaxClones + c] = r.tbest;
            cres[2 * (size_t)kNoAllocMaxClones + c] = r.vbest;
        }
    }
}

// one warp per pair, after all clones are traced (stream order).  The offsets are device memory the host cannot
// check: a pair whose clones do not lie inside [0, n_clones) -- the clones this call traced -- gets n = -1 instead
// of reading scratch the call did not write (or memory past it).
__global__ void __launch_bounds__(kMcThreads) k_pair_reduce_noalloc(int n_pairs, int n_clones,
                                                                    const int *__restrict__ clone_off,
                                                                    const double *__restrict__ r50,
                                                                    const double *__restrict__ rt,
                                                                    const double *cres, PhResultDev *res) {
    __shared__ double smem[kMcThreads / 32][1024];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int p = blockIdx.x * (kMcThreads / 32) + w;
    if (p >= n_pairs) return;
    const int o = clone_off[p], e = clone_off[p + 1];
    const bool bad = o < 0 || e < o || e > n_clones;
    const int m = bad ? -1 : e - o;
    if (m <= 0 || m > 1024) {
        if (lane == 0) {
            PhResultDev z;
            z.n = m == 0 ? 0 : -1;
            z.pad = 0;
            z.d05 = z.d50 = z.d95 = z.t05 = z.t50 = z.t95 = z.v05 = z.v50 = z.v95 = z.f_r50 = z.f_rtot = 0.0;
            res[p] = z;
        }
        return;
    }
    const double *b = cres + o, *t = cres + kNoAllocMaxClones + o, *v = cres + 2 * (size_t)kNoAllocMaxClones + o;
    if (m <= 32) warp_reduce_pair<1>(b, t, v, m, r50[p], rt[p], smem[w], res + p, lane);
    else if (m <= 64) warp_reduce_pair<2>(b, t, v, m, r50[p], rt[p], smem[w], res + p, lane);
    else if (m <= 128) warp_reduce_pair<4>(b, t, v, m, r50[p], rt[p], smem[w], res + p, lane);
    else if (m <= 256) warp_reduce_pair<8>(b, t, v, m, r50[p], rt[p], smem[w], res + p, lane);
    else if (m <= 512) warp_reduce_pair<16>(b, t, v, m, r50[p], rt[p], smem[w], res + p, lane);
    else warp_reduce_pair<32>(b, t, v, m, r50[p], rt[p], smem[w], res + p, lane);
}

namespace {
// set-up, once per device: the device addresses of the scratch arrays (in host code their names are host-side
// stand-ins, not device addresses) and the persistent grid size
struct NoAllocDevice {
    double *cres = nullptr;
    int *qhead = nullptr;
    int grid = 0;
    bool ready = false;
};
NoAllocDevice g_noalloc_dev[64];
std::mutex g_noalloc_mu;

int noalloc_setup(int dev, NoAllocDevice *&out) {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    NoAllocDevice &d = g_noalloc_dev[dev];
    if (!d.ready) {
        cudaError_t e = orbit_setup(dev) ? cudaErrorUnknown : cudaSuccess;
        if (e == cudaSuccess) e = cudaGetSymbolAddress((void **)&d.cres, g_noalloc_cres);
        if (e == cudaSuccess) e = cudaGetSymbolAddress((void **)&d.qhead, g_noalloc_qhead);
        int sms = 0, per_sm = 0;
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pair_mc_noalloc, kMcThreads, 0);
        if (e != cudaSuccess) {
            fprintf(stderr, "pgx_pair_noalloc: set-up on device %d failed: %s\n", dev, cudaGetErrorString(e));
            return PGX_E_CUDA;
        }
        d.grid = sms * (per_sm > 0 ? per_sm : 1);
        d.ready = true;
    }
    out = &d;
    return 0;
}
}  // namespace
}  // namespace pgx

extern "C" int pgx_pair_noalloc(void *stream, int n_pairs, int n_clones, const int *clone_off, const double *ps,
                                const int *steps, const double *dt, const double *r50_pc, const double *rtot_pc,
                                PhResult *res) {
    if (n_pairs < 0 || n_clones < 0 || (n_pairs > 0 && (!clone_off || !steps || !dt || !r50_pc || !rtot_pc || !res)) ||
        (n_clones > 0 && !ps)) {
        fprintf(stderr, "pgx_pair_noalloc: invalid arguments\n");
        return PGX_E_ARG;
    }
    if (n_clones > pgx::kNoAllocMaxClones) {
        fprintf(stderr, "pgx_pair_noalloc: %d clones in one call; its fixed scratch holds %d (use pgx_pair)\n",
                n_clones, pgx::kNoAllocMaxClones);
        return PGX_E_LIMIT;
    }
    if (n_pairs == 0) return 0;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 64) {
        fprintf(stderr, "pgx_pair_noalloc: no current device (%s)\n", cudaGetErrorString(e));
        return PGX_E_NODEV;
    }
    pgx::NoAllocDevice *d = nullptr;
    int rc = pgx::noalloc_setup(dev, d);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    e = cudaMemsetAsync(d->qhead, 0, sizeof(int), st);
    if (e == cudaSuccess && n_clones > 0) {
        const int grid = std::max(1, std::min(d->grid, (n_clones + 127) / 128));
        pgx::k_pair_mc_noalloc<<<grid, pgx::kMcThreads, 0, st>>>(n_pairs, n_clones, clone_off, ps, steps, dt,
                                                                  d->cres, d->qhead);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
        const int wpb = pgx::kMcThreads / 32;
        pgx::k_pair_reduce_noalloc<<<(n_pairs + wpb - 1) / wpb, pgx::kMcThreads, 0, st>>>(
            n_pairs, n_clones, clone_off, r50_pc, rtot_pc, d->cres, reinterpret_cast<pgx::PhResultDev *>(res));
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        fprintf(stderr, "pgx_pair_noalloc: launch failed: %s\n", cudaGetErrorString(e));
        return PGX_E_CUDA;
    }
    return 0;
}

namespace pgx {
// The halo power tables of pgx_force.cuh, filled once per device (before the first orbit kernel on it; call it
// outside any stream capture), and the shared memory k_pair_reduce_big may ask for: a limit of the function on the device,
// for every context and thread, so it is set to the most once and not to each launch's own.
int orbit_setup(int dev) {
    static std::mutex mu;
    static bool ready[64] = {};
    if (dev < 0 || dev >= 64) return 1;
    std::lock_guard<std::mutex> lk(mu);
    if (ready[dev]) return 0;
    long long b1, b2;                       // the force compares these bit patterns as integers
    std::memcpy(&b1, &kHaloCut, 8);
    std::memcpy(&b2, &kTinyR2, 8);
    if (b1 != kHaloCutBits || b2 != kTinyR2Bits) return 3;
    k_halo_tables<<<1, kHaloTableThreads>>>();
    k_halo32_table<<<(kHalo32N + 255) / 256, 256>>>();
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_pair_reduce_big, cudaFuncAttributeMaxDynamicSharedMemorySize, kSortMax * 8);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) return 2;
    ready[dev] = true;
    return 0;
}
}  // namespace pgx
