// pgx_force.cuh -- the Allen & Santillan (1991) Milky Way force and the kick-drift-kick step, FP64 (internal header
// of pgx_orbit.cu, which owns the halo power tables and fills them once per device).
#pragma once
#include "pgx_bits.cuh"
#include "pgx_internal.cuh"
#include "pgx_orbit32.cuh"

namespace pgx {

// x^(gamma - 1) of the halo term as x * x^a, a = (gamma - 1) - 1 = 0.02: x = 2^e m, m in [1, 2); m in sub-interval
// j of 1024 with centre c_j, m = c_j (1 + t), |t| <= 2^-11; x^a = 2^(a e) c_j^a (1 + t)^a with the first two from
// tables and (1 + t)^a by its binomial series to t^4 (the next term, |C(a, 5)| t^5 <= 0.0039 2^-55, is below 2^-63
// relative).  Eight FP64 operations and a few integer ones, in place of a log and an exp (about 50 FP64-pipe slots
// on this GPU), and closer: each table entry and the series are within a few ulp, where exp(a' ln x) inherits the
// log's absolute error times |a' ln x|.
constexpr int kPow2Bias = 80, kPow2N = 96, kPowSubLog = 10, kPowSub = 1 << kPowSubLog, kPowTerms = 4;
static __device__ double g_halo_pow2[kPow2N];      // 2^(a e), e = i - kPow2Bias
static __device__ double g_halo_powc[kPowSub];     // c_j^a, c_j = 1 + (2 j + 1) / 2048
static __device__ double g_halo_invc[kPowSub];     // 1 / c_j
static __device__ double g_halo_coef[kPowTerms + 1];   // binomial coefficients C(a, n)

// the tables (one thread per entry; launched once per device, before any kernel that integrates an orbit)
__global__ void k_halo_tables() {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const double a = kHaloG1 - 1.0;
    if (i < kPow2N) g_halo_pow2[i] = exp2(a * (double)(i - kPow2Bias));
    if (i < kPowSub) {
        const double c = 1.0 + (double)(2 * i + 1) / (2.0 * kPowSub);
        g_halo_powc[i] = pow(c, a);
        g_halo_invc[i] = 1.0 / c;
    }
    if (i == 0) {
        double c = 1.0;
        for (int n = 0; n <= kPowTerms; n++) {
            g_halo_coef[n] = c;
            c = c * (a - (double)n) / (double)(n + 1);
        }
    }
}
constexpr int kHaloTableThreads = kPowSub > kPow2N ? kPowSub : kPow2N;

// the same model for the FP32 orbit (pgx_orbit32.cuh): the constants above in floats
struct MwModel32 {
    static constexpr double bulge_GM = kBulgeGM, disk_GM = kDiskGM, halo_GM = kHaloGM, halo_inv_a = kHaloInvA;
    static constexpr double a = kHaloG1 - 1.0, s = -0.5 * a;
    static constexpr float cut2 = (float)(kHaloCut * kHaloCut);
    static constexpr float a1 = split2(s).h, a1l = split2(s).l, c2 = (float)(s * (s - 1) / 2),
                           c3 = (float)(s * (s - 1) * (s - 2) / 6), c4 = (float)(s * (s - 1) * (s - 2) * (s - 3) / 24);
    PGX_HD static constexpr F2 bulge_b2() { return split2(kBulgeB2); }
    PGX_HD static constexpr F2 disk_b2() { return split2(kDiskB2); }
    PGX_HD static constexpr F2 disk_a() { return split2(kDiskA); }
    PGX_HD static constexpr F3 far() { return split3(kHaloFar); }       // cut p / (1 + p), p = (cut / 12)^(1 + a)
};
static __device__ float4 g_halo32[kHalo32N];
struct HaloTable32 {
    __device__ __forceinline__ Halo32 operator()(int n) const {
        const float4 v = __ldg(&g_halo32[n]);
        return Halo32{v.x, v.y, v.z, v.w};
    }
};
__global__ void k_halo32_table() {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= kHalo32N) return;
    const Halo32 h = halo32_entry(n, MwModel32::a, kHaloInvA);
    g_halo32[n] = make_float4(h.i, h.u0, h.u1, h.u2);
}

// x^a for x > 0 normal (here x in [8e-14, 8.4])
__device__ __forceinline__ double halo_pow_a(double x) {
    const long long bits = __double_as_longlong(x);
    int e = (int)((bits >> 52) & 0x7ff) - 1023;
    e = e < -kPow2Bias ? -kPow2Bias : (e > kPow2N - 1 - kPow2Bias ? kPow2N - 1 - kPow2Bias : e);
    const int j = (int)((bits >> (52 - kPowSubLog)) & (kPowSub - 1));
    const double m = __longlong_as_double((bits & 0x000fffffffffffffLL) | 0x3ff0000000000000LL);
    const double t = fma(m, __ldg(&g_halo_invc[j]), -1.0);
    double s = __ldg(&g_halo_coef[kPowTerms]);
#pragma unroll
    for (int n = kPowTerms - 1; n >= 0; n--) s = fma(s, t, __ldg(&g_halo_coef[n]));
    return __ldg(&g_halo_pow2[e + kPow2Bias]) * __ldg(&g_halo_powc[j]) * s;
}

// x^-1/2 and 1/d in FP64 from the FP32 unit's seed and one third-order step (pgx_bits.cuh: within an ulp or two,
// 5 and 3 FP64 operations); an argument outside [2^-125, 2^125) -- none in a force evaluation of a bound orbit --
// takes the library's function instead.
__device__ __forceinline__ double rsqrt_h3(double x) {
    const uint32_t hi = f64_hi(x);
    if (!seed_ok(hi)) return rsqrt(x);
    return rsqrt_refine(x, widen_seed(fast_rsqrt(seed_arg(hi))));
}
__device__ __forceinline__ double rcp_h3(double d) {
    const uint32_t hi = f64_hi(d);
    if (!seed_ok(hi)) return 1.0 / d;
    return rcp_refine(d, widen_seed(__frcp_rn(seed_arg(hi))));
}

// Acceleration of the Milky Way model at (x, y, z), FP64.
//
// Same model as the reference's milkyway_accel (src/potential.c:60-101), written for a GPU whose FP64 pipe is the
// scarce resource: the three pow() and the divisions become the reciprocal square roots and reciprocal above and the
// table power, using
//   (r^2+b^2)^-3/2 = rsqrt(r^2+b^2)^3          (bulge)
//   aR * x / R     = -GM x / D^3                 (disk, the R of the radial force cancels)
//   az(disk)       = -GM z (a + s) / (s D^3), s = sqrt(z^2 + b^2): (a + s) / s = 1 + a / s
//   x^g / (1 + x^(g-1)) = x p / (1 + p), p = x^(g-1) = x * x^(g-2)   (halo)
// Mathematically identical; the last bits differ from glibc's as any libm's do.  59 FP64 operations.
__device__ __forceinline__ void mw_accel(double x, double y, double z, double &ax, double &ay, double &az) {
    const double R2 = fma(x, x, y * y);
    const double r2 = fma(z, z, R2);
    const double ib = rsqrt_h3(r2 + kBulgeB2);
    const double zb2 = fma(z, z, kDiskB2);
    const double iz = rsqrt_h3(zb2);
    const double s = fma(zb2, iz, kDiskA);                      // a + sqrt(z^2 + b^2)
    const double iD = rsqrt_h3(fma(s, s, R2));
    const double fd = -kDiskGM * (iD * iD * iD);
    // r2 > kTinyR2 and min(r, cut) as integer compares of the bit patterns (for doubles >= 0 they order as the values
    // do; a compare or min of doubles would take an FP64-pipe slot): the same selections for every r2 >= 0
    double r, ir;
    if (__double_as_longlong(r2) > kTinyR2Bits) {
        ir = rsqrt_h3(r2);
        r = r2 * ir;
    } else {
        r = 1e-12;
        ir = 1e12;
    }
    const double xh = (__double_as_longlong(r) < kHaloCutBits ? r : kHaloCut) * kHaloInvA;
    const double p = xh * halo_pow_a(xh);              // xh^(gamma - 1)
    const double q = p * rcp_h3(1.0 + p);
    const double fh = -kHaloGM * xh * q * ((ir * ir) * ir);
    const double fr = fma(-kBulgeGM * ib, ib * ib, fh);       // bulge + halo radial terms
    const double g = fr + fd;
    ax = g * x;
    ay = g * y;
    az = z * fma(fd * kDiskA, iz, g);
}

// out of line, for the four-lane step, where it is the rare case (inlined there, 301 stars' orbits took 3.06 ms and not 3.01)
struct Accel {
    double x, y, z;
};
__device__ __noinline__ Accel mw_accel_any(double x, double y, double z) {
    Accel a;
    mw_accel(x, y, z, a.x, a.y, a.z);
    return a;
}

// the FP32 orbit's force near the centre (accel_near), out of line: some steps of few orbits
struct MwBulge64 {
    __device__ __forceinline__ double operator()(double r2) const {
        const double i = rsqrt_h3(r2 + kBulgeB2);
        return (i * i) * (i * -kBulgeGM);
    }
};
__device__ __noinline__ Acc64i mw_accel_near(const Force32 K, const OrbitScale s, double dt, int64_t x, int64_t y, int64_t z) {
    return accel_near<MwModel32>(K, HaloTable32(), MwBulge64(), s, dt, x, y, z);
}
struct MwNear {
    __device__ __forceinline__ Acc64i operator()(const Force32 &K, const OrbitScale &s, double dt, int64_t x, int64_t y,
                                                 int64_t z) const {
        return mw_accel_near(K, s, dt, x, y, z);
    }
};

// One orbit: position, velocity and the acceleration carried over (one force evaluation per step).
struct Orbit {
    double x, y, z, vx, vy, vz, ax, ay, az;
    __device__ __forceinline__ void init() { mw_accel(x, y, z, ax, ay, az); }
    // kick-drift-kick leapfrog (reference body_step, src/phygas.c:91-96).  Two half kicks per step, as the reference
    // rounds them: merging a step's closing kick with the next one's opening kick would save three FP64 operations
    // but moves the last bits of the orbits enough to change printed digits of the reference's published rows.
    __device__ __forceinline__ void kdk(double dt, double h) {
        vx = fma(ax, h, vx); vy = fma(ay, h, vy); vz = fma(az, h, vz);
        x = fma(vx, dt, x); y = fma(vy, dt, y); z = fma(vz, dt, z);
        mw_accel(x, y, z, ax, ay, az);
        vx = fma(ax, h, vx); vy = fma(ay, h, vy); vz = fma(az, h, vz);
    }
};

// mw_accel and the step on four lanes per orbit: the same operations on the same operands, so the same bits, in 34 FP64
// warp instructions executed a step (ncu; 32 in the expressions) instead of 68.  An FP64 warp instruction costs the same with one lane active or 32, so where
// there are fewer orbits than the schedulers can use lanes, an orbit's independent operations go side by side: lane 0
// holds x and the bulge, lane 1 y and the disk, lane 2 z and the halo, lane 3 the halo's side products.  A product is
// issued as fma(a, b, -0.0), which rounds the same.  q: the lane's coordinate (lane 3: anything finite).
// The chains are written as C_k = fma(C_k-1, X_k, Y_k) with X_k and Y_k picked by lane beforehand: a pick between two FP64
// instructions that depend on one another would lengthen the step by its latency.
PGX_HD constexpr double halo_coef(int n) {                                     // g_halo_coef's values
    double c = 1.0;
    for (int k = 0; k < n; k++) c = c * ((kHaloG1 - 1.0) - (double)k) / (double)(k + 1);
    return c;
}
__device__ __forceinline__ double quad_accel(double q, int role) {
    const unsigned all = 0xffffffffu;
    const double x = __shfl_sync(all, q, 0, 4), y = __shfl_sync(all, q, 1, 4), z = __shfl_sync(all, q, 2, 4);
    const bool bulge = role == 0, disk = role == 1, halo = role == 2, help = role == 3;
    constexpr double c0 = halo_coef(0), c1 = halo_coef(1), c2 = halo_coef(2), c3 = halo_coef(3), c4 = halo_coef(4);
    static_assert(kPowTerms == 4, "the series below has four terms");
    const double R2 = fma(x, x, y * y);
    const double w = fma(z, z, disk ? kDiskB2 : R2);                      // r2, or z^2 + b^2 of the disk
    const double arg = w + (bulge ? kBulgeB2 : 0.0);
    const uint32_t hi = f64_hi(arg);
    bool ok = seed_ok(hi) && (disk || __double_as_longlong(w) > kTinyR2Bits);
    const double inv = rsqrt_refine(arg, widen_seed(fast_rsqrt(seed_arg(hi))));        // ib, iz, ir, ir
    const double iz = __shfl_sync(all, inv, 1, 4);
    // -GM ib | a + sqrt(z^2 + b^2) | r | r, then ib^2 | D^2 | r / 12 | r / 12
    const double A = fma(inv, bulge ? -kBulgeGM : w, disk ? kDiskA : -0.0);
    const double gb = __shfl_sync(all, A, 0, 4);
    const double Ac = disk || __double_as_longlong(A) < kHaloCutBits ? A : kHaloCut;
    const double B = fma(bulge ? inv : Ac, bulge ? inv : (disk ? A : kHaloInvA), disk ? R2 : -0.0);
    const double ib2 = __shfl_sync(all, B, 0, 4);
    // the halo's table entries (lanes 2 and 3), the disk's second seed
    const uint32_t hB = f64_hi(B);
    const int j = (int)((hB >> (20 - kPowSubLog)) & (kPowSub - 1));
    const double invc = __ldg(&g_halo_invc[j]), powc = __ldg(&g_halo_powc[j]);
    int e = (int)((hB >> 20) & 0x7ff) - 1023;
    e = e < -kPow2Bias ? -kPow2Bias : (e > kPow2N - 1 - kPow2Bias ? kPow2N - 1 - kPow2Bias : e);
    const double pow2 = __ldg(&g_halo_pow2[e + kPow2Bias]);
    const double m = __hiloint2double((int)((hB & 0xfffffu) | 0x3ff00000u), __double2loint(B));
    ok = ok && (!disk || seed_ok(hB));
    const double yD = widen_seed(fast_rsqrt(seed_arg(hB)));
    //                 disk: 1 / D     halo: x^a, 1 / (1 + p)     helper: ir^2, ir^3, -GM r / 12, c_j^a 2^(a e)
    const double C1 = fma(disk ? yD : (halo ? m : inv), disk ? yD : (halo ? invc : inv), halo ? -1.0 : -0.0);
    const double C2 = fma(C1, disk ? -B : (halo ? c4 : inv), disk ? 1.0 : (halo ? c3 : -0.0));
    const double ir3 = __shfl_sync(all, C2, 3, 4);
    const double C3 = fma(help ? B : C2, disk ? 0.375 : (halo ? C1 : -kHaloGM), disk ? 0.5 : (halo ? c2 : -0.0));
    const double gx = __shfl_sync(all, C3, 3, 4);
    const double C4 = fma(help ? powc : C3, disk ? C2 : (halo ? C1 : pow2), halo ? c1 : -0.0);
    const double pw = __shfl_sync(all, C4, 3, 4);
    const double C5 = fma(C4, disk ? yD : C1, disk ? yD : c0);
    const double C6 = C5 * (disk ? C5 : pw);                              // iD^2 | x^a
    const double C7 = C6 * (disk ? C5 : B);                               // iD^3 | p
    const double C8 = fma(C7, disk ? -kDiskGM : 1.0, disk ? -0.0 : 1.0);  // fd   | 1 + p
    const double fd = __shfl_sync(all, C8, 1, 4);
    const uint32_t h8 = f64_hi(C8);
    ok = ok && (!halo || seed_ok(h8));
    const double y8 = widen_seed(__frcp_rn(seed_arg(h8)));
    const bool redo = __any_sync(all, !ok && !help);                      // an argument outside the seeds' range
    const double C9 = fma(C8, disk ? kDiskA : -y8, disk ? -0.0 : 1.0);    // fd a | e
    const double fda = __shfl_sync(all, C9, 1, 4);
    const double q8 = C7 * fma(fma(C9, C9, C9), y8, y8);                  // p / (1 + p)
    const double fh = __shfl_sync(all, (gx * q8) * ir3, 2, 4);
    const double g = fma(gb, ib2, fh) + fd;
    double a = q * (halo ? fma(fda, iz, g) : g);
    if (redo) {
        const Accel f = mw_accel_any(x, y, z);
        a = bulge ? f.x : (disk ? f.y : f.z);
    }
    return a;
}

// One coordinate of an orbit on four lanes (Orbit's step)
struct QuadOrbit {
    double q, v, a;
    __device__ __forceinline__ void init(int role) { a = quad_accel(q, role); }
    __device__ __forceinline__ void kdk(double dt, double h, int role) {
        v = fma(a, h, v);
        q = fma(v, dt, q);
        a = quad_accel(q, role);
        v = fma(a, h, v);
    }
};

// force32 (pgx_orbit32.cuh) on four lanes per orbit, as quad_accel does it for FP64: the same operations on the same
// operands, so the same bits, in about 270 instructions a step for 8 orbits a warp where one lane per orbit takes 340
// for 32.  That is three times the issue slots, but a step is then some 900 cycles long for a warp alone and not 2,300:
// for batches that leave the schedulers idle.  Lane 0 holds x and the bulge, 1 y and the disk, 2 z and the halo, 3 a
// coordinate that stays 0.
__device__ __forceinline__ F2 quad_shfl(F2 v, int src) {
    return F2{__shfl_sync(0xffffffffu, v.h, src, 4), __shfl_sync(0xffffffffu, v.l, src, 4)};
}
__device__ __forceinline__ F2 f2_pick(bool a, F2 x, F2 y) { return F2{a ? x.h : y.h, a ? x.l : y.l}; }
// K's constant of the lane's role (lane 3: the halo's)
__device__ __forceinline__ F3 quad_constant(const Force32 &K, int role) {
    return role == 0 ? K.bulge : (role == 1 ? K.disk : K.halo);
}
// x: the lane's coordinate; its acceleration in displacement units
__device__ __forceinline__ int64_t quad_accel32(const F3 &k, float c, int64_t x, int role, float &r2out) {
    using M = MwModel32;
    const bool bulge = role == 0, disk = role == 1;
    const F2 f = fixed_to_f2(x, c), sq = f2_sqr(f);
    const F2 z2 = quad_shfl(sq, 2), R2 = f2_add(quad_shfl(sq, 0), quad_shfl(sq, 1)), r2 = f2_add(R2, z2);
    r2out = r2.h;
    const F2 u = halo32_power<M>(HaloTable32(), r2);
    const F2 arg = f2_add(f2_pick(disk, z2, r2), bulge ? M::bulge_b2() : (disk ? M::disk_b2() : F2{0.f, 0.f}));
    const F2 inv = f2_rsqrt(arg);                                                   // ib | iz | ir
    const F2 a = f2_add(f2_mul(f2_pick(disk, arg, inv), f2_pick(disk, inv, u)), disk ? M::disk_a() : F2{1.f, 0.f});
    const F2 q = f2_sqr(f2_pick(disk, a, inv));                                     // s^2 | ir^2
    const F2 iD = f2_rsqrt(f2_add(q, R2)), rc = f2_rcp(a);
    const F2 cube = f2_cube(f2_pick(disk, iD, inv));                                // ib^3 | D^-3 | ir^3
    F2 e = f2_mul3(f2_pick(role >= 2, f2_mul(q, rc), cube), k);                     // bulge | disk | halo
    if (role >= 2 && !inside_cut<M>(r2)) e = f2_mul3(f2_mul3(cube, k), M::far());
    const F2 ez = f2_mul(e, f2_mul(a, inv));                                        // (disk) along z
    const F2 g1 = f2_add(quad_shfl(e, 2), quad_shfl(e, 0)), fd = quad_shfl(e, 1), fz = quad_shfl(ez, 1);
    return acc_to_fixed(f2_mul(f2_norm(f2_add(g1, f2_pick(role == 2, fz, fd))), f));
}
// mw_accel_near's coordinate of the lane, its operations on four lanes (every lane of the warp calls)
__device__ __noinline__ int64_t quad_accel_near(const F3 k, const OrbitScale s, double dt, int64_t x, int role) {
    const unsigned all = 0xffffffffu;
    float r2;
    const int64_t a = quad_accel32(role == 0 ? F3{0.f, 0.f, 0.f} : k, s.c, x, role, r2);
    const double q = (double)x * pow2(s.e - 55);
    const double X = __shfl_sync(all, q, 0, 4), Y = __shfl_sync(all, q, 1, 4), Z = __shfl_sync(all, q, 2, 4);
    const double g = MwBulge64()(fma(X, X, fma(Y, Y, Z * Z))) * (dt * dt * pow2(61 - s.e + s.k));
    return a + f64_to_i64(g * q);
}

}  // namespace pgx
