// pgx_orbit32.cuh -- the Milky Way orbit on the FP32 and integer units (internal header; also compiles as plain host
// C++ with FP contraction off, so that its error can be measured on the CPU against 113-bit arithmetic).
//
// What bounds the FP64 step of pgx_force.cuh: an FP64 warp instruction occupies its scheduler for 64 to 76 cycles on
// this GPU, an FP32 one for one, so its 68 FP64 instructions a step leave nine issue slots in ten idle.  Here the same
// kick-drift-kick step takes about 340 FP32 and integer instructions and no FP64 one:
//  * positions are 64-bit integers in units of 2^-55 kpc, and the velocity is kept as the displacement of a step,
//    w = v dt at the half step, in units of 2^-61 kpc: x += w and w += a dt^2 are the leapfrog (the two half kicks
//    between drifts added up), exact but for the last unit, which is 64 times finer than FP64's at 8 kpc;
//  * the force is evaluated on pairs of floats (value = h + l, about 48 bits), each product and sum with its rounding
//    error carried along by fused multiply-adds; the constants are the FP64 ones, in three floats.
// The force's error, 2^-47.2 relative (rms) and random, enters w through a dt^2 ~ 2^-11 w, below FP64's own rounding
// of the velocity -- where an orbit turns slowly.  Within kOrbit32Near |dt| of the centre a dt is so large a part of v that
// it is not: there the bulge's part, nearly all of it, is FP64's (accel_near; FP64 throughout is no nearer).
//
// What is traced this way is what comes out no further from exact arithmetic than FP64 steps, measured against 113-bit
// arithmetic (tests/test_orbit32_range.py): 0.01 <= |dt| <= 0.125 Myr, a start at least 0.15 kpc from the centre and a reach
// of less than 10^6 kpc.  2,000 steps of 0.05 Myr end 8e-15 kpc off (rms; FP64 steps: 9e-14) at 8 kpc, 3e-14 (1.0e-13) at 1
// kpc, 1e-14 (2.7e-12) at 1,000 kpc and 7e-13 (4.5e-11) at 100,000.  Other orbits, and those that come within 2^-10 kpc of
// the centre, a caller traces in FP64.
//
// The units (OrbitScale): orbits that reach 256 kpc and more take positions' units 2^e times larger, those that stay within 64
// four times smaller.  A displacement's unit does not follow: it is 2^-61 kpc and finer at shorter steps, since FP64's
// rounding of a slow orbit's velocity is finer too (with a unit that grew with the scale, orbits beyond 5,000 kpc and
// slow ones at steps of 0.02 Myr came out up to ten times further off than FP64's).
#pragma once
#include <cstdint>
#include "pgx_bits.cuh"

namespace pgx {

struct F2 {
    float h, l;          // h + l; |l| is at most a few units of 2^-24 |h|
};
struct F3 {
    float a, b, c;       // a constant of 53 bits or more: a + b + c
};

PGX_HD constexpr F3 split3(double v) {
    const float a = (float)v, b = (float)(v - (double)a), c = (float)(v - (double)a - (double)b);
    return F3{a, b, c};
}
PGX_HD constexpr F2 split2(double v) {
    const float a = (float)v;
    return F2{a, (float)(v - (double)a)};
}
// c x^2 s in 72 bits, s a power of two: a rounding to FP64 here would be the same on every step
PGX_HD F3 split3_square(double c, double x, double s) {
    const double q = x * x, qe = fma(x, x, -q), p = c * q, e = fma(c, q, -p) + c * qe;
    F3 r = split3(p * s);
    r.c = (float)((p * s - (double)r.a - (double)r.b) + e * s);
    return r;
}

PGX_HD F2 f2_add(F2 a, F2 b) {                                        // any order of magnitudes
    const float s = a.h + b.h, t = s - a.h;
    return F2{s, ((a.h - (s - t)) + (b.h - t)) + (a.l + b.l)};
}
PGX_HD F2 f2_norm(F2 a) {                                             // |l| <= 2^-24 |h|
    const float s = a.h + a.l;
    return F2{s, a.l - (s - a.h)};
}
PGX_HD F2 f2_mul(F2 a, F2 b) {
    const float p = a.h * b.h;
    return F2{p, fmaf(a.l, b.h, fmaf(a.h, b.l, fmaf(a.h, b.h, -p)))};
}
// squares and cubes keep the product of the low parts: it has a sign there, and 2^-50 of the force, always the same
// way, moves an orbit by as much as all of FP64's random roundings
PGX_HD F2 f2_sqr(F2 a) {
    const float p = a.h * a.h;
    return F2{p, fmaf(a.h, a.l + a.l, fmaf(a.l, a.l, fmaf(a.h, a.h, -p)))};
}
PGX_HD F2 f2_cube(F2 a) {
    const F2 q = f2_sqr(a);
    const float p = q.h * a.h;
    return F2{p, fmaf(q.l, a.h, fmaf(q.h, a.l, fmaf(q.l, a.l, fmaf(q.h, a.h, -p))))};
}
PGX_HD F2 f2_mul3(F2 a, F3 c) {
    const float p = a.h * c.a;
    return F2{p, fmaf(a.l, c.a, fmaf(a.h, c.b, fmaf(a.h, c.c, fmaf(a.h, c.a, -p))))};
}
// a^-1/2 from the unit's result y (2^-22.9) as y (1 + e/2 + 3 e^2 / 8), e = 1 - a y^2 = e1 + e2 with e1 = 1 - p exact
// (a few bits) and e2 below 2^-22, so that neither is rounded at e's own size
PGX_HD F2 f2_rsqrt(F2 a) {
    const float y = fast_rsqrt(a.h), t = y * y, tl = fmaf(y, y, -t);
    const float p = a.h * t, e1 = 1.f - p;
    const float e2 = fmaf(-a.l, t, fmaf(-a.h, tl, -fmaf(a.h, t, -p)));
    const float e = e1 + e2, c = 0.5f * e1, d = fmaf(e * e, 0.375f, 0.5f * e2);
    const float yh = fmaf(y, c + d, y);
    return F2{yh, fmaf(y, d, fmaf(y, c, y - yh))};
}
// 1 / a likewise: y (1 + e + e^2)
PGX_HD F2 f2_rcp(F2 a) {
    const float y = fast_rcp(a.h), e1 = fmaf(-a.h, y, 1.f), e2 = -a.l * y, e = e1 + e2;
    const float d = fmaf(e, e, e2), yh = fmaf(y, e1 + d, y);
    return F2{yh, fmaf(y, d, fmaf(y, e1, y - yh))};
}

// ---- the halo's power --------------------------------------------------------------------------------------------
// (12 / r)^(1 + a) = r^-1 12^(1 + a) r2^-a', a' = a / 2 = 0.01.  r2 = 2^e m in sub-interval j of 256, i = 1 / centre
// in FP32, r2 i = 1 + t with |t| <= 2^-9, u = 12^(1 + a) i^a' from the table and (1 + t)^-a' by its series to t^4.
constexpr int kHalo32Lo = -20, kHalo32Exp = 34, kHalo32Sub = 256, kHalo32N = kHalo32Exp * kHalo32Sub;

struct Halo32 {
    float i, u0, u1, u2;
};
// entry n of the table (FP64 ldexp and pow, a few ulp)
PGX_HD Halo32 halo32_entry(int n, double a, double inv_a) {
    const int e = kHalo32Lo + n / kHalo32Sub, j = n % kHalo32Sub;
    const float i = (float)(ldexp(1.0, -e) / (1.0 + (j + 0.5) / kHalo32Sub));
    const F3 u = split3(pow(inv_a, -(1.0 + a)) * pow((double)i, 0.5 * a));
    return Halo32{i, u.a, u.b, u.c};
}

PGX_HD uint32_t f32_bits(float x) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(x);
#else
    uint32_t b;
    std::memcpy(&b, &x, 4);
    return b;
#endif
}
PGX_HD int32_t f32_rint(float x) {
#ifdef __CUDA_ARCH__
    return __float2int_rn(x);
#else
    return (int32_t)lrintf(x);
#endif
}

// 2^n, normal
PGX_HD double pow2(int n) {
#ifdef __CUDA_ARCH__
    return __hiloint2double((1023 + n) << 20, 0);
#else
    return ldexp(1.0, n);
#endif
}

// ---- units -------------------------------------------------------------------------------------------------------
// 2^e times 2^-55 kpc (positions) and 2^-(61 + k) kpc (displacements): c = 2^(e - 23) kpc, the unit of a position's high
// word
struct OrbitScale {
    float c;
    int e, k = 0;
};
constexpr double kOrbit32MinDt = 0.01, kOrbit32MaxDt = 0.125, kOrbit32MaxReach = 1e6;
constexpr double kOrbit32Near = 12.0, kOrbit32NearMin = 0.4;       // kpc per Myr of step; kpc
constexpr double kOrbit32MinStart = 0.15;
constexpr float kOrbit32MinR2 = 0x1p-20f;

PGX_HD float orbit32_near2(double dt) {
    const double r = fmax(kOrbit32Near * fabs(dt), kOrbit32NearMin);
    return (float)(r * r);
}

// The scale for orbits that reach at most `reach` kpc; false: trace them in FP64 (NaN included).
PGX_HD bool orbit32_scale(double reach, double dt, OrbitScale &s) {
    const double d = fabs(dt);
    if (!(reach < kOrbit32MaxReach && d >= kOrbit32MinDt && d <= kOrbit32MaxDt)) return false;
    s.e = reach < 64.0 ? -2 : 0;
    s.c = reach < 64.0 ? 0x1p-25f : 0x1p-23f;
    for (double lim = 256.0; lim <= reach; lim *= 2.0) { s.e++; s.c *= 2.f; }
    return true;
}
// The scale with the displacements' own unit: 2^-61 kpc at any e, and as much finer as a dt^2 of shorter steps leaves its
// integer room (to 2^-68 at 0.01 Myr) -- less where v dt would leave a quarter of the integer's range
PGX_HD bool orbit32_units(double reach, double vdt, double dt, OrbitScale &s) {
    if (!orbit32_scale(reach, dt, s)) return false;
    s.k = s.e;
    for (double t = kOrbit32MaxDt / dt * (kOrbit32MaxDt / dt); t >= 2.0; t *= 0.5) s.k++;
    while (s.k > 0 && vdt >= pow2(s.e - s.k - 1)) s.k--;
    return vdt < pow2(s.e - s.k - 1);
}
// The reach to ask for an orbit from q, v over `steps` steps: twice the straight line's, but an orbit of 0.3 kpc/Myr within
// 3 kpc hardly leaves 30 kpc and one of 0.4 within 20 kpc 200 (one that does is noticed: orbit32_max_r2)
PGX_HD double orbit32_reach(const double *q, const double *v, double steps, double dt, double &vdt) {
    const double x = fmax(fabs(q[0]), fmax(fabs(q[1]), fabs(q[2])));
    const double u = fmax(fabs(v[0]), fmax(fabs(v[1]), fabs(v[2])));
    vdt = u * fabs(dt);
    double drift = 2.0 * vdt * steps;
    if (u < 0.4 && x < 20.0) drift = fmin(drift, 200.0);
    if (u < 0.3 && x < 3.0) drift = fmin(drift, 30.0);
    return fmax(2.0 * x + drift + 20.0, 512.0 * vdt);
}
// r2 below this: inside the positions' range
PGX_HD float orbit32_max_r2(const OrbitScale &s) { return (s.c * 0x1p31f) * (s.c * 0x1p31f) * 0.98f; }

// the model's GM times dt^2 2^(37 + k) in the scale's units (a dt^2's high part is an integer multiple of 2^-(37 + k), the
// rest of 2^-(61 + k))
struct Force32 {
    F3 bulge, disk, halo;
};
// M: the model's FP64 constants
template <class M> PGX_HD Force32 force32_constants(double dt, const OrbitScale &s) {
    const double u = pow2(37 - s.e + s.k), h = M::halo_GM * M::halo_inv_a;
    Force32 k = {split3_square(-M::bulge_GM, dt, u), split3_square(-M::disk_GM, dt, u), split3_square(-h, dt, u)};
    k.halo.c -= (float)(fma(M::halo_GM, M::halo_inv_a, -h) * dt * dt * u);
    return k;
}

struct Acc32 {
    F2 x, y, z;          // a dt^2 2^(37 + k) in the scale's units
    float r2;
};

// 12^(1 + a) r2^-a'
template <class M, class Table> PGX_HD F2 halo32_power(const Table &table, F2 r2) {
    int n = (int)(f32_bits(r2.h) >> 15) - ((127 + kHalo32Lo) << 8);
    n = n < 0 ? 0 : (n > kHalo32N - 1 ? kHalo32N - 1 : n);
    const Halo32 T = table(n);
    const float p = r2.h * T.i, t = p - 1.f, tl = fmaf(r2.l, T.i, fmaf(r2.h, T.i, -p));
    const float tt = t + tl, w = (tt * tt) * fmaf(tt, fmaf(tt, M::c4, M::c3), M::c2);
    const float v = M::a1 * t, vl = fmaf(M::a1, tl, fmaf(M::a1l, t, fmaf(M::a1, t, -v))) + w;
    const float s0 = 1.f + v, s1 = (v - (s0 - 1.f)) + vl;
    return F2{s0 * T.u0, fmaf(s1, T.u0, fmaf(s0, T.u1, fmaf(s0, T.u2, fmaf(s0, T.u0, -(s0 * T.u0)))))};
}

// r2 < cut^2 with its low part: the halo's force has a kink there, and its high part alone, a few 10^-6 kpc off, took steps
// that end beside it 3e-8 of the force wrong
template <class M> PGX_HD bool inside_cut(F2 r2) { return (r2.h - M::cut2) + r2.l < 0.f; }

// M: the model's lengths as float pairs (bulge_b2(), disk_b2(), disk_a()), the halo's cut-off (cut2 = cut^2, and far() =
// cut q(cut) for the enclosed mass beyond it) and the series of (1 + t)^-a' (a1 + a1l, c2, c3, c4)
template <class M, class Table> PGX_HD Acc32 force32(const Force32 &K, const Table &table, F2 x, F2 y, F2 z) {
    const F2 z2 = f2_sqr(z), R2 = f2_add(f2_sqr(x), f2_sqr(y)), r2 = f2_add(R2, z2);
    const F2 ir = f2_rsqrt(r2);
    F2 fh;
    if (inside_cut<M>(r2)) {
        // halo: -K r^-2 / (1 + (12 / r)^(1 + a))
        const F2 u = halo32_power<M>(table, r2);
        const F2 q = f2_rcp(f2_add(f2_mul(ir, u), F2{1.f, 0.f}));
        fh = f2_mul3(f2_mul(f2_sqr(ir), q), K.halo);
    } else {
        fh = f2_mul3(f2_mul3(f2_cube(ir), K.halo), M::far());
    }
    // bulge: -K (r2 + b^2)^-3/2
    const F2 ib = f2_rsqrt(f2_add(r2, M::bulge_b2()));
    const F2 g1 = f2_add(fh, f2_mul3(f2_cube(ib), K.bulge));
    // disk: -K D^-3, and along z times (a + sqrt(z^2 + b^2)) / sqrt(z^2 + b^2)
    const F2 zb = f2_add(z2, M::disk_b2()), iz = f2_rsqrt(zb);
    const F2 s = f2_add(f2_mul(zb, iz), M::disk_a());
    const F2 fd = f2_mul3(f2_cube(f2_rsqrt(f2_add(f2_sqr(s), R2))), K.disk);
    const F2 g = f2_norm(f2_add(g1, fd)), gz = f2_norm(f2_add(g1, f2_mul(fd, f2_mul(s, iz))));
    return Acc32{f2_mul(g, x), f2_mul(g, y), f2_mul(gz, z), r2.h};
}

// ---- the state ---------------------------------------------------------------------------------------------------
// A position as a float pair (kpc), to 2^-49 relative: the high word's nearest float, then the other bits in two pieces
PGX_HD F2 fixed_to_f2(int64_t X, float c) {
    const int32_t hi = (int32_t)(X >> 32);
    const uint32_t lo = (uint32_t)X;
    const float f = (float)hi, high = f * c, c1 = c * 0x1p-24f;
    const uint32_t d = (uint32_t)(hi - f32_rint(f));
    const float mid = (float)(int32_t)((d << 24) | (lo >> 8)), s = fmaf(mid, c1, high);
    return F2{s, fmaf((float)(int32_t)(lo & 0xffu), c * 0x1p-32f, fmaf(mid, c1, high - s))};
}
// a dt^2 2^(37 + k) as an integer in units of 2^-(61 + k) kpc.  |a| < 0.18 kpc/Myr^2 anywhere in this model, so with
// |dt| <= 0.125 and k of its step |a.h| < 2^28.6 and, the force's factors being normalized, |a.l| < 3 2^-24 |a.h|: both integers fit 32 bits.
PGX_HD int64_t acc_to_fixed(F2 a) {
    const int32_t n = f32_rint(a.h);
    const int32_t m = f32_rint(((a.h - (float)n) + a.l) * 0x1p24f);
    return (int64_t)n * (1 << 24) + m;
}

// One orbit: position and the coming drift's displacement, the latter with half a position unit added once so that
// the drift's shift (by 6 + k) rounds to nearest.
struct Orbit32 {
    int64_t x, y, z, wx, wy, wz;
};
struct Acc64i {
    int64_t x, y, z;     // a dt^2 in displacement units
};

PGX_HD int64_t f64_to_i64(double x) {
#ifdef __CUDA_ARCH__
    return __double2ll_rn(x);
#else
    return (int64_t)llrint(x);
#endif
}
template <class M, class Table>
PGX_HD Acc64i accel32(const Force32 &K, const Table &table, float c, int64_t x, int64_t y, int64_t z, float &r2) {
    const Acc32 a = force32<M>(K, table, fixed_to_f2(x, c), fixed_to_f2(y, c), fixed_to_f2(z, c));
    r2 = a.r2;
    return Acc64i{acc_to_fixed(a.x), acc_to_fixed(a.y), acc_to_fixed(a.z)};
}

// The force near the centre, where the bulge is nearly all of it: its part in FP64 (bulge(r2) = -GM (r2 + b^2)^-3/2), the
// disk's and the halo's, a few percent, on pairs of floats
template <class M, class Table, class Bulge>
PGX_HD Acc64i accel_near(const Force32 &K, const Table &table, const Bulge &bulge, const OrbitScale &s, double dt, int64_t x,
                         int64_t y, int64_t z) {
    float r2;
    const Acc64i a = accel32<M>(Force32{F3{0.f, 0.f, 0.f}, K.disk, K.halo}, table, s.c, x, y, z, r2);
    const double u = pow2(s.e - 55), X = (double)x * u, Y = (double)y * u, Z = (double)z * u;
    const double g = bulge(fma(X, X, fma(Y, Y, Z * Z))) * (dt * dt * pow2(61 - s.e + s.k));
    return Acc64i{a.x + f64_to_i64(g * X), a.y + f64_to_i64(g * Y), a.z + f64_to_i64(g * Z)};
}
// a step's force: accel32, within near2 = orbit32_near2(dt) near's (accel_near)
template <class M, class Table, class Near>
PGX_HD Acc64i orbit32_accel(const Force32 &K, const Table &table, const Near &near, const OrbitScale &s, double dt, float near2,
                            int64_t x, int64_t y, int64_t z, float &r2) {
    Acc64i a = accel32<M>(K, table, s.c, x, y, z, r2);
    if (r2 < near2) a = near(K, s, dt, x, y, z);
    return a;
}

// v dt in displacement units, the product's rounding included
PGX_HD int64_t displacement(double v, double dt, double unit) {
    const double w = v * dt;
    return f64_to_i64(w * unit) + f64_to_i64(fma(v, dt, -w) * unit);
}
// whether an orbit may start at q: not where FP64's positions are much finer than the unit
PGX_HD bool orbit32_start_ok(const double *q) {
    return fma(q[0], q[0], fma(q[1], q[1], q[2] * q[2])) >= kOrbit32MinStart * kOrbit32MinStart;
}
// a displacement's drift in position units, sh = 6 + k
PGX_HD int64_t orbit32_drift(int64_t w, int sh) {
#ifdef __CUDA_ARCH__
    const int hi = (int)(w >> 32);
    return (int64_t)(hi >> sh) << 32 | __funnelshift_r((unsigned)w, (unsigned)hi, sh);
#else
    return w >> sh;
#endif
}

// position q and velocity v (kpc, kpc/Myr): displacements of the first drift, v dt + a dt^2 / 2; |q| and |v dt| below the
// scale's range; accel(x, y, z, r2): a position's force
template <class Accel>
PGX_HD void orbit32_start(Orbit32 &o, const Accel &accel, const OrbitScale &s, const double *q, const double *v, double dt,
                          float &r2) {
    const double ux = pow2(55 - s.e), uw = pow2(61 - s.e + s.k);
    const int64_t half = 1LL << (5 + s.k);
    o.x = f64_to_i64(q[0] * ux); o.y = f64_to_i64(q[1] * ux); o.z = f64_to_i64(q[2] * ux);
    const Acc64i a = accel(o.x, o.y, o.z, r2);
    o.wx = displacement(v[0], dt, uw) + a.x / 2 + half;
    o.wy = displacement(v[1], dt, uw) + a.y / 2 + half;
    o.wz = displacement(v[2], dt, uw) + a.z / 2 + half;
}
// the same with the force on pairs of floats anywhere
template <class M, class Table>
PGX_HD void orbit32_start(Orbit32 &o, const Force32 &K, const Table &table, const OrbitScale &s, const double *q,
                          const double *v, double dt, float &r2) {
    orbit32_start(o, [&](int64_t x, int64_t y, int64_t z, float &r) { return accel32<M>(K, table, s.c, x, y, z, r); }, s, q, v,
                  dt, r2);
}

}  // namespace pgx
