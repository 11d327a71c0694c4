// pgx_scan.cu -- the star x cluster screen of libphygas_gb300 in FP64, and the stages every screen path shares.
//
// Built with --fmad=false: the per-point chi2 (reference ph_screen_chi2_cut, src/phygas.c:370-407) and the
// 512-draw probabilities (reference ph_screen_finish, src/phygas.c:413-444) are evaluated with the reference's
// operation order and no contraction, so that on identical tracks they give the reference's bits, and so that the
// FP64 path and the FP64 rechecks of the mixed-precision path (pgx_mixed.cu, which includes the same functions)
// can never disagree.
//
//   k_scan64       warp = 32 stars x one cluster (same track length, the cluster's points are a broadcast load): the
//                  reference's trace rejection is decided per point on FP32 positions wherever their error leaves no
//                  doubt, the points left are queued and evaluated 32 at a time, one per lane; writes chi2, kb, sb per
//                  pair, cluster-major
//   k_count_kept / k_exclusive_scan / k_emit_kept   stable compaction of the pairs under the cut, (star, cluster)
//   k_finish_prep  one thread per kept pair: interpolated separation, speeds, sigma, Cholesky factor, pair seed
//   k_finish64     a warp for four kept pairs: their 512 draws x 3 Gaussians in FP64, a draw's first coordinate before the
//                  others and its random bits before that, each stage on full warps
#include "pgx_internal.cuh"
#include "pgx_kernels.h"
#include "pgx_screen_math.cuh"

namespace pgx {

// Bound by the FP64 pipe (one warp instruction per 19 cycles and SM).  With a lane walking its own pair, a warp paid for
// the full point (about 150 FP64 instructions) whenever one lane of 32 needed it, 186 a point on average: 22.9 ms for
// 250 stars x 4,087 clusters.  With the trace test on the FP32 units and full warps for the points that it leaves, 11.9;
// with the points whose form at the point is all (classify32) on their own full warps, 7.8 ms.  Every value is still the
// FP64 expression; tables without FP32 tracks (one pair of the drop-in API) take the whole of it for every point.
constexpr int kScan64Warps = 4, kScan64Queue = 64;

__global__ void __launch_bounds__(kScan64Warps * 32) k_scan64(ScreenTables T, double cut, double *__restrict__ chi2T,
                                                              int *__restrict__ kbT, double *__restrict__ sbT) {
    // two queues: points whose form at the point is all (kPointStart), and the others; owner lane | undecided << 5 |
    // point << 6
    __shared__ unsigned s_q[kScan64Warps][2][kScan64Queue];
    __shared__ double s_v[kScan64Warps][32], s_s[kScan64Warps][32];
    __shared__ unsigned s_own[kScan64Warps][32];
    const unsigned all = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, s0 = blockIdx.x * blockDim.x + w * 32;
    if (s0 >= T.nt) return;                                       // the whole warp: uniform
    const bool active = s0 + lane < T.nt;
    const int s = active ? s0 + lane : T.nt - 1;
    const size_t NT = T.nt, NC = T.nc;
    const float cutf = (float)cut;
    const bool test32 = T.t32 && (cut < 1e30 || cut == kInf);
    for (int c = blockIdx.y; c < T.nc; c += gridDim.y) {
        const int n = T.ns < T.cn[c] ? T.ns : T.cn[c];
        const double R2 = T.R2[c];
        ScanState st;
        st.begin();
        int qn[2] = {0, 0};
        // the first cnt points of a queue in FP64, one per lane; then each owner folds its own
        auto drain = [&](int which, int cnt) {
            __syncwarp();
            s_own[w][lane] = 0u;
            __syncwarp();
            if (lane < cnt) {
                const unsigned e = s_q[w][which][lane];
                const int k = (int)(e >> 6), so = s0 + (int)(e & 31u);
                const double *tk = T.t64 + (size_t)k * 12 * NT + so, *ck = T.c64 + (size_t)k * 12 * NC + c;
                double M[6], m0[3], m1[3], sv = 0.0;
#pragma unroll
                for (int i = 0; i < 6; i++) M[i] = tk[(6 + i) * NT] + __ldg(ck + (6 + i) * NC);
#pragma unroll
                for (int i = 0; i < 3; i++) m0[i] = tk[i * NT] - __ldg(ck + i * NC);
                if (which == 0) {
                    s_v[w][lane] = point_start64(M, R2, m0);
                } else {
                    const bool more = k + 1 < n;
#pragma unroll
                    for (int i = 0; i < 3; i++) m1[i] = more ? tk[(12 + i) * NT] - __ldg(ck + (12 + i) * NC) : m0[i];
                    s_v[w][lane] = point_chi2_64(M, R2, m0, m1, more, e & 32u ? cut : kInf, sv);
                }
                s_s[w][lane] = sv;
                atomicOr(&s_own[w][e & 31u], 1u << lane);
            }
            __syncwarp();
            for (unsigned mine = s_own[w][lane]; mine; mine &= mine - 1u) {
                const int j = __ffs(mine) - 1;
                st.fold((int)(s_q[w][which][j] >> 6), s_v[w][j], s_s[w][j]);
            }
            __syncwarp();
            const int rest = qn[which] - cnt;
            const unsigned v = lane < rest ? s_q[w][which][cnt + lane] : 0u;
            __syncwarp();
            if (lane < rest) s_q[w][which][lane] = v;
            qn[which] = rest;
        };
        float4 t0, t1, t2, c0, c1, c2;
        float mc[3], mn[3];
        if (test32) {
            const float4 *a = T.t32 + (size_t)s * 3, *b = T.c32 + (size_t)c * 3;
            t0 = a[0]; t1 = a[1]; t2 = a[2];
            c0 = __ldg(b); c1 = __ldg(b + 1); c2 = __ldg(b + 2);
            sep32(t0, t1, c0, c1, mc);
        }
        for (int k = 0; k < n; k++) {
            int kind = kPointOpen;
            if (test32) {
                const float tr = (t1.z + c1.z) + (t2.y + c2.y) + (t2.w + c2.w);
                mn[0] = mc[0]; mn[1] = mc[1]; mn[2] = mc[2];
                if (k + 1 < n) {
                    const float4 *a = T.t32 + ((size_t)(k + 1) * NT + s) * 3, *b = T.c32 + ((size_t)(k + 1) * NC + c) * 3;
                    t0 = a[0]; t1 = a[1]; t2 = a[2];
                    c0 = __ldg(b); c1 = __ldg(b + 1); c2 = __ldg(b + 2);
                    sep32(t0, t1, c0, c1, mn);
                }
                kind = classify32(mc, mn, tr, cutf);
                mc[0] = mn[0]; mc[1] = mn[1]; mc[2] = mn[2];
            }
            const unsigned entry = (unsigned)lane | (kind == kPointOpen ? 32u : 0u) | (unsigned)k << 6;
#pragma unroll
            for (int which = 0; which < 2; which++) {
                const bool mine = active && (which == 0 ? kind == kPointStart : (kind == kPointNear || kind == kPointOpen));
                const unsigned m = __ballot_sync(all, mine);
                if (mine) s_q[w][which][qn[which] + __popc(m & ((1u << lane) - 1u))] = entry;
                qn[which] += __popc(m);
                if (qn[which] >= 32) drain(which, 32);
            }
        }
#pragma unroll
        for (int which = 0; which < 2; which++)
            if (qn[which] > 0) drain(which, qn[which]);
        if (!active) continue;
        const size_t o = (size_t)c * NT + s;
        chi2T[o] = st.best;
        kbT[o] = st.kb;
        sbT[o] = st.sb;
    }
}

__global__ void k_count_kept(int nt, int nc, const double *__restrict__ chi2T, double cut, int *__restrict__ cnt) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nt) return;
    int n = 0;
    for (int c = 0; c < nc; c++) n += chi2T[(size_t)c * nt + s] < cut;
    cnt[s] = n;
}

// exclusive prefix sum of n ints by one CTA of 1024 threads (n is a star count: a few 10^4)
__global__ void __launch_bounds__(1024) k_exclusive_scan(int n, const int *__restrict__ in, int *__restrict__ out,
                                                         int *__restrict__ total) {
    __shared__ int part[1024];
    __shared__ int carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < n; base += 1024) {
        const int i = base + threadIdx.x;
        const int v = i < n ? in[i] : 0;
        part[threadIdx.x] = v;
        __syncthreads();
        for (int d = 1; d < 1024; d <<= 1) {
            const int add = threadIdx.x >= d ? part[threadIdx.x - d] : 0;
            __syncthreads();
            part[threadIdx.x] += add;
            __syncthreads();
        }
        if (i < n) out[i] = carry + part[threadIdx.x] - v;
        __syncthreads();
        if (threadIdx.x == 1023) carry += part[1023];
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

__global__ void k_emit_kept(int nt, int nc, const double *__restrict__ chi2T, const int *__restrict__ kbT,
                            const double *__restrict__ sbT, double cut, const int *__restrict__ off,
                            KeptPair *__restrict__ out) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nt) return;
    int j = off[s];
    for (int c = 0; c < nc; c++) {
        const size_t o = (size_t)c * nt + s;
        const double q = chi2T[o];
        if (q < cut) {
            KeptPair p;
            p.s = s; p.c = c; p.kb = kbT[o]; p.pad = 0; p.sb = sbT[o]; p.chi2 = q;
            out[j++] = p;
        }
    }
}

__global__ void k_finish_prep(ScreenTables T, int n, const KeptPair *__restrict__ kp, FinishIn *__restrict__ fin,
                              ScreenRowDev *__restrict__ rows) {
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= n) return;
    const KeptPair p = kp[h];
    FinishIn f;
    ScreenRowDev r;
    finish_prep_pair(T, p, f, r);
    fin[h] = f;
    rows[h] = r;
}

// The 512 draws of a kept pair in FP64, in three stages that each leave the next one few draws:
//   1  its random bits.  A draw is inside a radius only if |x| = |mx + l00 z0| < R = max(r50, rtot), so |z0| > (|mx| - R)
//      / l00 with the sign of -mx: its first uniform must be below exp(-z^2 / 2) for |z0| = sqrt(-2 ln u1) |cos| to get
//      there, and its second in the half circle where the cosine has the sign.  Margins cover the rounding.
//   2  z0 and x.  |x| >= R settles it: r >= |x| in FP64 too, the square root of the rounded square being |x|.
//   3  the other two Gaussians and the distance, as the reference computes them.
// Bound by the FP64 pipe (a Gaussian is a log, a cosine and a square root, about 80 instructions): all three of every
// draw took 22.7 ms for 108,702 pairs (250 stars x 4,087 clusters), these stages 1.9 ms.  A warp takes kPairs64 pairs
// so that stages 2 and 3 run on full warps.
constexpr int kFin64Warps = 4, kPairs64 = 4, kFin64Queue = 64;

__global__ void __launch_bounds__(kFin64Warps * 32) k_finish64(int n, const FinishIn *__restrict__ fin,
                                                               ScreenRowDev *__restrict__ rows) {
    __shared__ int s_i[kFin64Warps][kFin64Queue], s_j[kFin64Warps][kFin64Queue];      // pair << 9 | draw
    __shared__ double s_z[kFin64Warps][kFin64Queue];
    __shared__ int s_n[kFin64Warps][2 * kPairs64];
    const unsigned all = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long h0 = ((long)blockIdx.x * kFin64Warps + w) * kPairs64;
    if (h0 >= n) return;                                          // the whole warp: uniform
    if (lane < 2 * kPairs64) s_n[w][lane] = 0;
    int ni = 0, nj = 0;
    // stage 3 for the entries [0, cnt)
    auto inside = [&](int cnt) {
        __syncwarp();
        if (lane < cnt) {
            const int e = s_j[w][lane], p = e >> 9, i = e & 511;
            const FinishIn &f = fin[h0 + p];
            double x, y, z;
            draw_xyz64(f, i, s_z[w][lane], x, y, z);
            const double r = sqrt(x * x + y * y + z * z);
            if (r < f.r50) atomicAdd(&s_n[w][2 * p], 1);
            if (r < f.rt) atomicAdd(&s_n[w][2 * p + 1], 1);
        }
        __syncwarp();
    };
    // stage 2 for the entries [0, cnt)
    auto first = [&](int cnt) {
        __syncwarp();
        bool open = false;
        int e = 0;
        double z0 = 0.0;
        if (lane < cnt) {
            e = s_i[w][lane];
            const FinishIn &f = fin[h0 + (e >> 9)];
            const uint64_t c = 6ull * (uint64_t)(e & 511);
            z0 = gauss64(splitmix_at(f.seed, c + 1), splitmix_at(f.seed, c + 2));
            const double x = fabs(f.mx + f.l00 * z0);
            open = !(x >= fmax(f.r50, f.rt) && x > 1e-150);       // (below, the square may be subnormal)
        }
        const unsigned m = __ballot_sync(all, open);
        if (open) {
            const int at = nj + __popc(m & ((1u << lane) - 1u));
            s_j[w][at] = e;
            s_z[w][at] = z0;
        }
        nj += __popc(m);
        if (nj >= 32) {
            inside(32);
            nj -= 32;
            int v = 0;
            double vz = 0.0;
            if (lane < nj) { v = s_j[w][32 + lane]; vz = s_z[w][32 + lane]; }
            __syncwarp();
            if (lane < nj) { s_j[w][lane] = v; s_z[w][lane] = vz; }
        }
        __syncwarp();
    };
    const int np = (int)(n - h0 < kPairs64 ? n - h0 : kPairs64);
    for (int p = 0; p < np; p++) {
        const FinishIn &f = fin[h0 + p];
        const uint64_t seed = f.seed;
        // stage 1's bounds: the largest first uniform (in units of 2^-53, all ones: no bound) and the cosine's sign
        uint64_t umax = ~0ull;
        int sign = 0;
        const double R = fmax(f.r50, f.rt), ax = fabs(f.mx);
        const double zmin = (ax - R - 1e-15 * (ax + R)) / f.l00 * (1.0 - 1e-9);
        if (zmin > 1e-6 && zmin < 1e300) {
            umax = (uint64_t)(exp(-0.5 * zmin * zmin) * (1.0 + 1e-9) * 9007199254740992.0) + 1;
            sign = f.mx > 0 ? -1 : 1;                     // (l00 > 0)
        }
#pragma unroll 1
        for (int q = 0; q < 16; q++) {
            const int i = lane + 32 * q;
            const uint64_t c = 6ull * (uint64_t)i;
            bool open = (splitmix_at(seed, c + 1) >> 11) <= umax;
            if (open && sign) {
                const unsigned quad = (unsigned)(splitmix_at(seed, c + 2) >> 62);       // cos > 0 in quadrants 0, 3
                open = (quad == 0 || quad == 3) == (sign > 0);
            }
            const unsigned m = __ballot_sync(all, open);
            if (open) s_i[w][ni + __popc(m & ((1u << lane) - 1u))] = p << 9 | i;
            ni += __popc(m);
            if (ni >= 32) {
                first(32);
                ni -= 32;
                const int v = lane < ni ? s_i[w][32 + lane] : 0;
                __syncwarp();
                if (lane < ni) s_i[w][lane] = v;
            }
        }
    }
    if (ni > 0) first(ni);
    if (nj > 0) inside(nj);
    __syncwarp();
    if (lane < np) {
        rows[h0 + lane].p_r50 = (double)s_n[w][2 * lane] / 512.0;
        rows[h0 + lane].p_rtot = (double)s_n[w][2 * lane + 1] / 512.0;
    }
}

void launch_finish64(cudaStream_t st, int n, const FinishIn *fin, ScreenRowDev *rows) {
    const int per_block = kFin64Warps * kPairs64;
    k_finish64<<<(n + per_block - 1) / per_block, kFin64Warps * 32, 0, st>>>(n, fin, rows);
}

}  // namespace pgx
