// Real-space Ewald of the FP64 form (energies and forces; replaces the pair loop
// of forces.cpp:589-608 with its rwald, forces.cpp:141-177).
//
// What bounds it: the issue of integer instructions. This GPU runs two FP64 lanes a cycle
// an SM (a warp's FP64 multiply-add takes sixteen cycles of the SM, a 32 x 32 -> 64-bit
// integer one half a cycle), so the pair arithmetic is 64-bit fixed point:
//   * coordinates times kappa, in units of 2^-56: differences and images are exact;
//   * u = (kappa r)^2 and everything after it by 62-bit products of 31-bit limbs;
//   * erfc(x)/x and the force factor from degree-7 polynomials in u, their upper four
//     coefficients in 32 bits;
//   * pair forces in units of 2^-56 q_top^2 kappa^2, whose sums are exact.
// Every site pair is taken once (a warp holds 16 sites and visits the tiles of 32 sites at
// ring distances 0 .. T/2, as k_real_half does). The cutoff test comes first in FP32, on
// the wrapped coordinates with a margin above their rounding, and only the pairs that pass
// (31-52 % of them), packed into full warps, are evaluated, where r^2 < r_c^2 is decided.
// Both sides' forces are summed from the packed pairs' shared-memory copies, a lane a site,
// and added to the configuration's sums by integer atomics: no sum depends on the order
// the warps run. A pair below u = 2^-3 (or an Ewald tolerance below 1e-17) goes the FP64
// way instead. (Such tolerances send every pair there: the kernel takes 92 us instead of 58 for all
// ordered pairs in FP64 at 64 waters, 1 bead, 438 instead of 864 at 216, 8 beads; the calls, whose
// reciprocal part is then the longer, 377 instead of 1135 and 1505 instead of 7169.)
// 216 waters, 32 beads: 3283 us for the all-pairs FP64 form with library functions, 337 us
// with the same split and the polynomials in FP64 (37 FP64 instructions a pair), 121 us here
// (143 with the fewer blocks that launch_real64 gives it for the sake of the kernels beside
// it; 512 waters, 32 beads: 1228 us in FP64 arithmetic, 442 here, 498 so). Eight sites a warp run the
// kernel alone 11 % faster but the FP64 steps and calls, where it shares the GPU, no faster.
// The error against 80-bit sums is below the FP64 form's: 2.2e-15 of the real-space forces
// against 3.8e-15 at 64 waters, 1.2e-15 against 3.4e-15 at 216, 0.9e-15 against 6.5e-15 at 512.
#include <math.h>
#include <string.h>

#include <algorithm>

#include "fixed62.h"
#include "qtg_internal.h"

namespace qtg {

// ---- the pair-function tables -----------------------------------------------------
// With u = (kappa r)^2, G(u) = erfc(sqrt u) / sqrt u and W(u) = (G(u) + a exp(-u)) / u
// (a = 2 / sqrt(pi) with the reference's pi), a pair's energy is q_i q_j kappa G and its
// force q_i q_j kappa^3 W d. Both tables split each octave of u into 64 intervals, found
// from the top bits of u, and hold the Taylor coefficients of G and W about an interval's
// middle, degree 7 each. In an interval |t| <= u/128, so the truncated terms are below
// 3e-17 of the value for u < 8 and below 6e-15 for u < 16 (where the value itself is below
// 1e-4 of a near pair's). The coefficients follow from the two functions' differential
// equations,
//   2 u G' + G + (2/sqrt(pi)) e^-u = 0  and  u W = G + a e^-u,
// whose recurrences add terms of one sign only (no cancellation).
// FP64 table (u in [2^R64_LO, 2^R64_HI), 16 doubles an interval): G at the middle is
// erfc's value corrected to first order for the rounding of the square root.
void real64_table(double *tab) {
    const double a0 = 2.0 / sqrt(acos(-1.0)), a = 2.0 / sqrt(PI_REF);
    for (int i = 0; i < R64_INTERVALS; ++i) {
        const long long bits = ((long long)(i + ((1023 + R64_LO) << 6)) << 46) | (1ll << 45);
        double m;
        memcpy(&m, &bits, sizeof(m));
        const double x = sqrt(m), d = fma(-x, x, m), em = exp(-m);
        double g[8], w[8], e = em;
        g[0] = (erfc(x) - a0 * em * d / (2.0 * x)) / x;
        g[0] -= g[0] * d / (2.0 * m);  // 1 / sqrt(m) from 1 / x
        w[0] = (g[0] + a * e) / m;
        for (int k = 0; k < 7; ++k) {
            g[k + 1] = -((2 * k + 1) * g[k] + a0 * e) / (2.0 * m * (k + 1));
            e = -e / (k + 1);
            w[k + 1] = (g[k + 1] + a * e - w[k]) / m;
        }
        for (int k = 0; k < 8; ++k) {
            tab[16 * i + k] = g[k];
            tab[16 * i + 8 + k] = w[k];
        }
    }
}

// Fixed-point table (octaves RI_LO .. RI_LO + RI_OCT - 1): coefficient k times the interval
// width to the k, so that the polynomial's argument is tau in [-1/2, 1/2). An interval is
// W_0 .. W_3 in 64 bits, W_4 .. W_7 in 32 bits of 512 units, then G the same way; the unit
// is 2^-60 for G and 2^-59 for W (2^-57 in the lowest octave, where W reaches 22). The
// constants carry the half unit that the floors of the Horner steps take away.
void real64_int_table(long long *tab) {
    const long double a0 = 2.0L / sqrtl(acosl(-1.0L)), a = 2.0L / sqrtl((long double)PI_REF);
    for (int i = 0; i < RI_OCT * 64; ++i) {
        const long double w0 = ldexpl(1.0L, RI_LO + (i >> 6) - 6), m = ldexpl(1.0L, RI_LO + (i >> 6)) + w0 * ((i & 63) + 0.5L);
        const long double x = sqrtl(m), em = expl(-m);
        long double g[8], w[8], e = em;
        g[0] = erfcl(x) / x;
        w[0] = (g[0] + a * e) / m;
        for (int k = 0; k < 7; ++k) {
            g[k + 1] = -((2 * k + 1) * g[k] + a0 * e) / (2.0L * m * (k + 1));
            e = -e / (k + 1);
            w[k + 1] = (g[k + 1] + a * e - w[k]) / m;
        }
        long long *o = tab + 12 * i;
        for (int f = 0; f < 2; ++f, o += 6) {
            const int bits = f ? 60 : i < 64 ? 57 : 59;
            long double s = ldexpl(1.0L, bits);
            int hi[4];
            for (int k = 0; k < 8; ++k, s *= w0) {
                const long double c = (f ? g[k] : w[k]) * s;
                if (k < 4) o[k] = llrintl(c + (k == 3 ? 0.5L : 0.0L));
                else hi[k - 4] = (int)llrintl(c / 512.0L + (k < 7 ? 0.5L : 0.0L));
            }
            memcpy(o + 4, hi, sizeof(hi));
        }
    }
}

// kappa L_d in units of 2^-56, and (kappa r_c)^2 (-1: beyond what the fixed-point form holds)
void real64_system(const SysDev &S, long long *out) {
    for (int d = 0; d < 3; ++d) out[d] = kappa_fix(S.kappa, S.box[d]);
    const double uc = S.kappa * S.kappa * S.rc_sq;
    out[3] = uc < 38.0 ? llrint(uc * 72057594037927936.0) : -1;
}

namespace {

constexpr int RROWS = 16;          // sites a warp holds
constexpr int RW = 32 / RROWS;     // warps per block: the parts of a tile of 32 sites
constexpr int RLANES = 32 / RROWS;  // lanes that sum a held site's pairs
constexpr int RCAP = RROWS * 32;   // pairs of one visit

struct RSite {
    i64 y[3], q;                   // kappa x in units of 2^-56; charge / q_top in units of 2^-62
};
struct RWarp {
    RSite sj[32], si[RROWS];
    i64 f[3][RCAP];                // the packed pairs' forces on the held site
    float4 sif[RROWS];             // FP32 coordinates and the site's molecule
    unsigned mask[RROWS];          // row r's visited sites that passed
    int off[RROWS + 1];            // where row r's packed pairs start
    unsigned short code[RCAP];     // row, visited site and image of every packed pair
};

// one of the two functions: t = tau in units of 2^-62
__device__ __forceinline__ i64 horner(const longlong2 &c01, const longlong2 &c23, const int4 &c47, const Limbs &t, int t32) {
    int p = c47.w;
    p = c47.z + (int)(((i64)p * t32) >> 32);
    p = c47.y + (int)(((i64)p * t32) >> 32);
    p = c47.x + (int)(((i64)p * t32) >> 32);
    i64 v = c23.y + (((i64)p * t32) >> 23);
    v = c23.x + mul62(split62(v), t);
    v = c01.y + mul62(split62(v), t);
    return c01.x + mul62(split62(v), t);
}

// G and W in FP64: the FP64 table, or the functions themselves outside it
__device__ __noinline__ void pair_fp64(const double *tab, double u, double *g, double *w) {
    const int hi = __double2hiint(u), at = (hi >> 14) - ((1023 + R64_LO) << 6);
    if ((unsigned)at < (unsigned)R64_INTERVALS) {
        const double t = u - __hiloint2double((hi & ~0x3fff) | 0x2000, 0), *q = tab + 16 * at;
        *g = q[7];
        *w = q[15];
        for (int k = 6; k >= 0; --k) {
            *g = fma(*g, t, q[k]);
            *w = fma(*w, t, q[8 + k]);
        }
    } else {
        const double x = sqrt(u);
        *g = erfc(x) / x;
        *w = (*g + 2.0 / sqrt(PI_REF) * exp(-u)) / u;
    }
}

// adds v units to a site's sum, kept as hi 2^32 + lo
__device__ __forceinline__ void sum_add(i64 *p, i64 hi, i64 lo) {
    atomicAdd(reinterpret_cast<unsigned long long *>(p), (unsigned long long)hi);
    atomicAdd(reinterpret_cast<unsigned long long *>(p + 1), (unsigned long long)lo);
}
__device__ __forceinline__ void sum_add(i64 *p, double v) {
    const double h = floor(v * 2.3283064365386963e-10);
    sum_add(p, __double2ll_rn(h), __double2ll_rn(fma(h, -4294967296.0, v)));
}

// A pair the FP64 way: its energy over kappa is returned, its force goes to both sums.
__device__ __noinline__ double slow_pair(const EvalArgs &a, const SysDev &S, i64 y0, i64 y1, i64 y2, i64 qp, i64 qs,
                                         i64 *op, i64 *os) {
    const double n56 = 1.3877787807814457e-17, n62 = 2.168404344971009e-19;
    const double x = (double)y0 * n56, y = (double)y1 * n56, z = (double)y2 * n56;
    const double u = fma(z, z, fma(y, y, x * x));
    if (!(u < S.kappa * S.kappa * S.rc_sq)) return 0.0;
    double g, w;
    pair_fp64(a.real64_tab, u, &g, &w);
    const double qq = (double)qp * n62 * ((double)qs * n62);
    w *= qq * 72057594037927936.0;
    sum_add(op, w * x);
    sum_add(op + 2, w * y);
    sum_add(op + 4, w * z);
    sum_add(os, -(w * x));
    sum_add(os + 2, -(w * y));
    sum_add(os + 4, -(w * z));
    return qq * g;
}

__global__ void __launch_bounds__(32 * RW) k_real64(EvalArgs a, int n_ch) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    RWarp &W = reinterpret_cast<RWarp *>(smem_raw)[threadIdx.x >> 5];
    __shared__ i64 image[3][4];  // n kappa L_d at n + 1, n = -1 .. 1; kappa L_d / 2 at 3
    const int lane = threadIdx.x & 31;
    const Job J = a.jobs[blockIdx.z];
    const SysDev &S = a.sys[J.sys];
    const i64 *sysc = a.real64_sys + 4 * J.sys;
    if (threadIdx.x < 12) {
        const int d = threadIdx.x >> 2, n = (threadIdx.x & 3) - 1;
        // (sides of which r_c does not reach half need no second image, see below)
        image[d][n + 1] = n < 2 ? n * sysc[d] : S.kappa * S.box[d] < 64.0 ? sysc[d] >> 1 : 0x7fffffffffffffffll;
    }
    __syncthreads();
    const int ns = S.n_sites, T = (ns + 31) / 32, tI = blockIdx.x;
    const int i0 = tI * 32 + (threadIdx.x >> 5) * RROWS;
    if (i0 >= ns) return;  // (warps of a block are independent)
    const int maxd = T / 2;
    const int d0 = (int)(((long long)(maxd + 1) * blockIdx.y) / n_ch);
    const int d1 = (int)(((long long)(maxd + 1) * (blockIdx.y + 1)) / n_ch);
    if (d0 >= d1) return;
    const longlong2 *sites = reinterpret_cast<const longlong2 *>(a.sites) + 2 * (size_t)J.site_off;
    const float4 *sites32 = a.sites32 + J.site_off;
    const int nrow = min(RROWS, ns - i0);
    const float L0 = S.boxf[0], L1 = S.boxf[1], L2 = S.boxf[2];
    const float I0 = S.inv_boxf[0], I1 = S.inv_boxf[1], I2 = S.inv_boxf[2];
    const i64 uc = sysc[3];
    // FP32 rounding of two wrapped coordinates, their difference and its image is below
    // 2^-22 of the box in each dimension: r is below r_c plus that where r^2 < r_c^2
    const float lim = sqrtf(S.rc_sqf) * (1.0f + 1e-6f) + 5e-7f * (L0 + L1 + L2), lim2 = lim * lim;
    if (lane < nrow) {
        const longlong2 *o = sites + 2 * (i0 + lane);
        reinterpret_cast<longlong2 *>(&W.si[lane])[0] = o[0];
        reinterpret_cast<longlong2 *>(&W.si[lane])[1] = o[1];
        W.sif[lane] = sites32[i0 + lane];
    }
    // of row lane / 2, every other pair: sums of forces and energies as hi 2^32 + lo
    i64 hx = 0, hy = 0, hz = 0, lx = 0, ly = 0, lz = 0, he = 0, le = 0;
    double e = 0.0;
    for (int d = d0; d < d1; ++d) {
        if ((T % 2 == 0) && d == maxd && d > 0 && tI >= maxd) continue;
        const int j = ((tI + d) % T) * 32 + lane, jm = j / 3;
        longlong2 s0 = make_longlong2(0, 0), s1 = s0;
        float4 fj = make_float4(0.f, 0.f, 0.f, 0.f);
        if (j < ns) {
            s0 = sites[2 * j];
            s1 = sites[2 * j + 1];
            fj = sites32[j];
        }
        __syncwarp();  // the previous visit's copies have been read
        reinterpret_cast<longlong2 *>(&W.sj[lane])[0] = s0;
        reinterpret_cast<longlong2 *>(&W.sj[lane])[1] = s1;
        unsigned mine = 0u;  // the rows that my site passed with
        int cnt = 0;
        __syncwarp();
        for (int r = 0; r < RROWS; ++r) {
            bool hit = false;
            int img = 0;
            if (r < nrow) {
                const float4 p = W.sif[r];
                float dx = p.x - fj.x, dy = p.y - fj.y, dz = p.z - fj.z;
                const float nx = rintf(dx * I0), ny = rintf(dy * I1), nz = rintf(dz * I2);
                dx = fmaf(-L0, nx, dx);
                dy = fmaf(-L1, ny, dy);
                dz = fmaf(-L2, nz, dz);
                hit = fmaf(dx, dx, fmaf(dy, dy, dz * dz)) < lim2 && j < ns && __float_as_int(p.w) != jm &&
                      (d > 0 || j > i0 + r);
                img = ((int)nx + 1) | ((int)ny + 1) << 2 | ((int)nz + 1) << 4;
            }
            const unsigned m = __ballot_sync(0xffffffffu, hit);
            if (hit) {
                W.code[cnt + __popc(m & ((1u << lane) - 1u))] = (unsigned short)(img << 9 | r << 5 | lane);
                mine |= 1u << r;
            }
            if (lane == 0) {
                W.mask[r] = m;
                W.off[r] = cnt;
            }
            cnt += __popc(m);
        }
        if (lane == 0) W.off[RROWS] = cnt;
        __syncwarp();
        for (int b = lane; b < cnt; b += 32) {
            const int c = W.code[b], img = c >> 9;
            const RSite &p = W.si[(c >> 5) & 15], &s = W.sj[c & 31];
            const i64 y0 = p.y[0] - s.y[0] - image[0][img & 3], y1 = p.y[1] - s.y[1] - image[1][(img >> 2) & 3],
                      y2 = p.y[2] - s.y[2] - image[2][(img >> 4) & 3];
            // u in units of 2^-56; a fixed-point pair has u in [2^RI_LO, 2^(RI_LO + RI_OCT))
            const i64 u = sqr62(split62(y0 * 8)) + sqr62(split62(y1 * 8)) + sqr62(split62(y2 * 8));
            i64 fx = 0, fy = 0, fz = 0;
            if (u < uc && (unsigned)((int)(u >> 32) - RI_BOT) < (unsigned)(RI_TOP - RI_BOT)) {
                const int z = __clz((int)(u >> 32));
                const i64 n = (i64)((unsigned long long)u << z);  // the top bit at 63
                const int oct = 63 - 56 - RI_LO - z, at = oct << 6 | ((int)(n >> 57) & 63);
                const longlong2 *q = reinterpret_cast<const longlong2 *>(a.real64_int + 12 * at);
                const longlong2 w01 = __ldg(q), w23 = __ldg(q + 1), g01 = __ldg(q + 3), g23 = __ldg(q + 4);
                const int4 w47 = __ldg(reinterpret_cast<const int4 *>(q + 2)), g47 = __ldg(reinterpret_cast<const int4 *>(q + 5));
                const i64 t = (i64)((unsigned long long)(n << 7) >> 2) - (1ll << 61);
                const Limbs tl = split62(t);
                const int t32 = (int)(t >> 30);
                const Limbs qq = split62(mul62x(split62(p.q), split62(s.q)));
                const i64 eg = mul62x(qq, split62(horner(g01, g23, g47, tl, t32)));
                he += eg >> 32;
                le += (unsigned)eg;
                const Limbs w = split62(mul62x(qq, split62(horner(w01, w23, w47, tl, t32))));
                const int up = oct == 0 ? 5 : 3;  // the lowest octave's W has two bits less
                fx = mul62(w, split62(y0 << up));
                fy = mul62(w, split62(y1 << up));
                fz = mul62(w, split62(y2 << up));
            } else {
                // too near, or beyond r_c: the screen's margin lets in some pairs (one in 10^5),
                // and of a pair 1e-7 of a side from half a box its FP32 image may be the farther
                // one, where r_c reaches half the shortest side. Decided in FP64
                const auto nearer = [](i64 y, const i64 *im) { return y > im[3] ? y - im[2] : y < -im[3] ? y + im[2] : y; };
                i64 *rf = a.rfix + 6 * (size_t)J.site_off;
                e += slow_pair(a, S, nearer(y0, image[0]), nearer(y1, image[1]), nearer(y2, image[2]), p.q, s.q,
                               rf + 6 * (i0 + ((c >> 5) & 15)), rf + 6 * (((tI + d) % T) * 32 + (c & 31)));
            }
            W.f[0][b] = fx;
            W.f[1][b] = fy;
            W.f[2][b] = fz;
        }
        __syncwarp();
        // a pair's force is below 8 of its 2^56 units: sixteen of them add up in 64 bits
        i64 sx = 0, sy = 0, sz = 0;
        for (int b = W.off[lane / RLANES] + lane % RLANES; b < W.off[(lane / RLANES) + 1]; b += RLANES) {
            sx += W.f[0][b];
            sy += W.f[1][b];
            sz += W.f[2][b];
        }
        hx += sx >> 32;
        hy += sy >> 32;
        hz += sz >> 32;
        lx += (unsigned)sx;
        ly += (unsigned)sy;
        lz += (unsigned)sz;
        if (mine) {
            i64 vx = 0, vy = 0, vz = 0;
            for (unsigned m = mine; m; m &= m - 1) {
                const int r = __ffs(m) - 1, b = W.off[r] + __popc(W.mask[r] & ((1u << lane) - 1u));
                vx -= W.f[0][b];
                vy -= W.f[1][b];
                vz -= W.f[2][b];
            }
            i64 *o = a.rfix + 6 * ((size_t)J.site_off + j);
            sum_add(o, vx >> 32, (unsigned)vx);
            sum_add(o + 2, vy >> 32, (unsigned)vy);
            sum_add(o + 4, vz >> 32, (unsigned)vz);
        }
    }
    for (int o = 1; o < RLANES; o <<= 1) {
        hx += __shfl_xor_sync(0xffffffffu, hx, o);
        hy += __shfl_xor_sync(0xffffffffu, hy, o);
        hz += __shfl_xor_sync(0xffffffffu, hz, o);
        lx += __shfl_xor_sync(0xffffffffu, lx, o);
        ly += __shfl_xor_sync(0xffffffffu, ly, o);
        lz += __shfl_xor_sync(0xffffffffu, lz, o);
    }
    if (lane % RLANES == 0 && (lane / RLANES) < nrow) {
        i64 *o = a.rfix + 6 * ((size_t)J.site_off + i0 + (lane / RLANES));
        sum_add(o, hx, lx);
        sum_add(o + 2, hy, ly);
        sum_add(o + 4, hz, lz);
    }
    e = warp_sum(fma((double)he, 3.725290298461914e-09, fma((double)le, 8.673617379884035e-19, e)));
    if (lane == 0) atomicAdd(&a.energy[J.slot], S.kappa * S.q_top * S.q_top * e);
}

}  // namespace

void init_real64_attributes() {
    cudaFuncSetAttribute(k_real64, cudaFuncAttributeMaxDynamicSharedMemorySize, RW * (int)sizeof(RWarp));
}

// Chunks of ring distances: some eight blocks an SM, about a wave. More and shorter ones
// keep their slots from the kernels beside this one (with twenty-four: a Suzuki-Chin call of
// 216 waters, 8 beads 407 us against 390, FP64 forces of 336 waters, 8 beads 281 against 267, a
// step of 216 waters, 32 beads 411 against 398; with four the last two 284 and 409).
void launch_real64(const EvalArgs &a, cudaStream_t s) {
    const int T = (3 * a.max_mols + 31) / 32;
    const long long blocks = (long long)T * a.n_jobs, want = 152LL * 8;
    int n_ch = a.tune_rj > 0 ? a.tune_rj : (int)std::min<long long>(MAX_RJ, (want + blocks - 1) / blocks);
    n_ch = std::max(1, std::min(n_ch, T / 2 + 1));
    k_real64<<<dim3(T, n_ch, a.n_jobs), 32 * RW, RW * sizeof(RWarp), s>>>(a, n_ch);
}

}  // namespace qtg
