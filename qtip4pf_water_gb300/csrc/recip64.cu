// Site preparation and reciprocal-space Ewald of the FP64 form (replaces
// forces.cpp:180-448, :558-564).
//
// What bounds it: this GPU issues a warp's FP64 multiply-add in sixteen cycles of an
// SM, but a 32 x 32 -> 64-bit integer multiply-add in half a cycle, and everything
// that is multiplied here is bounded: phases lie in [-1, 1] and a batch's force weights
// can be scaled to it. So the two contractions (sites with k-vectors and back) run in
// 55-bit fixed point: a value v is round(v 2^55) = h 2^28 + l with signed 28-bit limbs,
// and a product is three integer multiply-adds into 64-bit sums,
//     hh += h h',   mid += h l' + l h'      (l l' <= 2^-56 and of both signs: left out),
// worth hh 2^-54 + mid 2^-82. Quantising is accurate to 2^-56 and the sums are exact,
// where the 53-bit multiply-adds they replace round every partial sum. 216 waters, 32 beads: structure factors 430 us, forces 731 us with FP64
// multiply-adds; the launchers state these kernels' times.
#include <math.h>

#include <algorithm>

#include "fixed62.h"
#include "qtg_internal.h"

namespace qtg {

namespace {

constexpr double TWO55 = 36028797018963968.0, IN54 = 2.0 / TWO55, IN82 = IN54 / 268435456.0;
constexpr int HALF = 1 << 26;  // half a unit of 2^-55 in units of 2^-82

// limbs of a value in units of 2^-55
__device__ __forceinline__ void limbs(i64 v, int &h, int &l) {
    h = (int)((v + (1 << 27)) >> 28);
    l = (int)((unsigned)v - ((unsigned)h << 28));
}
__device__ __forceinline__ int4 complex_limbs(double re, double im) {
    int4 o;
    limbs(__double2ll_rn(re * TWO55), o.x, o.y);
    limbs(__double2ll_rn(im * TWO55), o.z, o.w);
    return o;
}
// A = X Y (complex, limbs in and out; Y conjugated where s < 0)
__device__ __forceinline__ void column_factor(const int4 &x, const int4 &y, int s, int &rh, int &rl, int &ih, int &il) {
    const int yh = s * y.z, yl = s * y.w;
    const i64 r = madw(x.x, y.x, madw(-x.z, yh, 0));
    const i64 rm = madw(x.x, y.y, madw(x.y, y.x, madw(-x.z, yl, madw(-x.w, yh, HALF))));
    const i64 i = madw(x.x, yh, madw(x.z, y.x, 0));
    const i64 im = madw(x.x, yl, madw(x.y, yh, madw(x.z, y.y, madw(x.w, y.x, HALF))));
    limbs(r * 2 + (rm >> 27), rh, rl);
    limbs(i * 2 + (im >> 27), ih, il);
}

// Cosines and sines of the middles of 256 parts of a turn, units of 2^-62 (Taylor series on
// the first eighth, evaluated by the compiler in 128-bit integers; the others by symmetry).
struct TurnTable {
    i64 v[512];
};
constexpr i64 mul_r62(i64 a, i64 b) { return (i64)(((__int128)a * b + ((__int128)1 << 61)) >> 62); }
constexpr TurnTable make_turn_table() {
    TurnTable T{};
    for (int i = 0; i < 32; ++i) {
        const i64 ph = (i64)(((__int128)14488038916154245685ull * (2 * i + 1)) >> 8);  // pi 2^62 (2 i + 1) / 256
        const i64 sq = mul_r62(ph, ph);
        i64 c = 0, s = 0;
        for (int k = 10; k >= 1; --k) {
            const i64 one = (1ll << 62) - 1;
            c = -mul_r62(sq, one + c) / ((2 * k - 1) * (2 * k));
            s = -mul_r62(sq, one + s) / ((2 * k) * (2 * k + 1));
        }
        const i64 co = ((1ll << 62) - 1) + c, si = ph + mul_r62(ph, s);
        for (int o = 0; o < 4; ++o) {  // i + 64 o, and its mirror image in the quadrant
            const i64 u[4][2] = {{co, si}, {-si, co}, {-co, -si}, {si, -co}}, w[4][2] = {{si, co}, {-co, si}, {-si, -co}, {co, -si}};
            for (int k = 0; k < 2; ++k) {
                T.v[2 * (64 * o + i) + k] = u[o][k];
                T.v[2 * (64 * o + 63 - i) + k] = w[o][k];
            }
        }
    }
    return T;
}
__device__ const TurnTable turn_table = make_turn_table();

// exp(i 2 pi a / 2^64) in limbs. The turn is cut into 256 parts, whose middles' cosines and
// sines are tabled in units of 2^-62; the rest, |th| <= pi/256, goes through Taylor series
// to th^7, the leading terms in 62-bit products and the others in 32 bits (absolute errors
// below 2^-58).
__device__ __forceinline__ int4 turn_limbs(unsigned long long a) {
    const longlong2 cs = make_longlong2(turn_table.v[2 * (int)(a >> 56)], turn_table.v[2 * (int)(a >> 56) + 1]);
    const Limbs C = split62(cs.x), S = split62(cs.y);
    const i64 d = (i64)(a << 8 >> 8) - (1ll << 55);          // units of 2^-64 of a turn
    const i64 T = mul62(split62(d << 6), split62(3622009729038561421ll));  // th 2^67: pi / 2 in units of 2^-61
    const Limbs t = split62(T);
    const i64 z = sqr62(t);                                  // th^2 2^72
    const int w = (int)(z >> 29);                            // th^2 2^43
    // cos th - 1 = -th^2 / 2 + th^2 (th^2 (1/24 - th^2 / 720)), times 2^75
    const int i24 = 1431655765 - (int)(((i64)w * 23302) >> 32), x = (int)(((i64)w * i24) >> 31);
    const Limbs cm = split62(((i64)w * x >> 15) - 4 * z);
    // sin th = th - th (th^2 (1/6 - th^2 (1/120 - th^2 / 5040))), times 2^67
    const int i120 = 1145324612 - (int)(((i64)w * 13316) >> 32);
    const i64 y = mul62(split62(z), split62(1537228672809129301ll - ((i64)w * i120 >> 17)));
    const Limbs sn = split62(T - (mul62(t, split62(y)) >> 11));
    const i64 co = cs.x + (mul62(C, cm) >> 13) - (mul62(S, sn) >> 5);
    const i64 si = cs.y + (mul62(S, cm) >> 13) + (mul62(C, sn) >> 5);
    int4 o;
    limbs((co + 64) >> 7, o.x, o.y);
    limbs((si + 64) >> 7, o.z, o.w);
    return o;
}

__device__ __forceinline__ bool not_finite(double v) { return (__double2hiint(v) & 0x7ff00000) == 0x7ff00000; }
__host__ __device__ __forceinline__ int prep64_blocks(int max_mols) { return 3 * ((3 * max_mols + 127) / 128); }

// ---- k_prep64 -----------------------------------------------------------------------
// One thread per (site, dimension), blocks dimension-major as k_prep_f32: charge site
// (M, H1, H2) wrapped into the box in k_real64's fixed point, wrapped oxygen, zeroed sums, and the site's row of
// phases exp(i 2 pi m s_d), m = 0 .. k_max: powers 1, 2 and the multiples of four from the
// 64-bit fraction of s_d, whose multiples are exact, the others as products of those in
// limbs. The x row carries the charge over q_scale. (With the FP64 sincospi the kernel was
// bound by its FP64 instructions: 216 waters, 32 beads 30 us, 14.4 here; 64 waters, 1 bead,
// all latency, 12.4 and 8.3. The force's error against 80-bit sums falls from 2.0e-15 to 6.4e-16.)
// Fixed point has no NaN: a block that met a coordinate or charge that is not finite says so
// in its word of a.nonfinite, from which k_sk_reduce64 makes the whole configuration's
// reciprocal energy and forces NaN, as sums of such phases are.
__global__ void __launch_bounds__(128) k_prep64(EvalArgs a) {
    const Job J = a.jobs[blockIdx.y];
    const SysDev &S = a.sys[J.sys];
    const int ns = S.n_sites;
    const int tiles = (3 * a.max_mols + 127) / 128;
    const int d = blockIdx.x / tiles, s = (blockIdx.x - d * tiles) * 128 + threadIdx.x;
    if (s == 0 && d == 0) a.energy[J.slot] = 0.0;
    const int mol = s / 3, kind = s - 3 * mol;
    const double *q = a.pos + J.pos_off;
    const double g = a.c.gamma_vs;
    const bool own = s < ns;
    double x = 0.0;
    if (own && (a.sites_are_input || kind != 0)) {
        x = q[3 * s + d];
    } else if (own) {
        // M site (forces.cpp:558-564)
        x = g * q[9 * mol + d] + 0.5 * (1.0 - g) * (q[9 * mol + 3 + d] + q[9 * mol + 6 + d]);
        const double t = q[9 * mol + d] * S.inv_box[d];
        const size_t at = 4 * ((size_t)J.site_off / 3 + mol) + d;
        reinterpret_cast<float *>(a.opos32)[at] = (float)((t - floor(t)) * S.box[d]);
        a.lj64[at] = 0.0;  // k_lj64's forces
    }
    const double chg = d == 0 && own ? a.charge[S.chg_off + s] : 0.0;
    const int bad = __syncthreads_or(not_finite(x) || not_finite(chg));
    if (threadIdx.x == 0) a.nonfinite[(size_t)J.slot * gridDim.x + blockIdx.x] = bad;
    if (!own) return;
    // wrapped with one rounding (while the quotient is exact enough for it), and the 64-bit
    // fraction of the box
    const double t = x * S.inv_box[d];
    const double wr = fabs(t) < 1e9 ? fma(-floor(t), S.box[d], x) : (t - floor(t)) * S.box[d];
    const double fh = wr * S.inv_box[d], fl = fma(-fh, S.box[d], wr) * S.inv_box[d];
    const unsigned long long frac = ((unsigned long long)__double2ll_rn(fh * 4611686018427387904.0) << 2) +
                                    (unsigned long long)__double2ll_rn(fl * 18446744073709551616.0);
    if (a.sites32) {  // k_real64's form of the site (reciprocal space alone may have none)
        i64 *sv = reinterpret_cast<i64 *>(a.sites) + 4 * ((size_t)J.site_off + s);
        sv[d] = kappa_fix(S.kappa, wr);
        float *sf = reinterpret_cast<float *>(a.sites32 + (size_t)J.site_off + s);
        sf[d] = (float)wr;
        if (d == 0) {
            const double h = chg * S.inv_q_top, l = fma(-h, S.q_top, chg) * S.inv_q_top, two62 = 4611686018427387904.0;
            sv[3] = __double2ll_rn(h * two62) + __double2ll_rn(l * two62);
            sf[3] = __int_as_float(mol);
        }
        // its sums start from nothing
        i64 *rf = a.rfix + 6 * ((size_t)J.site_off + s) + 2 * d;
        rf[0] = rf[1] = 0;
    }
    const int km1 = S.k_max + 1;
    int4 *ph = reinterpret_cast<int4 *>(a.phase) + J.phase_off + (size_t)d * km1 * ns + s;
    auto seed = [&](int m) { return turn_limbs((unsigned long long)m * frac); };
    auto times = [](const int4 &p, const int4 &q) {
        int4 o;
        column_factor(p, q, 1, o.x, o.y, o.z, o.w);
        return o;
    };
    const int4 p1 = seed(1), p2 = seed(2), p3 = times(p2, p1), qd = complex_limbs(d == 0 ? chg * S.inv_q_scale : 1.0, 0.0);
    for (int m = 0; m < km1; m += 4) {
        const int4 b = m ? times(seed(m), qd) : qd;
        ph[(size_t)m * ns] = b;
        if (m + 1 < km1) ph[(size_t)(m + 1) * ns] = times(b, p1);
        if (m + 2 < km1) ph[(size_t)(m + 2) * ns] = times(b, p2);
        if (m + 3 < km1) ph[(size_t)(m + 3) * ns] = times(b, p3);
    }
}

// ---- k_ksk64: structure factors -------------------------------------------------------
// One thread per group of at most KZ |kz| of one column over the half set (kx = 0, ky < 0
// columns left out); with A = X Y and Z the site's phases it sums the four real products
// Ar Zr, Ai Zi, Ar Zi, Ai Zr, from which S(+kz) = T1 - T2 + i (T3 + T4) and S(-kz) =
// T1 + T2 + i (T4 - T3). Sites come through shared memory in chunks of CH64, double-
// buffered by cp.async; mid holds CARRY chunks before its high part moves into hh, and
// hh FLUSH chunks (256 sites) before it goes to FP64: a high limb reaches 2^27 (a scaled
// charge within 2^-28 of 1), so 512 sites in phase would make 2^63.
constexpr int KT64 = 128, CH64 = 32, CARRY = 4, FLUSH = 8;
static_assert((long long)FLUSH * CH64 << 54 <= 1ll << 62, "k_ksk64's high sums overflow");

__device__ __forceinline__ void copy16(void *dst, const void *src, bool valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int n = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(n) : "memory");
}

template <int KZ>
__global__ void __launch_bounds__(KT64) k_ksk64(EvalArgs a) {
    const int sc = blockIdx.y;
    const Job J = a.jobs[blockIdx.z];
    const SysDev &S = a.sys[J.sys];
    const int ng = S.n_grp_half, ns = S.n_sites, km1 = S.k_max + 1;
    if (blockIdx.x * KT64 >= ng) return;
    const int t = blockIdx.x * KT64 + threadIdx.x;
    const bool act = t < ng;
    const int s0 = (int)(((i64)ns * sc) / a.n_sc), s1 = (int)(((i64)ns * (sc + 1)) / a.n_sc);
    extern __shared__ __align__(16) int4 tab64[];  // [2][3 km1][CH64 + 1]
    KGroup G = {0, 0, 0, 0};
    KCol C = {0, 0, 0, 0};
    if (act) {
        G = a.kgrp[S.grp_off + t];
        C = a.kcol[S.col_off + G.col];
    }
    const int xrow = C.kx * (CH64 + 1), yrow = (km1 + abs(C.ky)) * (CH64 + 1), sy = C.ky < 0 ? -1 : 1;
    int zrow[KZ];
#pragma unroll
    for (int g = 0; g < KZ; ++g) zrow[g] = (2 * km1 + min(G.kz0 + g, km1 - 1)) * (CH64 + 1);
    double T[KZ][4];
    i64 H[KZ][4], M[KZ][4];
#pragma unroll
    for (int g = 0; g < KZ; ++g)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            T[g][k] = 0.0;
            H[g][k] = M[g][k] = 0;
        }
    const int4 *ph = reinterpret_cast<const int4 *>(a.phase) + J.phase_off;
    const int rows = 3 * km1, nchunk = s1 > s0 ? (s1 - s0 + CH64 - 1) / CH64 : 0;
    auto stage = [&](int ci) {
        const int c0 = s0 + ci * CH64;
        int4 *tb = tab64 + (ci & 1) * rows * (CH64 + 1);
        for (int idx = threadIdx.x; idx < rows * CH64; idx += KT64) {
            const int row = idx / CH64, c = idx - row * CH64, s = c0 + c;
            copy16(tb + row * (CH64 + 1) + c, ph + (size_t)row * ns + min(s, s1 - 1), s < s1);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    if (nchunk > 0) stage(0);
    for (int ci = 0; ci < nchunk; ++ci) {
        __syncthreads();
        if (ci + 1 < nchunk) stage(ci + 1);
        else asm volatile("cp.async.commit_group;\n" ::: "memory");
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();
        const int4 *tb = tab64 + (ci & 1) * rows * (CH64 + 1);
        const int nc = min(CH64, s1 - s0 - ci * CH64);
#pragma unroll 2
        for (int c = 0; c < nc; ++c) {
            int rh, rl, ih, il;
            column_factor(tb[xrow + c], tb[yrow + c], sy, rh, rl, ih, il);
#pragma unroll
            for (int g = 0; g < KZ; ++g) {
                const int4 z = tb[zrow[g] + c];
                H[g][0] = madw(rh, z.x, H[g][0]);
                M[g][0] = madw(rh, z.y, madw(rl, z.x, M[g][0]));
                H[g][1] = madw(ih, z.z, H[g][1]);
                M[g][1] = madw(ih, z.w, madw(il, z.z, M[g][1]));
                H[g][2] = madw(rh, z.z, H[g][2]);
                M[g][2] = madw(rh, z.w, madw(rl, z.z, M[g][2]));
                H[g][3] = madw(ih, z.x, H[g][3]);
                M[g][3] = madw(ih, z.y, madw(il, z.x, M[g][3]));
            }
        }
        if (ci % CARRY == CARRY - 1) {
#pragma unroll
            for (int g = 0; g < KZ; ++g)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    H[g][k] += M[g][k] >> 28;
                    M[g][k] &= (1 << 28) - 1;
                }
        }
        if (ci % FLUSH == FLUSH - 1 || ci + 1 == nchunk) {
#pragma unroll
            for (int g = 0; g < KZ; ++g)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    T[g][k] += fma((double)H[g][k], IN54, (double)M[g][k] * IN82);
                    H[g][k] = M[g][k] = 0;
                }
        }
    }
    if (!act) return;
    const double qs = S.q_scale;
#pragma unroll
    for (int g = 0; g < KZ; ++g) {
        if (g >= G.n) continue;
        const int az = G.kz0 + g;
        double2 *o = a.skp + (size_t)sc * a.total_k + J.sk_off + C.k_begin + C.m;
        o[az] = make_double2(qs * (T[g][0] - T[g][1]), qs * (T[g][2] + T[g][3]));
        if (az) o[-az] = make_double2(qs * (T[g][0] + T[g][1]), qs * (T[g][3] - T[g][2]));
    }
}

// v 2^(58 - ex) rounded, for |v| < 2^ex, by shifts (an FP64 product and conversion take
// sixteen cycles of an SM each)
__device__ __forceinline__ i64 fix58(double v, int ex) {
    const int hi = __double2hiint(v), e = (hi >> 20) & 0x7ff, s = e - 1017 - ex;
    const i64 m = (i64)((hi & 0xfffff) | 0x100000) << 32 | (unsigned)__double2loint(v);
    const i64 u = e == 0 || s < -54 ? 0 : s >= 0 ? m << s : (m + (1ll << (-s - 1))) >> -s;
    return hi < 0 ? -u : u;
}

// ---- k_sk_reduce64 --------------------------------------------------------------------
// A block per force batch (whole columns, at most 128 vectors), a thread per k: S(k) from
// the site chunks' partials in order, the batch's energy, and the weights W = 2 c_k S(k)
// packed for k_kforce64: with s, d = W(+kz) +- W(-kz), the slot of |kz| holds the limbs
// of (s.x, d.y, d.x, s.y) and of kz / 2^kshift times (d.x, s.y, s.x, d.y), all over the
// power of two above the batch's largest |s|, |d|, whose worth goes to wsk[k0]. (kshift
// keeps kz / 2^kshift below 16 and its sum over a column below 121, so that the limbs
// and k_kforce64's sums fit; it is 0 for k_max <= 15.) Bound by FP64 issue, so that only the
// sums and the weights themselves are FP64 (the packing too: 14.5 us at 216 waters, 32 beads,
// 10.2 here; 512 waters 18.6 and 10.4).
__global__ void __launch_bounds__(128) k_sk_reduce64(EvalArgs a) {
    const Job J = a.jobs[blockIdx.y];
    const SysDev &S = a.sys[J.sys];
    if ((int)blockIdx.x >= S.n_batch_half) return;
    const KBatch B = a.kbatch[S.batch_off + blockIdx.x];
    const int k = B.k0 + threadIdx.x;
    const bool on = k < B.k1;
    __shared__ double2 wl[128];
    __shared__ double red[4];
    __shared__ unsigned top[4];
    double e = 0.0;
    int code = -1;
    // whether a site of the configuration is not finite (k_prep64): on its way during the sums
    const int words = prep64_blocks(a.max_mols);
    const int *nf = a.nonfinite + (size_t)J.slot * words;
    int word = (int)threadIdx.x < words ? nf[threadIdx.x] : 0;
    if (on) {
        const KVec kv = a.kvec[S.kvec_off + k];
        const double w = 2.0 * kv.coef * (kv.twin ? 2.0 : 1.0);  // kx = 0, ky > 0: its conjugate partner too
        double sr = 0.0, si = 0.0;
        for (int sc = 0; sc < a.n_sc; ++sc) {
            const double2 p = a.skp[(size_t)sc * a.total_k + J.sk_off + k];
            sr += p.x;
            si += p.y;
        }
        e = 0.5 * w * (sr * sr + si * si);
        wl[threadIdx.x] = make_double2(w * sr, w * si);
        code = a.kpk[S.kvec_off + k];
    }
    const double nan = __hiloint2double(0x7ff80000, 0);
    for (int i = threadIdx.x + 128; i < words; i += 128) word |= nf[i];
    const bool bad = __syncthreads_or(word);
    if (bad) e = nan;
    const int az = code & 255;
    double sx = 0.0, sy = 0.0, dx = 0.0, dy = 0.0;
    if (code >= 0) {
        const double2 wp = wl[threadIdx.x], wm = az ? wl[threadIdx.x - 2 * az] : make_double2(0.0, 0.0);
        sx = wp.x + wm.x;
        sy = wp.y + wm.y;
        dx = wp.x - wm.x;
        dy = wp.y - wm.y;
    }
    // the largest magnitude's exponent, from the high words
    const auto high = [](double v) { return (unsigned)__double2hiint(v) & 0x7fffffffu; };
    unsigned m = max(max(high(sx), high(sy)), max(high(dx), high(dy)));
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) top[threadIdx.x >> 5] = m;
    const double te = block_sum(e, red);  // (its barriers also publish top)
    if (threadIdx.x == 0) atomicAdd(&a.energy[J.slot], te);
    m = max(max(top[0], top[1]), max(top[2], top[3]));
    // every value < 2^ex; tiny batches (all weights zero or subnormal) take the smallest scale kept
    const int ex = max((int)(m >> 20) - 1022, -900);
    const double scale = __hiloint2double((1023 + ex) << 20, 0), inv = __hiloint2double((1023 - ex) << 20, 0);
    if (threadIdx.x == 0) a.wsk64[J.sk_off + B.k0] = make_double2(bad ? nan : scale, 0.0);
    if (code < 0) return;
    int4 *o = reinterpret_cast<int4 *>(a.wpk) + 4 * ((size_t)J.sk_off + B.k0 + (code >> 8));
    const i64 isx = fix58(sx, ex), isy = fix58(sy, ex);
    const auto pack = [](i64 re, i64 im) {
        int4 v;
        limbs((re + 4) >> 3, v.x, v.y);
        limbs((im + 4) >> 3, v.z, v.w);
        return v;
    };
    if (az == 0) {
        o[0] = pack(isx, isy);
        return;
    }
    const i64 idx = fix58(dx, ex), idy = fix58(dy, ex);
    o[0] = pack(isx, idy);
    o[1] = pack(idx, isy);
    if (a.kshift == 0) {  // az <= 15
        o[2] = pack(idx * az, isy * az);
        o[3] = pack(isx * az, idy * az);
        return;
    }
    const double f = inv * az * __hiloint2double((1023 - a.kshift) << 20, 0);
    o[2] = complex_limbs(dx * f, sy * f);
    o[3] = complex_limbs(sx * f, dy * f);
}

// ---- k_kforce64: reciprocal-space site forces -------------------------------------------
// One thread per site, batches of whole columns (see k_kforce_f32 for the sums U1 .. U4
// and how the column's A enters once). U keeps units of 2^-55 and v = pi U1 + pr U2 of 2^-54 in 64
// bits (|U1|, |U2| < 2^6.5 for k_max <= 62, |U3|, |U4| < 2^7.5); the sums of kx v, ky v
// and vz over a batch are kept as two 64-bit integers each (above and below bit 31) and
// go to FP64 once a batch.
constexpr int FT64 = 128;

// a u + b w in units of 2^-54: a, b in limbs, u, w (units of 2^-55) split at bit SH
template <int SH>
__device__ __forceinline__ i64 close_pair(int ah, int al, i64 u, int bh, int bl, i64 w) {
    const int uh = (int)((u + (1ll << (SH - 1))) >> SH), ul = (int)(u - ((i64)uh << SH));
    const int wh = (int)((w + (1ll << (SH - 1))) >> SH), wl = (int)(w - ((i64)wh << SH));
    const i64 hh = madw(ah, uh, madw(bh, wh, 0));                                // units of 2^(SH - 82)
    const i64 m1 = madw(al, uh, madw(bl, wh, 0));                                // 2^(SH - 110)
    const i64 m2 = madw(ah, ul, madw(bh, wl, 1 << 27));                          // 2^-82
    const i64 ll = madw(al, ul, madw(bl, wl, 0));                                // 2^-110
    return (hh << (SH - 28)) + (((m1 << (SH - 28)) + m2 + (ll >> 28)) >> 28);
}

__global__ void __launch_bounds__(FT64) k_kforce64(EvalArgs a) {
    const int kc = blockIdx.y;
    const Job J = a.jobs[blockIdx.z];
    const SysDev &S = a.sys[J.sys];
    const int nb = S.n_batch_half, ns = S.n_sites, km1 = S.k_max + 1;
    if (blockIdx.x * FT64 >= ns) return;
    const int i = blockIdx.x * FT64 + threadIdx.x;
    const bool act = i < ns;
    const int ii = act ? i : 0;
    const int bt0 = (int)(((i64)nb * kc) / a.n_kc), bt1 = (int)(((i64)nb * (kc + 1)) / a.n_kc);
    __shared__ int4 P[128][4];
    __shared__ int4 cs[128];
    extern __shared__ __align__(16) int4 zr64[];  // [km1][FT64]: this block's sites' Z rows
    const int4 *ph = reinterpret_cast<const int4 *>(a.phase) + J.phase_off + ii;
    for (int m = 0; m < km1; ++m) zr64[m * FT64 + threadIdx.x] = ph[(size_t)(2 * km1 + m) * ns];
    const double bx = 2.0 * PI_REF * S.inv_box[0], by = 2.0 * PI_REF * S.inv_box[1];
    const double bz = 2.0 * PI_REF * S.inv_box[2] * __hiloint2double((1023 + a.kshift) << 20, 0);
    const int4 *wpk = reinterpret_cast<const int4 *>(a.wpk) + 4 * (size_t)J.sk_off;
    double Fx = 0.0, Fy = 0.0, Fz = 0.0;
    for (int bt = bt0; bt < bt1; ++bt) {
        const KBatch B = a.kbatch[S.batch_off + bt];
        const int ncol = B.c1 - B.c0;
        __syncthreads();
        for (int idx = threadIdx.x; idx < ncol; idx += FT64) cs[idx] = a.kfc[S.col_off + B.c0 + idx];
        for (int idx = threadIdx.x; idx < 4 * (B.k1 - B.k0); idx += FT64) P[idx >> 2][idx & 3] = wpk[4 * B.k0 + idx];
        const double scale = a.wsk64[J.sk_off + B.k0].x * S.q_scale * IN54;
        __syncthreads();
        i64 xh = 0, xl = 0, yh = 0, yl = 0, zh = 0, zl = 0;
        for (int cc = 0; cc < ncol; ++cc) {
            const int4 C = cs[cc];
            int rh, rl, ih, il;
            column_factor(ph[(size_t)C.x * ns], ph[(size_t)(km1 + abs(C.y)) * ns], C.y < 0 ? -1 : 1, rh, rl, ih, il);
            const int4 w0 = P[C.w][0];
            i64 h1 = (i64)w0.x << 27, m1 = ((i64)w0.y << 27) + HALF;
            i64 h2 = -((i64)w0.z << 27), m2 = HALF - ((i64)w0.w << 27);
            i64 h3 = 0, m3 = HALF, h4 = 0, m4 = HALF;
            for (int az = 1; az <= C.z; ++az) {
                const int4 z = zr64[az * FT64 + threadIdx.x];
                const int4 p = P[C.w + az][0], q = P[C.w + az][1], r = P[C.w + az][2], s = P[C.w + az][3];
                const int nh = -z.x, nl = -z.y;
                h1 = madw(z.x, p.x, madw(z.z, p.z, h1));
                m1 = madw(z.x, p.y, madw(z.y, p.x, madw(z.z, p.w, madw(z.w, p.z, m1))));
                h2 = madw(z.z, q.x, madw(nh, q.z, h2));
                m2 = madw(z.z, q.y, madw(z.w, q.x, madw(nh, q.w, madw(nl, q.z, m2))));
                h3 = madw(z.x, r.x, madw(z.z, r.z, h3));
                m3 = madw(z.x, r.y, madw(z.y, r.x, madw(z.z, r.w, madw(z.w, r.z, m3))));
                h4 = madw(z.z, s.x, madw(nh, s.z, h4));
                m4 = madw(z.z, s.y, madw(z.w, s.x, madw(nh, s.w, madw(nl, s.z, m4))));
            }
            const i64 v = close_pair<31>(ih, il, h1 * 2 + (m1 >> 27), rh, rl, h2 * 2 + (m2 >> 27));
            const i64 vz = close_pair<32>(ih, il, h3 * 2 + (m3 >> 27), rh, rl, h4 * 2 + (m4 >> 27));
            const int vh = (int)(v >> 31), vl = (int)((unsigned)v & 0x7fffffffu);
            xh = madw(C.x, vh, xh);
            xl = madw(C.x, vl, xl);
            yh = madw(C.y, vh, yh);
            yl = madw(C.y, vl, yl);
            zh += vz >> 31;
            zl += vz & 0x7fffffffll;
        }
        Fx = fma(bx * scale, fma((double)xh, 2147483648.0, (double)xl), Fx);
        Fy = fma(by * scale, fma((double)yh, 2147483648.0, (double)yl), Fy);
        Fz = fma(bz * scale, fma((double)zh, 2147483648.0, (double)zl), Fz);
    }
    if (act) {
        double *o = a.part + 3 * ((size_t)(a.n_rj + kc) * a.total_sites + J.site_off + i);
        o[0] = Fx;
        o[1] = Fy;
        o[2] = Fz;
    }
}

size_t ksk64_smem(int kmax) { return (size_t)2 * 3 * (kmax + 1) * (CH64 + 1) * sizeof(int4); }
size_t kforce64_smem(int kmax) { return (size_t)(kmax + 1) * FT64 * sizeof(int4); }

}  // namespace

void init_recip64_attributes() {
    const int big = 200 * 1024;
    cudaFuncSetAttribute(k_ksk64<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
    cudaFuncSetAttribute(k_ksk64<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
    cudaFuncSetAttribute(k_kforce64, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
}

void launch_prep64(const EvalArgs &a, cudaStream_t s) {
    k_prep64<<<dim3(prep64_blocks(a.max_mols), a.n_jobs), 128, 0, s>>>(a);
}
// 216 waters, 32 beads: 430 us with FP64 multiply-adds, 99 us here; 512 waters: 309 us.
// Against a long-double sum the forces are as near as before (64 waters: 2.0e-15 and
// 1.9e-15 relative); 54 bits instead of 55 had 2.5e-15, |kz| weights scaled by 1/16 6e-15.
void launch_ksk64(const EvalArgs &a, cudaStream_t s) {
    const dim3 g((a.max_grp + KT64 - 1) / KT64, a.n_sc, a.n_jobs);
    if (a.kz == 3) k_ksk64<3><<<g, KT64, ksk64_smem(a.max_kmax), s>>>(a);
    else k_ksk64<4><<<g, KT64, ksk64_smem(a.max_kmax), s>>>(a);
}
void launch_sk_reduce64(const EvalArgs &a, cudaStream_t s) {
    k_sk_reduce64<<<dim3(a.max_batch, a.n_jobs), 128, 0, s>>>(a);
}
// 216 waters, 32 beads: 731 us with FP64 multiply-adds, 109 us here; 512 waters: 315 us
void launch_kforce64(const EvalArgs &a, cudaStream_t s) {
    k_kforce64<<<dim3((3 * a.max_mols + FT64 - 1) / FT64, a.n_kc, a.n_jobs), FT64, kforce64_smem(a.max_kmax), s>>>(a);
}

}  // namespace qtg
