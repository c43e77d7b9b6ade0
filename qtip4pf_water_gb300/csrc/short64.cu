// Short-range terms of the FP64 form: O-O Lennard-Jones over the Verlet list
// (forces.cpp:25-59, :489-515), the intramolecular terms, and the sum of a molecule's
// forces.
//
// Lennard-Jones: one warp per list row. What bounds it is FP64 issue (a warp's FP64 instruction takes
// sixteen cycles of an SM), and of the list's pairs, which reach to r_skin = 1.3 r_cut,
// only 45 % lie inside r_cut. So the entries are screened in FP32 on wrapped positions,
// with a margin above their rounding, and the pairs that pass are packed into full warps
// before anything is done in FP64: 216 waters, 32 beads 151 us for the former kernel,
// which took every entry's image and cutoff in FP64, 66 us with the screen. Of the 40 FP64
// instructions a pair then took, image and cutoff tests now read the high words, the
// reciprocal is two Newton steps from an FP32 one, constants wait for the row's sums, and
// these take six additions instead of twenty: 51 us (512 waters: 138 -> 105).
//
// The pair's displacement and the cutoff decision r^2 < r_cut^2 are the reference's: a
// pair within 1e-12 of the cutoff, or near half a box in some dimension (where the two
// images tie and the rounding rule picks the sign), is recomputed with its arithmetic
// (x - L round(x / L), each operation rounded).
//
// FULL: the stepper's symmetric list; a row's force needs no atomics and the energy is
// halved. Else the caller's half list (entries j > i), forces added by atomics. The oxygen
// forces go to their own array, which k_combine64 adds, so that the kernel can run beside
// the Ewald kernels.
#include <math.h>

#include "qtg_internal.h"

namespace qtg {

namespace {

// Wrapped FP32 oxygens and cleared forces, where no preparation pass made them (the
// displaced configurations of the Suzuki-Chin force gradient).
__global__ void __launch_bounds__(128) k_lj64_prep(EvalArgs a) {
    const Job J = a.jobs[blockIdx.y];
    const SysDev &S = a.sys[J.sys];
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= S.n_mols) return;
    float w[3];
    for (int d = 0; d < 3; ++d) {
        const double t = a.pos[J.pos_off + 9 * m + d] * S.inv_box[d];
        w[d] = (float)((t - floor(t)) * S.box[d]);
        a.lj64[4 * ((size_t)J.site_off / 3 + m) + d] = 0.0;
    }
    a.opos32[J.site_off / 3 + m] = make_float4(w[0], w[1], w[2], 0.f);
}

// The float at or below |x| in magnitude, to 2^-20, from x's high word: a conversion
// instruction takes as long as an FP64 one.
__device__ __forceinline__ float float_of(double x) {
    const int hi = __double2hiint(x), m = (hi & 0x7fffffff) - (896 << 20);  // exponent bias 1023 to 127
    return m < (1 << 20) ? 0.0f : __int_as_float((hi & 0x80000000) | min(m, (255 << 20) - 1) << 3);
}

template <int FULL>
__global__ void __launch_bounds__(128) k_lj64(EvalArgs a) {
    const Job J = a.jobs[blockIdx.y];
    const SysDev &S = a.sys[J.sys];
    const int N = S.n_mols;
    if (blockIdx.x * 4 >= N) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, i = blockIdx.x * 4 + w;
    __shared__ int queue[4][64];
    __shared__ double red[4];
    double e = 0.0;
    const Consts &C = a.c;
    const double rc2 = C.r_cut_sq;
    if (i < (FULL ? N : N - 1)) {
        const double *q = a.pos + J.pos_off;
        const int cap = FULL ? 2 * S.list_size : S.list_size;
        const int *pt = FULL ? a.point_full + S.pf_off + (size_t)J.bead * (N + 1) : a.point + S.pt_off + (size_t)J.bead * N;
        const int *ls = FULL ? a.list_full + S.lf_off + (size_t)J.bead * cap : a.list + S.ls_off + (size_t)J.bead * cap;
        // a row outside [0, capacity] (overflowed or caller-corrupted list) or an index
        // outside the row's range is skipped and flagged instead of being read out of bounds
        int n0 = pt[i], n1 = pt[i + 1];
        if (n0 < 0 || n1 > cap || n0 > n1) {
            if (lane == 0) atomicOr(a.status, (unsigned)ST_LIST_OVERFLOW);
            n0 = max(0, min(n0, cap));
            n1 = max(n0, min(n1, cap));
        }
        const float4 *opos = a.opos32 + J.site_off / 3;
        double *plane = a.lj64 + 4 * ((size_t)J.site_off / 3);
        const float4 oi = opos[i];
        const double xi[3] = {q[9 * i], q[9 * i + 1], q[9 * i + 2]};
        const float L[3] = {S.boxf[0], S.boxf[1], S.boxf[2]}, I[3] = {S.inv_boxf[0], S.inv_boxf[1], S.inv_boxf[2]};
        const float lim = C.ljf[6] * (1.0f + 1e-6f) + 5e-7f * (L[0] + L[1] + L[2]), lim2 = lim * lim;
        double f0 = 0.0, f1 = 0.0, f2 = 0.0, el = 0.0;
        int npair = 0;
        const int rc2h = __double2hiint(rc2);
        auto pair = [&](int j) {
            const double *qj = q + 9 * j;
            double r[3], r2 = 0.0;
            bool exact = false;
            for (int d = 0; d < 3; ++d) {
                const double x = xi[d] - qj[d];
                const float t = float_of(x) * I[d], n = rintf(t);
                // (the quotient is good to 2^-19: a hundred boxes apart that is a fifth of the margin)
                exact |= fabsf(fabsf(t - n) - 0.5f) < 1e-3f || fabsf(t) > 100.0f;
                r[d] = n == 0.0f ? x : x - (n == 1.0f ? S.box[d] : n == -1.0f ? -S.box[d] : S.box[d] * (double)n);
                r2 = fma(r[d], r[d], r2);
            }
            // near the cutoff: the high words' last place is 2^-20 of the value
            if (exact || abs(__double2hiint(r2) - rc2h) <= 1) r2 = lj_exact_disp(xi, qj, S, r);
            if (!(__double_as_longlong(r2) < __double_as_longlong(rc2))) return;  // (both are positive)
            // 1 / r^2 by Newton's iteration for the reciprocal from an FP32 start
            // (2^-19, then 2^-38, then rounding)
            const float r2f = float_of(r2);
            const int b = __float_as_int(1.0f / r2f);
            double i2 = __hiloint2double((b >> 3) + (896 << 20), b << 29);
            i2 = fma(fma(-r2, i2, 1.0), i2, i2);
            i2 = fma(fma(-r2, i2, 1.0), i2, i2);
            if (r2f < 1e-30f) i2 = 1.0 / r2;
            const double s6 = i2 * i2 * i2 * C.sigmalj6, s12 = s6 * s6, en = s12 - s6;
            el += en;
            ++npair;
            const double ff = (en + s12) * i2;
            f0 = fma(ff, r[0], f0);
            f1 = fma(ff, r[1], f1);
            f2 = fma(ff, r[2], f2);
            if (!FULL) {
                const double fn = -24.0 * C.epslj * ff;
                for (int d = 0; d < 3; ++d) atomicAdd(plane + 4 * j + d, fn * r[d]);
            }
        };
        int *qu = queue[w];
        int cnt = 0;
        for (int base = n0; base < n1; base += 32) {
            const int n = base + lane;
            int j = n < n1 ? ls[n] : i;
            bool hit = false;
            if (n < n1 && ((FULL ? j == i : j <= i) || j < 0 || j >= N)) {
                atomicOr(a.status, (unsigned)ST_LIST_OVERFLOW);
                j = i;
            }
            if (j != i) {
                const float4 o = opos[j];
                float dx = oi.x - o.x, dy = oi.y - o.y, dz = oi.z - o.z;
                dx = fmaf(-L[0], rintf(dx * I[0]), dx);
                dy = fmaf(-L[1], rintf(dy * I[1]), dy);
                dz = fmaf(-L[2], rintf(dz * I[2]), dz);
                hit = fmaf(dx, dx, fmaf(dy, dy, dz * dz)) < lim2;
            }
            const unsigned m = __ballot_sync(0xffffffffu, hit);
            if (hit) qu[cnt + __popc(m & ((1u << lane) - 1u))] = j;
            cnt += __popc(m);
            __syncwarp();
            if (cnt >= 32) {
                pair(qu[lane]);
                cnt -= 32;
                const int rest = lane < cnt ? qu[32 + lane] : 0;
                __syncwarp();
                qu[lane] = rest;
                __syncwarp();
            }
        }
        if (lane < cnt) pair(qu[lane]);
        __syncwarp();
        // the warp's four sums by a reduce-scatter (six additions instead of twenty): lanes
        // 0, 8, 16, 24 end up with f0, f1, f2 and el
        npair = __reduce_add_sync(0xffffffffu, npair);
        const bool up = lane & 16, odd = lane & 8;
        double v0 = up ? f2 : f0, v1 = up ? el : f1;
        v0 += __shfl_xor_sync(0xffffffffu, up ? f0 : f2, 16);
        v1 += __shfl_xor_sync(0xffffffffu, up ? f1 : el, 16);
        double v = (odd ? v1 : v0) + __shfl_xor_sync(0xffffffffu, odd ? v0 : v1, 8);
        for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((lane & 7) == 0) {
            if (lane == 24) e = (v * (4.0 * C.epslj) - npair * C.e_cut) * (FULL ? 0.5 : 1.0);
            else if (FULL) plane[4 * i + (lane >> 3)] = 24.0 * C.epslj * v;
            else atomicAdd(plane + 4 * i + (lane >> 3), 24.0 * C.epslj * v);
        }
    }
    if (lane == 24) red[w] = e;
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(&a.energy[J.slot], (red[0] + red[1]) + (red[2] + red[3]));
}

// ---- k_intra64: intramolecular terms (forces.cpp:65-138, :141-177, :519-554) ----------
// Four threads a molecule, as what bounds it is the length of the chains of FP64 library
// functions: the three same-molecule Ewald pairs (erfc - 1) a thread each, the quartic
// Morse bonds and the HOH angle the fourth (one thread for all of it took 30 us whatever
// the batch). Per molecule 18 doubles, site forces (M, H1, H2) and atom forces (O, H1,
// H2), for k_combine64; the energy with the Ewald self term into the job's slot.

__global__ void __launch_bounds__(128) k_intra64(EvalArgs a) {
    const Job J = a.jobs[blockIdx.y];
    const SysDev &S = a.sys[J.sys];
    const int N = S.n_mols;
    if ((int)(blockIdx.x * blockDim.x) >= 4 * N) return;
    const int t = blockIdx.x * blockDim.x + threadIdx.x, k = t & 3, m = min(t >> 2, N - 1);
    const bool act = (t >> 2) < N;
    __shared__ double red[4];
    const double *q = a.pos + J.pos_off + 9 * m;
    double *o = a.intra64 + 18 * ((size_t)J.site_off / 3 + m);
    const Consts &C = a.c;
    double e = 0.0, f[3] = {0.0, 0.0, 0.0};  // k < 3: the pair's force on its first site
    if (k < 3) {
        const int i = k == 2 ? 1 : 0, j = k == 0 ? 1 : 2;
        const double g = C.gamma_vs;
        double r[3];
        for (int d = 0; d < 3; ++d) {
            const double si = i ? q[3 * i + d] : g * q[d] + 0.5 * (1.0 - g) * (q[3 + d] + q[6 + d]);
            r[d] = si - q[3 * j + d];
        }
        min_image3(r, S);
        const double *chg = a.charge + S.chg_off + 3 * m;
        const double qq = chg[i] * chg[j], r2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
        if (r2 < S.rc_sq) {
            const double rl = sqrt(r2), inv = 1.0 / rl, kap = S.kappa;
            e = qq * inv * (erfc(kap * rl) - 1.0);
            const double ff = (e + qq * S.ewald_pref * exp(-(kap * kap) * r2)) * inv * inv;
            for (int d = 0; d < 3; ++d) f[d] = ff * r[d];
        }
    } else {
        double fa[9];
        for (int d = 0; d < 9; ++d) fa[d] = 0.0;
        // quartic Morse bonds (forces.cpp:65-93, :519-551)
        double r[2][3], l[2];
        for (int b = 0; b < 2; ++b) {
            for (int d = 0; d < 3; ++d) r[b][d] = q[d] - q[3 + 3 * b + d];
            min_image3(r[b], S);
            l[b] = sqrt(r[b][0] * r[b][0] + r[b][1] * r[b][1] + r[b][2] * r[b][2]);
            const double x = l[b] - C.roheq, x2 = x * x, x3 = x2 * x, x4 = x2 * x2;
            e += C.Dr * (C.ar2 * x2 - C.ar3 * x3 + C.ar4fac * x4);
            const double gg = (2.0 * C.ar2 * x - 3.0 * C.ar3 * x2 + 4.0 * C.ar4fac * x3) * C.Dr / l[b];
            for (int d = 0; d < 3; ++d) {
                fa[d] -= gg * r[b][d];
                fa[3 + 3 * b + d] += gg * r[b][d];
            }
        }
        // harmonic HOH angle (forces.cpp:96-138)
        const double dot = r[0][0] * r[1][0] + r[0][1] * r[1][1] + r[0][2] * r[1][2];
        const double ia = 1.0 / l[0], ib = 1.0 / l[1], iab = ia * ib, c = dot * iab;
        const double dacos = 1.0 / sqrt(1.0 - c * c), ca = dot * ia * ia * iab, cb = dot * ib * ib * iab;
        const double dth = acos(c) - C.theta_eq;
        e += 0.5 * C.ktheta * dth * dth;
        const double gp = C.ktheta * dth * dacos;
        for (int d = 0; d < 3; ++d) {
            fa[d] += gp * (iab * (r[0][d] + r[1][d]) - ca * r[0][d] - cb * r[1][d]);
            fa[3 + d] -= gp * (iab * r[1][d] - ca * r[0][d]);
            fa[6 + d] -= gp * (iab * r[0][d] - cb * r[1][d]);
        }
        if (act)
            for (int d = 0; d < 9; ++d) o[9 + d] = fa[d];
        if (m == 0 && !a.sr_only) e -= S.self_energy;
    }
    // site k takes its two pairs' forces: M +(0) +(1), H1 -(0) +(2), H2 -(1) -(2)
    for (int d = 0; d < 3; ++d) {
        const int base = threadIdx.x & 28;
        const double p = __shfl_sync(0xffffffffu, f[d], base + (k == 2 ? 1 : 0));
        const double s = __shfl_sync(0xffffffffu, f[d], base + (k == 0 ? 1 : 2));
        if (act && k < 3) o[3 * k + d] = (k == 0 ? p : -p) + (k == 2 ? -s : s);
    }
    const double te = block_sum(act ? e : 0.0, red);
    if (threadIdx.x == 0) atomicAdd(&a.energy[J.slot], te);
}

// ---- k_combine64 ------------------------------------------------------------------------
// Three threads a molecule (one a dimension): the k-force planes in order, k_real64's
// two-limb sums, the intramolecular and Lennard-Jones forces, and the M-site chain rule
// (forces.cpp:613-619).
__global__ void __launch_bounds__(96) k_combine64(EvalArgs a) {
    const Job J = a.jobs[blockIdx.y];
    const SysDev &S = a.sys[J.sys];
    const int t = blockIdx.x * 96 + threadIdx.x, m = t / 3, d = t - 3 * m;
    if (m >= S.n_mols) return;
    double fs[3] = {0.0, 0.0, 0.0};
    if (!a.sr_only) {
        const size_t at = 3 * ((size_t)J.site_off + 3 * m) + d;
        for (int p = 0; p < a.n_kc; ++p)
            for (int s = 0; s < 3; ++s) fs[s] += a.part[3 * (size_t)p * a.total_sites + at + 3 * s];
        // units of 2^-56 q_top^2 kappa^2
        const double unit = S.q_top * S.kappa * (S.q_top * S.kappa);
        for (int s = 0; s < 3; ++s) {
            const long long *rf = a.rfix + 2 * (at + 3 * s);
            fs[s] += unit * fma((double)rf[0], 5.960464477539063e-08, (double)rf[1] * 1.3877787807814457e-17);
        }
    }
    const size_t mol = (size_t)J.site_off / 3 + m;
    const double *in = a.intra64 + 18 * mol + d;
    for (int s = 0; s < 3; ++s) fs[s] += in[3 * s];
    const double g = a.c.gamma_vs, h = 0.5 * (1.0 - g);
    double *f = a.out + J.out_off + 9 * m + d;
    f[0] = (in[9] + g * fs[0]) + a.lj64[4 * mol + d];
    f[3] = in[12] + fs[1] + h * fs[0];
    f[6] = in[15] + fs[2] + h * fs[0];
}

}  // namespace

void launch_intra64(const EvalArgs &a, cudaStream_t s) {
    k_intra64<<<dim3((a.max_mols + 31) / 32, a.n_jobs), 128, 0, s>>>(a);
}
void launch_combine64(const EvalArgs &a, cudaStream_t s) {
    k_combine64<<<dim3((a.max_mols + 31) / 32, a.n_jobs), 96, 0, s>>>(a);
}

void launch_lj64_prep(const EvalArgs &a, cudaStream_t s) {
    k_lj64_prep<<<dim3((a.max_mols + 127) / 128, a.n_jobs), 128, 0, s>>>(a);
}

void launch_lj64(const EvalArgs &a, cudaStream_t s) {
    const dim3 g((a.max_mols + 3) / 4, a.n_jobs);
    if (a.lj_full) k_lj64<1><<<g, 128, 0, s>>>(a);
    else k_lj64<0><<<g, 128, 0, s>>>(a);
}

}  // namespace qtg
