// Real-space Ewald of the FP64 form (energies and forces; replaces the pair loop
// of forces.cpp:589-608 with its rwald, forces.cpp:141-177).
//
// What bounds it: FP64 issue. This GPU runs two FP64 lanes a cycle an SM (a warp's
// FP64 instruction takes sixteen cycles of the SM, an FP32 one a quarter), so the time
// is the number of FP64 instructions and everything else is nearly free. Hence
//   * every site pair once (a warp holds 16 sites and visits the tiles of 32 sites at
//     ring distances 0 .. T/2, as k_real_half does);
//   * the cutoff test first in FP32, on the wrapped coordinates with a margin above
//     their rounding, and only the pairs that pass (31-52 % of them), packed into full
//     warps, evaluated in FP64, where r^2 < r_c^2 is decided;
//   * erfc(x)/x and the force factor from degree-7 polynomials in u = (kappa r)^2
//     (14 multiply-adds a pair for both) instead of erfc, exp, sqrt and a division
//     (some 150 instructions);
//   * both sides' forces summed from the packed pairs' shared-memory copies in a fixed
//     order, a lane a site, and added to the configuration's sums as two-limb fixed
//     point by integer atomics, so the totals do not depend on the order the warps run.
// 216 waters, 32 beads: 3283 us for k_real<double> (all pairs from both sides, library
// functions), 337 us here.
#include <math.h>
#include <string.h>

#include <algorithm>

#include "qtg_internal.h"

namespace qtg {

// ---- the pair-function table ------------------------------------------------------
// With u = (kappa r)^2, G(u) = erfc(sqrt u) / sqrt u and W(u) = (G(u) + a exp(-u)) / u
// (a = 2 / sqrt(pi) with the reference's pi), a pair's energy is q_i q_j kappa G and its
// force q_i q_j kappa^3 W d. The table splits each octave of u in [2^R64_LO, 2^R64_HI)
// into 64 intervals, found from the top bits of u, and holds the Taylor coefficients of
// G and W about an interval's middle, degree 7 each (16 doubles, one 128-byte line). In
// an interval |t| <= u/128, so the truncated terms are below 3e-17 of the value for
// u < 8 and below 6e-15 for u < 16 (where the value itself is below 1e-4 of a near
// pair's). The coefficients follow from the two functions' differential equations,
//   2 u G' + G + (2/sqrt(pi)) e^-u = 0  and  u W = G + a e^-u,
// whose recurrences add terms of one sign only (no cancellation); G at the middle is
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

namespace {

constexpr int RW = 2;              // warps per block: the two halves of a tile of 32 sites
constexpr int RROWS = 16;          // sites a warp holds
constexpr int RCAP = RROWS * 32;   // pairs of one visit

struct RWarp {
    double4 sj[32], si[RROWS];
    double f[3][RCAP];             // the packed pairs' forces on the held site
    float4 sif[RROWS];             // FP32 coordinates and the site's molecule
    unsigned mask[RROWS];          // row r's visited sites that passed
    int off[RROWS + 1];            // where row r's packed pairs start
    unsigned short code[RCAP];     // row, visited site and image of every packed pair
};

// u outside the table (below 2^R64_LO; above 2^R64_HI only with an Ewald tolerance below 1e-13)
__device__ __noinline__ void pair_far(double u, double *g, double *w) {
    const double x = sqrt(u);
    *g = erfc(x) / x;
    *w = (*g + 2.0 / sqrt(PI_REF) * exp(-u)) / u;
}

// Adds v to a two-limb fixed-point sum: hi in units of 2^-8, lo in units of 2^-60, each
// rounded by adding a power of two whose last place is the unit (exact for |v| < 2^42).
__device__ __forceinline__ void limb_add(long long *p, double v) {
    const double C1 = 26388279066624.0, C2 = 0.005859375;  // 1.5 2^44, 1.5 2^-8
    const double h = __dadd_rn(v, C1), l = __dadd_rn(__dsub_rn(v, __dsub_rn(h, C1)), C2);
    atomicAdd(reinterpret_cast<unsigned long long *>(p),
              (unsigned long long)(__double_as_longlong(h) - __double_as_longlong(C1)));
    atomicAdd(reinterpret_cast<unsigned long long *>(p + 1),
              (unsigned long long)(__double_as_longlong(l) - __double_as_longlong(C2)));
}

__global__ void __launch_bounds__(32 * RW) k_real64(EvalArgs a, int n_ch) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    RWarp &W = reinterpret_cast<RWarp *>(smem_raw)[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const Job J = a.jobs[blockIdx.z];
    const SysDev &S = a.sys[J.sys];
    const int ns = S.n_sites, T = (ns + 31) / 32, tI = blockIdx.x;
    const int i0 = tI * 32 + (threadIdx.x >> 5) * RROWS;
    if (i0 >= ns) return;  // (warps of a block are independent)
    const int maxd = T / 2;
    const int d0 = (int)(((long long)(maxd + 1) * blockIdx.y) / n_ch);
    const int d1 = (int)(((long long)(maxd + 1) * (blockIdx.y + 1)) / n_ch);
    if (d0 >= d1) return;
    const double4 *sites = reinterpret_cast<const double4 *>(a.sites) + J.site_off;
    const int nrow = min(RROWS, ns - i0);
    const float L0 = S.boxf[0], L1 = S.boxf[1], L2 = S.boxf[2];
    const float I0 = S.inv_boxf[0], I1 = S.inv_boxf[1], I2 = S.inv_boxf[2];
    const double B0 = S.box[0], B1 = S.box[1], B2 = S.box[2];
    const double rc2 = S.rc_sq, kap2 = S.kappa * S.kappa, k3 = kap2 * S.kappa;
    // FP32 rounding of two wrapped coordinates, their difference and its image is below
    // 2^-22 of the box in each dimension: r is below r_c plus that where r^2 < r_c^2
    const float lim = sqrtf(S.rc_sqf) * (1.0f + 1e-6f) + 5e-7f * (L0 + L1 + L2), lim2 = lim * lim;
    if (lane < nrow) {
        const double4 s = sites[i0 + lane];
        W.si[lane] = s;
        W.sif[lane] = make_float4((float)s.x, (float)s.y, (float)s.z, __int_as_float((i0 + lane) / 3));
    }
    double sx = 0.0, sy = 0.0, sz = 0.0, e = 0.0;  // of row lane / 2, every other pair
    for (int d = d0; d < d1; ++d) {
        if ((T % 2 == 0) && d == maxd && d > 0 && tI >= maxd) continue;
        const int j = ((tI + d) % T) * 32 + lane, jm = j / 3;
        double4 sj = make_double4(0.0, 0.0, 0.0, 0.0);
        if (j < ns) sj = sites[j];
        __syncwarp();  // the previous visit's copies have been read
        W.sj[lane] = sj;
        const float jx = (float)sj.x, jy = (float)sj.y, jz = (float)sj.z;
        unsigned mine = 0u;  // the rows that my site passed with
        int cnt = 0;
        __syncwarp();
        for (int r = 0; r < RROWS; ++r) {
            bool hit = false;
            int img = 0;
            if (r < nrow) {
                const float4 p = W.sif[r];
                float dx = p.x - jx, dy = p.y - jy, dz = p.z - jz;
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
            const double4 p = W.si[(c >> 5) & 15], s = W.sj[c & 31];
            const int nx = img & 3, ny = (img >> 2) & 3, nz = img >> 4;
            const double dx = (p.x - s.x) - (nx == 1 ? 0.0 : nx == 0 ? -B0 : B0);
            const double dy = (p.y - s.y) - (ny == 1 ? 0.0 : ny == 0 ? -B1 : B1);
            const double dz = (p.z - s.z) - (nz == 1 ? 0.0 : nz == 0 ? -B2 : B2);
            const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
            double w = 0.0;
            if (r2 < rc2) {
                const double u = kap2 * r2;
                const int hi = __double2hiint(u), at = (hi >> 14) - ((1023 + R64_LO) << 6);
                double g;
                if ((unsigned)at < (unsigned)R64_INTERVALS) {
                    const double t = u - __hiloint2double((hi & ~0x3fff) | 0x2000, 0);
                    const double2 *q = reinterpret_cast<const double2 *>(a.real64_tab) + 8 * at;
                    const double2 g3 = __ldg(q + 3), g2 = __ldg(q + 2), g1 = __ldg(q + 1), g0 = __ldg(q);
                    const double2 w3 = __ldg(q + 7), w2 = __ldg(q + 6), w1 = __ldg(q + 5), w0 = __ldg(q + 4);
                    g = fma(g3.y, t, g3.x);
                    w = fma(w3.y, t, w3.x);
                    g = fma(g, t, g2.y);
                    w = fma(w, t, w2.y);
                    g = fma(g, t, g2.x);
                    w = fma(w, t, w2.x);
                    g = fma(g, t, g1.y);
                    w = fma(w, t, w1.y);
                    g = fma(g, t, g1.x);
                    w = fma(w, t, w1.x);
                    g = fma(g, t, g0.y);
                    w = fma(w, t, w0.y);
                    g = fma(g, t, g0.x);
                    w = fma(w, t, w0.x);
                } else {
                    pair_far(u, &g, &w);
                }
                const double qq = p.w * s.w;
                e = fma(qq, g, e);
                w *= qq;
            }
            W.f[0][b] = w * dx;
            W.f[1][b] = w * dy;
            W.f[2][b] = w * dz;
        }
        __syncwarp();
        for (int b = W.off[lane >> 1] + (lane & 1); b < W.off[(lane >> 1) + 1]; b += 2) {
            sx += W.f[0][b];
            sy += W.f[1][b];
            sz += W.f[2][b];
        }
        if (mine) {
            double vx = 0.0, vy = 0.0, vz = 0.0;
            for (unsigned m = mine; m; m &= m - 1) {
                const int r = __ffs(m) - 1, b = W.off[r] + __popc(W.mask[r] & ((1u << lane) - 1u));
                vx -= W.f[0][b];
                vy -= W.f[1][b];
                vz -= W.f[2][b];
            }
            long long *o = a.rfix + 6 * ((size_t)J.site_off + j);
            limb_add(o, k3 * vx);
            limb_add(o + 2, k3 * vy);
            limb_add(o + 4, k3 * vz);
        }
    }
    sx += __shfl_xor_sync(0xffffffffu, sx, 1);
    sy += __shfl_xor_sync(0xffffffffu, sy, 1);
    sz += __shfl_xor_sync(0xffffffffu, sz, 1);
    if (!(lane & 1) && (lane >> 1) < nrow) {
        long long *o = a.rfix + 6 * ((size_t)J.site_off + i0 + (lane >> 1));
        limb_add(o, k3 * sx);
        limb_add(o + 2, k3 * sy);
        limb_add(o + 4, k3 * sz);
    }
    e = warp_sum(e);
    if (lane == 0) atomicAdd(&a.energy[J.slot], S.kappa * e);
}

}  // namespace

void init_real64_attributes() {
    cudaFuncSetAttribute(k_real64, cudaFuncAttributeMaxDynamicSharedMemorySize, RW * (int)sizeof(RWarp));
}

// 216 waters, 32 beads: 3283 us before, 337 us here; 512 waters 1.22 ms.
// Chunks of ring distances: enough blocks for a few waves of the six that fit an SM, so
// that small beads spread over the GPU and the last wave is short.
void launch_real64(const EvalArgs &a, cudaStream_t s) {
    const int T = (3 * a.max_mols + 31) / 32;
    const long long blocks = (long long)T * a.n_jobs, want = 152LL * 24;
    int n_ch = a.tune_rj > 0 ? a.tune_rj : (int)std::min<long long>(MAX_RJ, (want + blocks - 1) / blocks);
    n_ch = std::max(1, std::min(n_ch, T / 2 + 1));
    k_real64<<<dim3(T, n_ch, a.n_jobs), 32 * RW, RW * sizeof(RWarp), s>>>(a, n_ch);
}

}  // namespace qtg
