// Structure factors of the mixed form for batches that fill the GPU (forces.cpp:180-448),
// as a register-tiled product. Small batches take k_ksk (see ksk2_ok in forces.cu).
#include <math.h>

#include <algorithm>

#include "packed.h"
#include "qtg_internal.h"

namespace qtg {

namespace {

// ---- k_ksk2: structure factors --------------------------------------------------------
// S(k) = sum_i q_i X_i(kx) Y_i(ky) Z_i(kz) is a product of column factors A = X Y with the
// Z rows, and what bounds it is how often shared memory is read for its multiply-adds:
// k_ksk reads five 8-byte entries a site for the twelve of a column's three |kz| (its
// shared-memory pipe runs at 80 %, the FMA pipe at 41 %). Here a thread holds a pair of
// columns (kx, +-ky), whose factors come from one X and one Y entry, and four |kz|, whose
// Z come in two 16-byte loads (real parts, imaginary parts): four loads for 38
// multiply-adds, of which the 32 products run packed, two |kz| an instruction. The sums
// are T1 = Ar Zr, T2 = Ai Zi, T3 = Ar Zi, T4 = Ai Zr per column and |kz|: S(+kz) = T1 - T2
// + i (T3 + T4), S(-kz) = T1 + T2 + i (T4 - T3). Sites lie in shared memory a record each
// (X, Y, Zr, Zi), so that the lanes of a warp, on neighbouring (kx, ky) and mostly one
// group of |kz|, read one or two 128-byte lines an access; CH2 sites at a time, double-
// buffered by cp.async. Sums: 16 sites in FP32, six of these HELD chunks, the two halves of a
// block (at most 192 sites, see set_ksk2_chunks in forces.cu; the first half's sums wait in
// shared memory), the blocks with compensation (k_sk_reduce). Errors against FP64 sums of the
// same factors, 1536 sites: random phases 1.05e-7 of S (k_ksk's 32 sites and compensation from
// there on 1.60e-7), sites in phase as in a crystal 3.34e-8 (k_ksk 3.6e-8 in four blocks, 3.3e-8
// in sixteen); with 192 sites in a plain sum 3.5e-8. Kahan's compensation after each chunk (3.2e-8)
// takes as much shared memory again: 512 waters, 32 beads 34.9 -> 38.3 us, 1000 waters, 16 beads 5 %
// of a step.
constexpr int CH2 = 48, SUB2 = 16, HELD = 2;

__host__ __device__ constexpr int ksk2_km4(int km1) { return (km1 + 3) & ~3; }
// floats a site record takes: an odd number of 16-byte units, so that the 16-byte
// accesses of eight neighbouring sites' copies fall into different banks
__host__ __device__ constexpr int ksk2_record(int km1) {
    const int n = 4 * km1 + 2 * ksk2_km4(km1);
    return (n / 4) % 2 ? n : n + 4;
}

__global__ void __launch_bounds__(256) k_ksk2(EvalArgs a) {
    const int sc = blockIdx.y;
    const Job J = a.jobs[blockIdx.z];
    const SysDev &S = a.sys[J.sys];
    const int np = S.n_pair, ns = S.n_sites, km1 = S.k_max + 1, km4 = ksk2_km4(km1), R = ksk2_record(km1);
    const int s0 = sc * a.sk_sites, s1 = min(ns, s0 + a.sk_sites);  // this block's sites
    if ((int)(blockIdx.x * blockDim.x) >= np || s0 >= ns) return;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const KGroup G = a.kpair[S.pair_off + min(t, np - 1)];
    const KCol C = a.kcol[S.col_off + G.col];
    extern __shared__ __align__(16) float rec[];  // [2][CH2][R]
    const int xat = 2 * C.kx, yat = 2 * (km1 + C.ky), zat = 4 * km1 + G.kz0;
    const float2 *ph = reinterpret_cast<const float2 *>(a.phase) + J.phase_off;
    const int nchunk = (s1 - s0 + CH2 - 1) / CH2;
    // a warp copies eight sites of four rows at a time
    auto stage = [&](int ci) {
        const int c0 = s0 + ci * CH2;
        float *buf = rec + (ci & 1) * CH2 * R;
        for (int idx = threadIdx.x; idx < 2 * km1 * CH2; idx += blockDim.x) {
            const int c = (idx & 7) | ((idx >> 3) / (2 * km1)) << 3, row = (idx >> 3) % (2 * km1), s = c0 + c;
            cp_async<8>(buf + c * R + 2 * row, ph + (size_t)row * ns + min(s, s1 - 1), s < s1);
        }
        const float *z = reinterpret_cast<const float *>(ph + (size_t)2 * km1 * ns);
        for (int idx = threadIdx.x; idx < km1 * CH2; idx += blockDim.x) {
            const int c = (idx & 7) | ((idx >> 3) / km1) << 3, row = (idx >> 3) % km1, s = c0 + c;
            const float *src = z + 2 * ((size_t)row * ns + min(s, s1 - 1));
            float *dst = buf + c * R + 4 * km1 + row;
            cp_async<4>(dst, src, s < s1);
            cp_async<4>(dst + km4, src + 1, s < s1);
        }
        cp_async_commit();
    };
    // the pad of the Z rows is multiplied but not stored: it has to be finite
    for (int idx = threadIdx.x; idx < 2 * CH2 * 2 * (km4 - km1); idx += blockDim.x) {
        const int c = idx / (2 * (km4 - km1)), k = idx - c * 2 * (km4 - km1), im = k / (km4 - km1);
        rec[c * R + 4 * km1 + im * km4 + km1 + k - im * (km4 - km1)] = 0.f;
    }
    const F2 zero = pk(0.f, 0.f);
    F2 T[2][4][2];  // [column][T1..T4][|kz| pair]
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int k = 0; k < 4; ++k) T[h][k][0] = T[h][k][1] = zero;
    stage(0);
    ulonglong2 *held = reinterpret_cast<ulonglong2 *>(rec + 2 * CH2 * R) + threadIdx.x;  // the first half's sums
    for (int ci = 0; ci < nchunk; ++ci) {
        if (ci == HELD) {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                F2 *c = T[k >> 2][k & 3];
                held[k * blockDim.x] = make_ulonglong2(c[0].v, c[1].v);
                c[0] = c[1] = zero;
            }
        }
        __syncthreads();  // every thread is done with buffer (ci + 1) & 1
        if (ci + 1 < nchunk) stage(ci + 1);
        else cp_async_commit();
        cp_async_wait<1>();  // this thread's copies of chunk ci have landed
        __syncthreads();     // and every other thread's
        const float *buf = rec + (ci & 1) * CH2 * R;
        const int nc = min(CH2, s1 - s0 - ci * CH2);
        for (int c0 = 0; c0 < nc; c0 += SUB2) {
            F2 v[2][4][2];
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int k = 0; k < 4; ++k) v[h][k][0] = v[h][k][1] = zero;
            auto site = [&](int c) {
                const float *r = buf + c * R;
                const float2 x = *reinterpret_cast<const float2 *>(r + xat), y = *reinterpret_cast<const float2 *>(r + yat);
                const float4 zr = *reinterpret_cast<const float4 *>(r + zat), zi = *reinterpret_cast<const float4 *>(r + zat + km4);
                const F2 zr0 = pk(zr.x, zr.y), zr1 = pk(zr.z, zr.w), zi0 = pk(zi.x, zi.y), zi1 = pk(zi.z, zi.w);
                const float p = x.x * y.x, q = x.y * y.x;
                const float re[2] = {fmaf(-x.y, y.y, p), fmaf(x.y, y.y, p)}, im[2] = {fmaf(x.x, y.y, q), fmaf(-x.x, y.y, q)};
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const F2 ar = pk(re[h], re[h]), ai = pk(im[h], im[h]);
                    v[h][0][0] = fma2(ar, zr0, v[h][0][0]);
                    v[h][0][1] = fma2(ar, zr1, v[h][0][1]);
                    v[h][1][0] = fma2(ai, zi0, v[h][1][0]);
                    v[h][1][1] = fma2(ai, zi1, v[h][1][1]);
                    v[h][2][0] = fma2(ar, zi0, v[h][2][0]);
                    v[h][2][1] = fma2(ar, zi1, v[h][2][1]);
                    v[h][3][0] = fma2(ai, zr0, v[h][3][0]);
                    v[h][3][1] = fma2(ai, zr1, v[h][3][1]);
                }
            };
            if (c0 + SUB2 <= nc) {
#pragma unroll 8
                for (int c = 0; c < SUB2; ++c) site(c0 + c);
            } else {
                for (int c = c0; c < nc; ++c) site(c);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    T[h][k][0] = add2(T[h][k][0], v[h][k][0]);
                    T[h][k][1] = add2(T[h][k][1], v[h][k][1]);
                }
        }
    }
    if (t >= np) return;
    if (nchunk > HELD) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const ulonglong2 o = held[k * blockDim.x];
            F2 *c = T[k >> 2][k & 3];
            c[0] = add2(c[0], F2{o.x});
            c[1] = add2(c[1], F2{o.y});
        }
    }
    float2 *skp = reinterpret_cast<float2 *>(a.skp) + (size_t)sc * a.total_k + J.sk_off;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int col = h ? G.col2 : G.col;
        if (col < 0) continue;
        const KCol D = a.kcol[S.col_off + col];
        float2 *o = skp + D.k_begin + D.m;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            float ts[4][2];
#pragma unroll
            for (int k = 0; k < 4; ++k) unpk(T[h][k][u], ts[k][0], ts[k][1]);
#pragma unroll
            for (int w = 0; w < 2; ++w) {
                const int az = G.kz0 + 2 * u + w;
                if (2 * u + w >= G.n) continue;
                o[az] = make_float2(ts[0][w] - ts[1][w], ts[2][w] + ts[3][w]);
                if (az) o[-az] = make_float2(ts[0][w] + ts[1][w], ts[3][w] - ts[2][w]);
            }
        }
    }
}

size_t ksk2_smem(int kmax, int threads) {
    return (size_t)2 * CH2 * ksk2_record(kmax + 1) * sizeof(float) + (size_t)threads * 8 * sizeof(ulonglong2);
}

}  // namespace

void init_recip32_attributes() {
    cudaFuncSetAttribute(k_ksk2, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
}

int ksk2_blocks(const EvalArgs &a) { return (a.max_pair + a.pair_threads - 1) / a.pair_threads; }

void launch_ksk2(const EvalArgs &a, cudaStream_t s) {
    k_ksk2<<<dim3(ksk2_blocks(a), a.n_sc, a.n_jobs), a.pair_threads, ksk2_smem(a.max_kmax, a.pair_threads), s>>>(a);
}
}  // namespace qtg
