// 62-bit fixed-point products from 32 x 32 -> 64-bit integer multiply-adds.
#pragma once

namespace qtg {

typedef long long i64;

__device__ __forceinline__ i64 madw(int a, int b, i64 c) { return (i64)a * b + c; }
// v in limbs: h 2^31 + l, 0 <= l < 2^31; |v| < 2^62
struct Limbs {
    int h, l;
};
__device__ __forceinline__ Limbs split62(i64 v) { return Limbs{(int)(v >> 31), (int)v & 0x7fffffff}; }
// x y 2^-62 to within a unit: the product of the low limbs (a quarter unit in the mean) is
// left out and the floor takes half a unit, which the added constant makes up
__device__ __forceinline__ i64 mul62(const Limbs &x, const Limbs &y) {
    return (i64)x.h * y.h + (madw(x.h, y.l, madw(x.l, y.h, 0x60000000ll)) >> 31);
}
// the same with the low limbs' product, for a factor that many pairs share
__device__ __forceinline__ i64 mul62x(const Limbs &x, const Limbs &y) {
    return (i64)x.h * y.h + (madw(x.h, y.l, madw(x.l, y.h, ((i64)x.l * y.l >> 31) + 0x40000000ll)) >> 31);
}
__device__ __forceinline__ i64 sqr62(const Limbs &x) { return (i64)x.h * x.h + (madw(x.h, x.l, 0x30000000ll) >> 30); }

}  // namespace qtg
