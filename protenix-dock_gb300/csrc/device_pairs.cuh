// FP32 pairs: a number held as the unevaluated sum hi + lo of two floats, ~47 bits. On GB300
// an FP64 operation costs 64 FP32 ones, so values that need more than FP32 (energies of
// clashes, sums that cancel) are formed in pairs: products keep their rounding error by
// fma, sums by two-sum. The intrinsics keep the compiler from contracting the pieces.
#pragma once

#include <cuda_runtime.h>

namespace pxd {

struct F2 {
    float h, l;
};

// hi + lo += v + e, the rounding of hi + v kept (two-sum)
__device__ __forceinline__ void pair_acc(float& hi, float& lo, float v, float e) {
    const float s = __fadd_rn(hi, v);
    const float b = __fsub_rn(s, hi);
    const float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, b)), __fsub_rn(v, b));
    hi = s;
    lo = __fadd_rn(lo, __fadd_rn(err, e));
}
__device__ __forceinline__ void pair_acc(F2& a, F2 b) { pair_acc(a.h, a.l, b.h, b.l); }

// a - b exactly
__device__ __forceinline__ F2 two_diff(float a, float b) {
    const float d = __fsub_rn(a, b);
    const float c = __fsub_rn(d, a);
    return {d, __fsub_rn(__fsub_rn(a, __fsub_rn(d, c)), __fadd_rn(b, c))};
}
__device__ __forceinline__ F2 pair_sub(F2 a, F2 b) {
    const F2 d = two_diff(a.h, b.h);
    return {d.h, __fadd_rn(d.l, __fsub_rn(a.l, b.l))};
}
// a hi part that carries the leading bits again (|h| >= |l| on entry)
__device__ __forceinline__ F2 pair_norm(F2 a) {
    const float s = __fadd_rn(a.h, a.l);
    return {s, __fadd_rn(a.l, __fsub_rn(a.h, s))};
}
__device__ __forceinline__ F2 pair_mul(F2 a, F2 b) {
    const float p = __fmul_rn(a.h, b.h);
    return {p, __fmaf_rn(a.l, b.h, __fmaf_rn(a.h, b.l, __fmaf_rn(a.h, b.h, -p)))};
}
__device__ __forceinline__ F2 pair_mul(F2 a, float b) {
    const float p = __fmul_rn(a.h, b);
    return {p, __fmaf_rn(a.l, b, __fmaf_rn(a.h, b, -p))};
}
__device__ __forceinline__ F2 pair_square(F2 a) {
    const float p = __fmul_rn(a.h, a.h);
    return {p, __fmaf_rn(__fadd_rn(a.h, a.h), a.l, __fmaf_rn(a.h, a.h, -p))};
}

// x^2 + y^2 + z^2
__device__ __forceinline__ F2 pair_norm2(F2 x, F2 y, F2 z) {
    const float sx = __fmul_rn(x.h, x.h), sy = __fmul_rn(y.h, y.h), sz = __fmul_rn(z.h, z.h);
    F2 r{sx, __fadd_rn(__fmaf_rn(x.h, x.h, -sx), __fadd_rn(__fmaf_rn(y.h, y.h, -sy), __fmaf_rn(z.h, z.h, -sz)))};
    r.l = __fmaf_rn(2.f, __fmaf_rn(x.h, x.l, __fmaf_rn(y.h, y.l, __fmul_rn(z.h, z.l))), r.l);
    pair_acc(r.h, r.l, sy, 0.f);
    pair_acc(r.h, r.l, sz, 0.f);
    return r;
}

// 1/r and 1/r^2 of r2 = r^2 (finite, away from 0): the FP32 rsqrt y and the third-order
// correction from h = 1 - r2 y^2
__device__ __forceinline__ void pair_rsqrt(F2 r2, F2& rinv, F2& rinv2) {
    const float y = rsqrtf(r2.h);
    const float ih = __fmul_rn(y, y);
    const float yl = __fmaf_rn(y, y, -ih);
    float h = __fmaf_rn(-r2.h, ih, 1.f);
    h = __fmaf_rn(-r2.h, yl, h);
    h = __fmaf_rn(-r2.l, ih, h);
    rinv = {y, __fmul_rn(y, __fmul_rn(h, __fmaf_rn(h, 0.375f, 0.5f)))};
    rinv2 = {ih, __fmaf_rn(ih, __fmaf_rn(h, h, h), yl)};
}

}  // namespace pxd
