// FP32 pairs and triples: a number held as the unevaluated sum of two floats (~47 bits) or three
// (~60 bits). On GB300 an FP64 operation costs 64 FP32 ones, so values that need more than
// FP32 (energies of clashes, sums that cancel) are formed in pairs, and in triples where FP64's
// 53 bits have to be met: products keep their rounding error by fma, sums by two-sum. The
// intrinsics keep the compiler from contracting the pieces.
#pragma once

#include <cuda_runtime.h>

namespace pxd {

struct F2 {
    float h, l;
};
struct F3 {
    float h, l, m;
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

// x^2 + y^2 + z^2 of normalised pairs (the squares of the low parts are left out)
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

// a + b exactly
__device__ __forceinline__ F2 two_sum(float a, float b) {
    const float s = __fadd_rn(a, b);
    const float c = __fsub_rn(s, a);
    return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, c)), __fsub_rn(b, c))};
}

// l += v, what rounds off added to m
__device__ __forceinline__ void low_acc(float& l, float& m, float v) {
    const F2 t = two_sum(l, v);
    l = t.h;
    m = __fadd_rn(m, t.l);
}

// x^2 + y^2 + z^2 to ~2^-60 of itself
__device__ __forceinline__ F3 triple_norm2(F3 x, F3 y, F3 z) {
    const float sx = __fmul_rn(x.h, x.h), sy = __fmul_rn(y.h, y.h), sz = __fmul_rn(z.h, z.h);
    const float x2 = __fadd_rn(x.h, x.h), y2 = __fadd_rn(y.h, y.h), z2 = __fadd_rn(z.h, z.h);
    const float cx = __fmul_rn(x2, x.l), cy = __fmul_rn(y2, y.l), cz = __fmul_rn(z2, z.l);
    const F2 a = two_sum(sx, sy), b = two_sum(a.h, sz);
    float m = __fmaf_rn(x2, x.m, __fmaf_rn(y2, y.m, __fmul_rn(z2, z.m)));
    m = __fmaf_rn(x.l, x.l, __fmaf_rn(y.l, y.l, __fmaf_rn(z.l, z.l, m)));
    m = __fadd_rn(m, __fadd_rn(__fmaf_rn(x2, x.l, -cx), __fadd_rn(__fmaf_rn(y2, y.l, -cy), __fmaf_rn(z2, z.l, -cz))));
    float l = a.l;
    low_acc(l, m, b.l);
    low_acc(l, m, __fmaf_rn(x.h, x.h, -sx));
    low_acc(l, m, __fmaf_rn(y.h, y.h, -sy));
    low_acc(l, m, __fmaf_rn(z.h, z.h, -sz));
    low_acc(l, m, cx);
    low_acc(l, m, cy);
    low_acc(l, m, cz);
    const float s = __fadd_rn(b.h, l);
    return {s, __fsub_rn(l, __fsub_rn(s, b.h)), m};
}

// 1/r (triple) and 1/r^2 (pair) of r2 = r^2 (finite, away from 0): the FP32 rsqrt with one Newton
// step, so that what is left of 1 - r2 y^2 is below 2^-23 and its sum rounds below 2^-70, and
// the third-order correction
__device__ __forceinline__ void triple_rsqrt(F3 r2, F3& rinv, F2& rinv2) {
    const float y0 = rsqrtf(r2.h);
    const float t = __fmul_rn(r2.h, y0);
    const float y = __fmaf_rn(__fmul_rn(0.5f, y0), __fmaf_rn(-t, y0, __fmaf_rn(__fmaf_rn(r2.h, y0, -t), -y0, 1.f)), y0);
    const float ih = __fmul_rn(y, y);
    const float il = __fmaf_rn(y, y, -ih);
    // h + e = 1 - r2 y^2
    const float q = __fmul_rn(r2.h, il), p = __fmul_rn(r2.l, ih);
    float h = __fmaf_rn(-r2.h, ih, 1.f), e = 0.f;
    low_acc(h, e, -q);
    low_acc(h, e, -p);
    e = __fsub_rn(e, __fadd_rn(__fmaf_rn(r2.h, il, -q), __fmaf_rn(r2.l, ih, -p)));
    e = __fmaf_rn(-r2.m, ih, __fmaf_rn(-r2.l, il, e));
    // 1/r = y (1 + h / 2 + e / 2 + 3 h^2 / 8)
    const float g = __fmul_rn(0.5f, h);
    const float l = __fmul_rn(y, g);
    rinv = {y, l, __fmaf_rn(y, __fmaf_rn(__fmul_rn(1.5f, g), g, __fmul_rn(0.5f, e)), __fmaf_rn(y, g, -l))};
    rinv2 = {ih, __fmaf_rn(ih, __fmaf_rn(h, h, h), il)};
}

// a += q r; returns q r as a pair
__device__ __forceinline__ F2 triple_acc(F3& a, F2 q, F3 r) {
    const float p = __fmul_rn(q.h, r.h), s = __fmul_rn(q.h, r.l), t = __fmul_rn(q.l, r.h);
    const float e = __fmaf_rn(q.h, r.h, -p);
    float m = __fmaf_rn(q.h, r.m, __fmul_rn(q.l, r.l));
    m = __fadd_rn(m, __fadd_rn(__fmaf_rn(q.h, r.l, -s), __fmaf_rn(q.l, r.h, -t)));
    const F2 k = two_sum(a.h, p);
    a.h = k.h;
    a.m = __fadd_rn(a.m, m);
    low_acc(a.l, a.m, k.l);
    low_acc(a.l, a.m, e);
    low_acc(a.l, a.m, s);
    low_acc(a.l, a.m, t);
    return {p, __fadd_rn(e, __fadd_rn(s, t))};
}

}  // namespace pxd
