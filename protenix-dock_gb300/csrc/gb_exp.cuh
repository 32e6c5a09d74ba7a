// The exponential of the GB/SA pair terms.
#pragma once

#include <cmath>

namespace pxd {

// exp(y) by Tang's table-driven method (ACM Trans. Math. Softw. 15, 144, 1989): y = n ln2 / 128 + r,
// exp(y) = 2^(n / 128) (1 + p(r)), |r| <= 0.0028, p to r^5 (the next term is 6e-19). Ten FP64
// operations. table[k] = 2^(k / 128), rounded once: with the last fma, within 1.01 ulp of exp.
// Beyond |y| = 690, and for NaN, the library's exp.
constexpr int kExpTable = 128;

struct GbExpTable {
    double v[kExpTable];
};

inline GbExpTable gb_exp_table() {
    GbExpTable t;
    for (int k = 0; k < kExpTable; ++k) t.v[k] = static_cast<double>(std::exp2(static_cast<long double>(k) / kExpTable));
    return t;
}

__device__ __forceinline__ double gb_exp(double y, const double* table) {
    const int top = __double2hiint(y) & 0x7fffffff;
    if (top > 0x40859000) return exp(y);
    const double round = 6755399441055744.0;  // 1.5 * 2^52: the sum's low bits are the nearest integer
    const double t = fma(y, 184.6649652337873, round);
    const int n = __double2loint(t);
    const double nd = t - round;
    const double r = fma(nd, -1.2655086083325438e-13, fma(nd, -0.005415212347998022, y));
    const double q = fma(r, fma(r, fma(r, 1.0 / 120.0, 1.0 / 24.0), 1.0 / 6.0), 0.5);
    const double p = fma(q, r * r, r);
    const double v = table[n & (kExpTable - 1)];
    const double e = fma(v, p, v);
    return __hiloint2double(__double2hiint(e) + ((n >> 7) << 20), __double2loint(e));
}

}  // namespace pxd
