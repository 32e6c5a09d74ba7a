// gb_exp on the host: its CUDA intrinsics as plain C++. Prints the largest error in ulps against
// the extended-precision exponential over n arguments spread over [-750, 715], dense at the ends
// of its own range and next to 0, then the values of special arguments.
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <limits>

#define __device__
#define __forceinline__ inline
static int64_t bits(double v) {
    int64_t b;
    std::memcpy(&b, &v, 8);
    return b;
}
static int __double2hiint(double v) { return static_cast<int>(bits(v) >> 32); }
static int __double2loint(double v) { return static_cast<int>(bits(v) & 0xffffffff); }
static double __hiloint2double(int hi, int lo) {
    const uint64_t b = (static_cast<uint64_t>(static_cast<uint32_t>(hi)) << 32) | static_cast<uint32_t>(lo);
    double v;
    std::memcpy(&v, &b, 8);
    return v;
}
using std::exp;
using std::fma;
#include "gb_exp.cuh"

int main(int argc, char** argv) {
    const int n = argc > 1 ? std::atoi(argv[1]) : 100000;
    const pxd::GbExpTable t = pxd::gb_exp_table();
    uint64_t s = 88172645463325252ULL;
    auto uniform = [&s] {
        s ^= s << 13;
        s ^= s >> 7;
        s ^= s << 17;
        return static_cast<double>(s >> 11) / 9007199254740992.0;
    };
    double worst = 0.0;
    for (int i = 0; i < n; ++i) {
        const double u = uniform();
        double y = -707.0 + 1414.0 * u;
        if (i % 5 == 1) y = 690.0 + 2.0 * (u - 0.5);
        if (i % 5 == 2) y = -690.0 + 2.0 * (u - 0.5);
        if (i % 5 == 3) y = std::ldexp(u - 0.5, -static_cast<int>(60 * uniform()));
        if (i % 5 == 4) y = -20.0 * u;
        const long double ref = std::exp(static_cast<long double>(y));
        const double r = static_cast<double>(ref), ulp = std::nextafter(std::fabs(r), DBL_MAX) - std::fabs(r);
        const double err = std::fabs(static_cast<double>((static_cast<long double>(pxd::gb_exp(y, t.v)) - ref) / ulp));
        if (!(err <= worst)) worst = err;
    }
    std::printf("%.6f\n", worst);
    const double inf = std::numeric_limits<double>::infinity();
    const double special[] = {0.0, -0.0, inf, -inf, std::nan(""), 800.0, -800.0, DBL_MIN, -DBL_MIN, 5e-324, 690.0, -690.0};
    for (double y : special) std::printf("%.17g %.17g\n", pxd::gb_exp(y, t.v), std::exp(y));
    return 0;
}
