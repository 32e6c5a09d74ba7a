// Receptor map build on the GPU: replaces receptor_cache::populate and
// partial_worker::populate (grid.cpp:115-195).
//
// The Lennard-Jones energy of every ligand type is a combination of the same sums over the
// receptor: with the receptor atoms grouped by (sigma, epsilon) into classes c,
//   E_t(p) = sum_c C_tc (s_tc^12 m12_c - s_tc^6 m6_c),     m_n = sum_i r_i^-n
// (s_tc the mean sigma, C_tc = 4 sqrt(eps_t eps_c)). grid_moment_kernel walks the receptor
// once per point for the Coulomb map and the sums of every class, so the exact part of the
// work no longer grows with the number of types; grid_lj_kernel forms the LJ gradients of a
// few types per walk and combines the sums into their energies.
//
// Precision. FP64 runs at 1/64 of FP32 here and bounded the build (84 % of the FP64 pipe busy)
// when the Coulomb terms and the LJ terms near a point were FP64 per (point, map). The terms
// of grid_moment_kernel are FP32 pairs and triples instead (device_pairs.cuh):
//   - atom and point coordinates are split into three parts, two of them on common power-of-two
//     grids, so that the differences of these parts are exact;
//   - the Coulomb energy is formed and summed in triples: its q/r terms of both signs cancel to
//     a small part of their size, and 1,900 terms of ~7 kcal/mol a unit charge in pairs left
//     1e-12 kcal/mol. The triple sum, and the pair sums of the gradient, are folded into FP64
//     every kMomentTile atoms or so;
//   - r^-6 and r^-12 are pairs; of atoms closer than 2 A they are formed and summed in FP64 from
//     the FP64 coordinates (the 12th power of a clash amplifies the coordinates' rounding most);
//   - the classes' energies are combined in FP64, and kept as the FP32 record and the FP32
//     remainder below it.
// Against exact sums over the same points, 1,866 atoms, points off the atoms: the Coulomb
// energies of a unit charge are off by 1.1e-13 kcal/mol in the median and 7e-13 at most, with
// or without an atom far away (4e-13 and 5e-12 with an FP64 loop over coordinates of two FP32
// parts); the LJ energies by 1e-15 of themselves in the median, and where |E| < 10 by 2e-13 kcal/mol
// in the median and 2e-11 at most (4e-8 and 2e-7 with FP32 terms under 1e-2 kcal/mol).
// The LJ gradients are FP32 per pair from hi + lo coordinate differences, folded into FP64
// every kGridTile atoms. Squared distances are floored at 1e-4 A^2 (a point that sits on an
// atom cannot overflow FP32) and records clamped to +-1e30 before the FP32 store.
//
// Measured, 81^3 points x 1,866 atoms: 12 maps in 14.9 ms (104 ms with FP64 terms per point and
// map): 8.4 ms for grid_moment_kernel (4.4 with Coulomb terms in pairs) and 3.0 ms for each
// walk of grid_lj_kernel over 6 types, both near the FP32 issue rate; all 99 types over
// 55 x 49 x 53 points in 16.7 ms (239 ms).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <vector>

#include "device_eval.cuh"
#include "device_pairs.cuh"
#include "../../include/pxdock_gb300_vdw.h"

namespace pxd {

constexpr int kGridThreads = 128;
constexpr int kMomentTile = 128;
constexpr int kGridTile = 256;  // atoms per FP32 partial sum of the LJ gradients
constexpr float kR2Floor = 1e-4f;
constexpr float kNearR2 = 4.f;  // A^2: closer atoms' LJ powers are FP64
constexpr float kFarR2 = 1e30f;  // A^2: farther atoms, whose squares FP32 does not hold, are FP64
// Systems that reach further than this from an atom to a point (A) give up the common hi
// grid, whose step would grow with them (an outlying atom would cost every point precision),
// for two-sum differences: 15 operations a pair more.
constexpr double kGridReach = 256.0;
constexpr double kRecordCeil = 1e30;
constexpr double kCoulombD = 332.0637141491396;  // kCoulombFactor, system.h:83
constexpr size_t kMomentBytes = 2 * sizeof(double);  // per point and class
// Workspace of the sums; larger boxes run in chunks of points. A chunk is at least four blocks per
// SM: a receptor whose atoms all have parameters of their own (1,866 classes) would get 26
// blocks in 96 MB, and 160 launches for 81^3 points.
constexpr size_t kMomentLimit = size_t(96) << 20, kMomentMost = size_t(2) << 30;

struct GridClass {
    int first, count;  // atoms [first, first + count) of the class-ordered list
    int slot;          // index of its sums, -1: epsilon 0, Coulomb only
};

struct FoldCoef {
    double a12, a6;  // C s^12, C s^6
};

// The atoms with LJ terms in receptor order, in tiles of kGridTile receptor atoms.
struct LjAtoms {
    const float4* hi;     // x, y, z rounded to FP32; class slot (int bits)
    const float4* lo;     // x, y, z remainders
    const int2* tiles;    // [n_tiles] first, count
    int n_tiles;
    const float2* kind;   // [n_slots] sigma, epsilon of a class
    const float2* types;  // [n_types] sigma, epsilon of a ligand type
};

struct GridArgs {
    const float4* hi;        // class order: first parts of the coordinates relative to `origin`, and charge
    const float4* lo;        // second parts
    const float4* rest;      // third parts of the coordinates
    const double4* x64;      // FP64 coordinates, charge
    const GridClass* classes;
    int n_classes, n_slots;  // n_slots: classes with sums
    int3 npts;
    double3 init;
    double spacing;
    double3 origin;
    double step, step_inv;   // hi grid
    int p0, n_points;        // points [p0, p0 + n_points) of the box in this launch
    int P;
    double* m6;              // [n_slots][n_points]
    double* m12;
    LjAtoms lj;
    const FoldCoef* coef;    // [n_types][n_slots]
    int n_types;
    float4* maps;            // [1 + n_types][P]
    float* e_lo;
};

__device__ __forceinline__ float clampf_rec(double v) {
    return static_cast<float>(fmin(fmax(v, -kRecordCeil), kRecordCeil));
}

__device__ __forceinline__ void store_record(const GridArgs& a, int slot, int p, double E, float gx, float gy, float gz) {
    const float hi = clampf_rec(E);
    a.maps[static_cast<size_t>(slot) * a.P + p] = make_float4(hi, gx, gy, gz);
    a.e_lo[static_cast<size_t>(slot) * a.P + p] =
        fabs(E) < kRecordCeil ? static_cast<float>(E - static_cast<double>(hi)) : 0.f;
}

__device__ __forceinline__ double to_double(F2 a) { return static_cast<double>(a.h) + static_cast<double>(a.l); }
__device__ __forceinline__ double to_double(F3 a) {
    return static_cast<double>(a.h) + (static_cast<double>(a.l) + static_cast<double>(a.m));
}

struct PointSums {
    F3 e;                   // Coulomb energy
    F2 x, y, z;             // and gradient
    double E, GX, GY, GZ;   // folded before
    F2 m6, m12;             // LJ sums of the current class
    double m6d, m12d;       // its FP64 atoms

    __device__ __forceinline__ void fold() {
        E += to_double(e);
        GX += to_double(x);
        GY += to_double(y);
        GZ += to_double(z);
        e = {0.f, 0.f, 0.f};
        x = y = z = {0.f, 0.f};
    }
};

// One coordinate of an atom or a point as three parts. The first two on the grids of `step` and
// 2^-24 step, so that the differences of two of them are exact; kWide: each the rounding of
// what is left.
template <bool kWide>
__host__ __device__ __forceinline__ F3 coord_parts(double r, double step, double step_inv) {
    constexpr double k24 = 16777216.0;
    const double h = kWide ? static_cast<double>(static_cast<float>(r)) : rint(r * step_inv) * step;
    const double d = r - h;
    const double l = kWide ? static_cast<double>(static_cast<float>(d)) : rint(d * step_inv * k24) * (step / k24);
    return {static_cast<float>(h), static_cast<float>(l), static_cast<float>(d - l)};
}

// a - p, its first part carrying the leading bits.
template <bool kWide>
__device__ __forceinline__ F3 coord_diff(float ah, float al, float am, F3 p) {
    float h = __fsub_rn(ah, p.h), l = __fsub_rn(al, p.l), m = __fsub_rn(am, p.m);
    if (kWide) {
        const F2 e = two_diff(ah, p.h), g = two_diff(al, p.l);
        const F2 k = two_sum(e.l, g.h);
        h = e.h;
        l = k.h;
        m = __fadd_rn(m, __fadd_rn(k.l, g.l));
    }
    const float s = __fadd_rn(h, l);
    return {s, __fsub_rn(l, __fsub_rn(s, h)), m};
}

// The vector from the point to the atom, its squared length in w.
__device__ __forceinline__ double4 vector64(double4 x, double3 p) {
    const double vx = x.x - p.x, vy = x.y - p.y, vz = x.z - p.z;
    return make_double4(vx, vy, vz, fmax(vx * vx + vy * vy + vz * vz, static_cast<double>(kR2Floor)));
}

__device__ __forceinline__ void add_powers64(double r2, PointSums& s) {
    const double inv = 1.0 / r2, n6 = inv * inv * inv;
    s.m6d += n6;
    s.m12d += n6 * n6;
}

// Adds one receptor atom to the sums of the point (px, py, pz; FP64 p64).
template <bool kLj, bool kWide>
__device__ __forceinline__ void grid_pair(const float4 ah, const float4 al, const float4 am, const double4* x64, F3 px,
                                          F3 py, F3 pz, double3 p64, PointSums& s) {
    const F3 dx = coord_diff<kWide>(ah.x, al.x, am.x, px), dy = coord_diff<kWide>(ah.y, al.y, am.y, py),
             dz = coord_diff<kWide>(ah.z, al.z, am.z, pz);
    F3 r2 = triple_norm2(dx, dy, dz);
    if (kWide && !(r2.h < kFarR2)) {  // also a coordinate that is not finite
        const double4 x = *x64, v = vector64(x, p64);
        const double rinv = rsqrt(v.w), qr = x.w * rinv, w = qr * rinv * rinv;
        s.E += qr;
        s.GX = fma(v.x, w, s.GX);
        s.GY = fma(v.y, w, s.GY);
        s.GZ = fma(v.z, w, s.GZ);
        if (kLj) add_powers64(v.w, s);
        return;
    }
    const bool near = r2.h < kNearR2;
    if (near) {
        if (r2.h < kR2Floor) r2 = {kR2Floor, 0.f, 0.f};
        if (kLj) add_powers64(vector64(*x64, p64).w, s);
    }
    F3 rinv;
    F2 inv;
    triple_rsqrt(r2, rinv, inv);
    // Coulomb: q/r and q (x - p)/r^3
    const F2 q = triple_acc(s.e, {ah.w, al.w}, rinv);
    const F2 w = pair_mul(q, inv);
    pair_acc(s.x, pair_mul(F2{dx.h, dx.l}, w));
    pair_acc(s.y, pair_mul(F2{dy.h, dy.l}, w));
    pair_acc(s.z, pair_mul(F2{dz.h, dz.l}, w));
    if (kLj) {
        F2 i6 = pair_mul(pair_square(inv), inv);
        F2 i12 = pair_square(i6);
        if (near) i6 = i12 = {0.f, 0.f};  // summed in FP64 above
        pair_acc(s.m6, i6);
        pair_acc(s.m12, i12);
    }
}

// One thread per point, 128 consecutive points (k fastest) per block, so that every thread
// reads the same atom of a shared-memory tile (broadcast). About 280 FP32 operations a pair:
// bound by FP32 issue.
template <bool kWide>
__global__ void __launch_bounds__(kGridThreads) grid_moment_kernel(const __grid_constant__ GridArgs a) {
    __shared__ float4 s_hi[kMomentTile];
    __shared__ float4 s_lo[kMomentTile];
    __shared__ float4 s_rest[kMomentTile];
    const int t = blockIdx.x * kGridThreads + threadIdx.x;
    const int p = a.p0 + t;
    const int nz = a.npts.z, ny = a.npts.y;
    const int k = p % nz;
    const int j = (p / nz) % ny;
    const int i = p / (nz * ny);
    // grid.cpp:159-163: point = init + spacing * index, formed in FP64
    const double3 p64 = make_double3(a.init.x + a.spacing * i, a.init.y + a.spacing * j, a.init.z + a.spacing * k);
    const F3 px = coord_parts<kWide>(p64.x - a.origin.x, a.step, a.step_inv);
    const F3 py = coord_parts<kWide>(p64.y - a.origin.y, a.step, a.step_inv);
    const F3 pz = coord_parts<kWide>(p64.z - a.origin.z, a.step, a.step_inv);
    PointSums s{};
    int since = 0;  // atoms since the last fold
    for (int c = 0; c < a.n_classes; ++c) {
        const GridClass gc = a.classes[c];
        for (int t0 = 0; t0 < gc.count; t0 += kMomentTile) {
            const int n = min(kMomentTile, gc.count - t0);
            const int base = gc.first + t0;
            __syncthreads();
            for (int u = threadIdx.x; u < n; u += kGridThreads) {
                s_hi[u] = a.hi[base + u];
                s_lo[u] = a.lo[base + u];
                s_rest[u] = a.rest[base + u];
            }
            __syncthreads();
            if (gc.slot >= 0) {
                for (int u = 0; u < n; ++u)
                    grid_pair<true, kWide>(s_hi[u], s_lo[u], s_rest[u], a.x64 + base + u, px, py, pz, p64, s);
            } else {
                for (int u = 0; u < n; ++u)
                    grid_pair<false, kWide>(s_hi[u], s_lo[u], s_rest[u], a.x64 + base + u, px, py, pz, p64, s);
            }
            // the low part of a long sum would round by more than its terms do
            since += n;
            if (since >= kMomentTile) {
                s.fold();
                since = 0;
            }
        }
        if (gc.slot >= 0) {
            if (t < a.n_points) {
                const size_t o = static_cast<size_t>(gc.slot) * a.n_points + t;
                a.m6[o] = s.m6d + to_double(s.m6);
                a.m12[o] = s.m12d + to_double(s.m12);
            }
            s.m6 = s.m12 = {0.f, 0.f};
            s.m6d = s.m12d = 0.0;
        }
    }
    s.fold();
    if (t < a.n_points) {
        store_record(a, 0, p, s.E * kCoulombD, clampf_rec(s.GX * kCoulombD), clampf_rec(s.GY * kCoulombD),
                     clampf_rec(s.GZ * kCoulombD));
    }
}

// LJ records of kTypes ligand types per thread: the FP32 gradients from one walk over the
// receptor (~38 operations a pair that the types share, 11 a type), the energies from the
// classes' sums (two FP64 operations a type and class). Bound by FP32 issue.
template <int kTypes>
__global__ void __launch_bounds__(kGridThreads) grid_lj_kernel(const __grid_constant__ GridArgs a) {
    __shared__ float4 s_x[kGridTile];
    __shared__ float4 s_lo[kGridTile];
    __shared__ float2 s_p[kGridTile][kTypes];  // (mean sigma)^2, 4 sqrt(eps eps) of an atom and a type
    const int t = blockIdx.x * kGridThreads + threadIdx.x;
    const int t0 = blockIdx.y * kTypes;
    const int p = a.p0 + t;
    const int nz = a.npts.z, ny = a.npts.y;
    const int k = p % nz;
    const int j = (p / nz) % ny;
    const int i = p / (nz * ny);
    const double px = a.init.x + a.spacing * i, py = a.init.y + a.spacing * j, pz = a.init.z + a.spacing * k;
    const float3 pt = make_float3(static_cast<float>(px), static_cast<float>(py), static_cast<float>(pz));
    const float3 pl = make_float3(static_cast<float>(px - pt.x), static_cast<float>(py - pt.y),
                                  static_cast<float>(pz - pt.z));
    double GX[kTypes], GY[kTypes], GZ[kTypes];
#pragma unroll
    for (int g = 0; g < kTypes; ++g) GX[g] = GY[g] = GZ[g] = 0.0;
    for (int b = 0; b < a.lj.n_tiles; ++b) {
        const int2 tile = a.lj.tiles[b];
        __syncthreads();
        for (int u = threadIdx.x; u < tile.y; u += kGridThreads) {
            s_x[u] = a.lj.hi[tile.x + u];
            s_lo[u] = a.lj.lo[tile.x + u];
            const float2 se = a.lj.kind[__float_as_int(s_x[u].w)];
            for (int g = 0; g < kTypes; ++g) {
                const float2 tse = a.lj.types[min(t0 + g, a.n_types - 1)];
                const float s = (tse.x + se.x) * 0.5f;
                s_p[u][g] = make_float2(s * s, sqrtf(tse.y * se.y) * 4.f);
            }
        }
        __syncthreads();
        float gx[kTypes], gy[kTypes], gz[kTypes];
#pragma unroll
        for (int g = 0; g < kTypes; ++g) gx[g] = gy[g] = gz[g] = 0.f;
        for (int u = 0; u < tile.y; ++u) {
            const float4 at = s_x[u];
            const float4 lo = s_lo[u];
            const float vx = (at.x - pt.x) + (lo.x - pl.x), vy = (at.y - pt.y) + (lo.y - pl.y),
                        vz = (at.z - pt.z) + (lo.z - pl.z);
            const float r2 = fmaxf(vx * vx + vy * vy + vz * vz, kR2Floor);
            const float rinv2 = 1.f / r2;
#pragma unroll
            for (int g = 0; g < kTypes; ++g) {
                const float2 sc = s_p[u][g];
                const float x = sc.x * rinv2;
                const float u6 = x * x * x;
                const float u12 = u6 * u6;
                // grad_point -= vec * de_dr_r, de_dr_r = C(-12 u12 + 6 u6) / r^2 (pair.h:42-60)
                const float w = sc.y * (12.f * u12 - 6.f * u6) * rinv2;
                gx[g] = fmaf(vx, w, gx[g]);
                gy[g] = fmaf(vy, w, gy[g]);
                gz[g] = fmaf(vz, w, gz[g]);
            }
        }
#pragma unroll
        for (int g = 0; g < kTypes; ++g) {
            GX[g] += gx[g];
            GY[g] += gy[g];
            GZ[g] += gz[g];
        }
    }
    if (t >= a.n_points) return;
    double E[kTypes];
#pragma unroll
    for (int g = 0; g < kTypes; ++g) E[g] = 0.0;
    for (int c = 0; c < a.n_slots; ++c) {
        const size_t o = static_cast<size_t>(c) * a.n_points + t;
        const double m6 = a.m6[o], m12 = a.m12[o];
#pragma unroll
        for (int g = 0; g < kTypes; ++g) {
            const FoldCoef f = a.coef[static_cast<size_t>(min(t0 + g, a.n_types - 1)) * a.n_slots + c];
            E[g] += f.a12 * m12 - f.a6 * m6;
        }
    }
#pragma unroll
    for (int g = 0; g < kTypes; ++g)
        if (t0 + g < a.n_types)
            store_record(a, 1 + t0 + g, p, E[g], clampf_rec(GX[g]), clampf_rec(GY[g]), clampf_rec(GZ[g]));
}

// Types per thread: as even as groups of at most 8 allow (a smaller group repeats the walk's
// shared part more often, a larger one no longer fits the registers).
static void launch_lj(const GridArgs& a, int blocks, cudaStream_t s) {
    const int groups = (a.n_types + 7) / 8;
    const int per = (a.n_types + groups - 1) / groups;
    const dim3 grid(blocks, groups);
    if (per > 6)
        grid_lj_kernel<8><<<grid, kGridThreads, 0, s>>>(a);
    else if (per > 4)
        grid_lj_kernel<6><<<grid, kGridThreads, 0, s>>>(a);
    else if (per > 2)
        grid_lj_kernel<4><<<grid, kGridThreads, 0, s>>>(a);
    else
        grid_lj_kernel<2><<<grid, kGridThreads, 0, s>>>(a);
}

// Builds the Coulomb map (slot 0) and the maps of `types` (slots 1..) over the context's
// box from every non-rotor receptor atom (grid.cpp:119-123, 173). Synchronous.
int launch_grid_build(pxd_context* ctx, const std::vector<int>& types) {
    // (epsilon, sigma) -> atoms, by the numbers' bits: a NaN has no place among numbers
    std::map<std::pair<int64_t, int64_t>, std::vector<int>> by_kind;
    for (int i = 0; i < ctx->n_rec; ++i)
        if (!ctx->is_mov[i]) by_kind[{number_bits(ctx->rec_epsilon[i]), number_bits(ctx->rec_sigma[i])}].push_back(i);
    GridArgs a{};
    a.npts = make_int3(ctx->box.npoints[0], ctx->box.npoints[1], ctx->box.npoints[2]);
    a.init = make_double3(ctx->box.init_xyz[0], ctx->box.init_xyz[1], ctx->box.init_xyz[2]);
    a.spacing = ctx->box.spacing;
    a.P = ctx->grid.P;
    a.maps = ctx->maps;
    a.e_lo = const_cast<float*>(ctx->grid.e_lo);
    a.n_types = static_cast<int>(types.size());
    // the hi grid: 2^24 steps span the largest coordinate difference of an atom and a point
    double half[3], reach = 0.0;
    for (int d = 0; d < 3; ++d) {
        half[d] = 0.5 * (ctx->box.npoints[d] - 1) * ctx->box.spacing;
        (&a.origin.x)[d] = ctx->box.init_xyz[d] + half[d];
        reach = std::max(reach, half[d]);
    }
    bool wide = !(reach < kGridReach);
    for (const auto& [bits, atoms] : by_kind)
        for (int i : atoms)
            for (int d = 0; d < 3; ++d) {
                const double r = std::fabs(ctx->rec_xyz[3 * i + d] - (&a.origin.x)[d]) + half[d];
                if (r < kGridReach)
                    reach = std::max(reach, r);
                else  // also where r is not a number
                    wide = true;
            }
    a.step = std::ldexp(1.0, std::ilogb(std::max(reach, 1.0)) + 1 - 24);
    a.step_inv = 1.0 / a.step;
    std::vector<float4> hi, lo, rest;
    std::vector<double4> x64;
    std::vector<GridClass> classes;
    std::vector<int> order;  // receptor atoms in class order
    std::vector<std::pair<double, double>> kinds;  // of the classes with sums
    for (const auto& [bits, atoms] : by_kind) {
        const std::pair<double, double> kind(ctx->rec_epsilon[atoms[0]], ctx->rec_sigma[atoms[0]]);
        const bool lj = kind.first != 0.0;
        classes.push_back({static_cast<int>(hi.size()), static_cast<int>(atoms.size()),
                           lj ? static_cast<int>(kinds.size()) : -1});
        if (lj) kinds.push_back(kind);
        for (int i : atoms) {
            order.push_back(i);
            F3 x[3];
            for (int d = 0; d < 3; ++d) {
                const double r = ctx->rec_xyz[3 * i + d] - (&a.origin.x)[d];
                x[d] = wide ? coord_parts<true>(r, a.step, a.step_inv) : coord_parts<false>(r, a.step, a.step_inv);
            }
            const float q = static_cast<float>(ctx->rec_charge[i]);
            hi.push_back(make_float4(x[0].h, x[1].h, x[2].h, q));
            lo.push_back(make_float4(x[0].l, x[1].l, x[2].l, static_cast<float>(ctx->rec_charge[i] - q)));
            rest.push_back(make_float4(x[0].m, x[1].m, x[2].m, 0.f));
            x64.push_back(make_double4(ctx->rec_xyz[3 * i], ctx->rec_xyz[3 * i + 1], ctx->rec_xyz[3 * i + 2],
                                       ctx->rec_charge[i]));
        }
    }
    a.n_classes = static_cast<int>(classes.size());
    a.n_slots = static_cast<int>(kinds.size());
    std::vector<FoldCoef> coef;
    for (int t : types)
        for (const auto& [eps, sigma] : kinds) {
            const double s = (PXD_VDW_SIGMA[t] + sigma) * 0.5, s6 = std::pow(s, 6.0);
            const double C = std::sqrt(PXD_VDW_EPSILON[t] * eps) * 4.0;
            coef.push_back({C * s6 * s6, C * s6});
        }
    // the LJ atoms in receptor order, cut at every kGridTile receptor atoms
    std::vector<float4> lj_hi, lj_lo;
    std::vector<int2> tiles;
    std::vector<float2> kind_se, type_se;
    for (const auto& [eps, sigma] : kinds)
        kind_se.push_back(make_float2(static_cast<float>(sigma), static_cast<float>(eps)));
    for (int t : types)
        type_se.push_back(make_float2(static_cast<float>(PXD_VDW_SIGMA[t]), static_cast<float>(PXD_VDW_EPSILON[t])));
    std::vector<int> slot_of(ctx->n_rec, -1);
    for (const GridClass& c : classes)
        for (int u = 0; u < c.count; ++u) slot_of[order[c.first + u]] = c.slot;
    for (int i = 0, seen = 0; i < ctx->n_rec; ++i) {
        if (ctx->is_mov[i]) continue;
        if (seen++ % kGridTile == 0) tiles.push_back(make_int2(static_cast<int>(lj_hi.size()), 0));
        if (slot_of[i] < 0) continue;
        const double* x = &ctx->rec_xyz[3 * i];
        const float3 h = make_float3(static_cast<float>(x[0]), static_cast<float>(x[1]), static_cast<float>(x[2]));
        float bits;
        std::memcpy(&bits, &slot_of[i], sizeof(bits));
        lj_hi.push_back(make_float4(h.x, h.y, h.z, bits));
        lj_lo.push_back(make_float4(static_cast<float>(x[0] - h.x), static_cast<float>(x[1] - h.y),
                                    static_cast<float>(x[2] - h.z), 0.f));
        ++tiles.back().y;
    }
    a.lj.n_tiles = static_cast<int>(tiles.size());
    // one allocation: inputs, then the sums of a chunk of points
    const size_t n_slots = std::max(1, a.n_slots);
    const size_t per_point = kMomentBytes * n_slots, fill = size_t(4) * ctx->n_sm * kGridThreads;
    const size_t fit = std::max(kMomentLimit / per_point, std::min(fill, kMomentMost / per_point));
    size_t chunk = std::min<size_t>(a.P, std::max<size_t>(fit / kGridThreads, 1) * kGridThreads);
    std::vector<unsigned char> in;
    auto put = [&in](const auto& v) {
        const size_t off = in.size(), bytes = v.size() * sizeof(v[0]);
        in.resize(off + (bytes + 31) / 32 * 32 + 32);
        if (bytes) std::memcpy(in.data() + off, v.data(), bytes);
        return off;
    };
    const size_t o_hi = put(hi), o_lo = put(lo), o_rest = put(rest), o_x = put(x64), o_cls = put(classes), o_coef = put(coef);
    const size_t o_lh = put(lj_hi), o_ll = put(lj_lo), o_tile = put(tiles), o_kind = put(kind_se), o_type = put(type_se);
    cudaStream_t s = ctx->stream;
    char* mem = nullptr;
    int rc;
    for (;; chunk = (chunk / 2 + kGridThreads - 1) / kGridThreads * kGridThreads) {  // smaller where memory is short
        rc = cuda_check(ctx, cudaMallocAsync(reinterpret_cast<void**>(&mem), in.size() + per_point * chunk, s),
                        "map build workspace");
        if (rc != PXD_ERR_NOMEM || chunk <= kGridThreads) break;
        cudaGetLastError();
    }
    if (rc) return rc;
    queue_copy(ctx, &rc, mem, in.data(), in.size(), cudaMemcpyHostToDevice, s, "map build inputs");
    a.hi = reinterpret_cast<const float4*>(mem + o_hi);
    a.lo = reinterpret_cast<const float4*>(mem + o_lo);
    a.rest = reinterpret_cast<const float4*>(mem + o_rest);
    a.x64 = reinterpret_cast<const double4*>(mem + o_x);
    a.classes = reinterpret_cast<const GridClass*>(mem + o_cls);
    a.coef = reinterpret_cast<const FoldCoef*>(mem + o_coef);
    a.lj.hi = reinterpret_cast<const float4*>(mem + o_lh);
    a.lj.lo = reinterpret_cast<const float4*>(mem + o_ll);
    a.lj.tiles = reinterpret_cast<const int2*>(mem + o_tile);
    a.lj.kind = reinterpret_cast<const float2*>(mem + o_kind);
    a.lj.types = reinterpret_cast<const float2*>(mem + o_type);
    a.m6 = reinterpret_cast<double*>(mem + in.size());
    a.m12 = a.m6 + n_slots * chunk;
    for (int p0 = 0; p0 < a.P && !rc; p0 += static_cast<int>(chunk)) {
        a.p0 = p0;
        a.n_points = std::min(static_cast<int>(chunk), a.P - p0);
        const int blocks = (a.n_points + kGridThreads - 1) / kGridThreads;
        if (wide)
            grid_moment_kernel<true><<<blocks, kGridThreads, 0, s>>>(a);
        else
            grid_moment_kernel<false><<<blocks, kGridThreads, 0, s>>>(a);
        if (a.n_types > 0) launch_lj(a, blocks, s);
        rc = cuda_check(ctx, cudaGetLastError(), "map build launch");
    }
    cudaFreeAsync(mem, s);
    return sync_copies(ctx, rc, s, "grid build");
}

}  // namespace pxd
