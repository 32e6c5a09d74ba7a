// Reported energy of one pose, no gradient: the value of
// binding_system_interactions::put_gradients (interaction.cpp:259-350) at the pose that an
// optimiser or a search returns, to within 1e-3 kcal/mol of the FP64 reference at any
// energy. The optimiser steers on the FP32 evaluation (device_eval.cuh); this evaluation
// gives the reported number. One warp per pose, every lane returns the same value.
//
// The ligand's moderate terms and the map lookups are FP32 pairs (device_pairs.cuh): a pose's
// coordinates are FP32, so their differences are exact pairs. In FP64 the pair terms over
// 1 kcal/mol alone (present in nearly every round of 32) held the FP64 pipe for 20,000 of
// the 25,000 cycles of a 42-atom pose: score_kernel took 6.6 ms for 65,536 poses, and takes 2.2.
//
// Precision per term, against the FP64 objective:
//   - grid lookups (grid.cpp:197-303): an atom's place in its cell from the box's geometry in
//     three FP32 parts, weights and the cell's sum in pairs, over map energies E = FP32
//     record + FP32 residual of the FP64 sum (grid build): 6e-16 of the cell's largest energy
//     in the median (1.2e-15 with weights from an FP64 place in the box, whose fraction of a
//     cell rounds at 1e-14). The penalty of an atom outside is FP64;
//   - bonds (interaction.cpp:27-47) of the ligand: pairs;
//   - its intra pairs (pair.h:25-60): FP32 terms up to 1 kcal/mol, with ~1e-6 of their larger
//     part (Coulomb or LJ; the 12th power multiplies the rounding of 1/r twelvefold), pairs
//     above, with ~2e-13 of themselves;
//   - terms and lookups over kPairTop, of coincident atoms or of atoms flung apart: FP64, and
//     summed in FP64, so that what pairs round off stays below 1e-8 kcal/mol, a hundredth of
//     what FP32 angles leave;
//   - angles and dihedrals (interaction.cpp:49-117): FP32 geometry, sums in pairs. These are
//     bounded (0.5 k pi^2, 2 sum k): an FP32 angle error of ~1e-7 rad moves a term by at
//     most k |theta - theta0| 1e-7, ~1e-5 kcal/mol;
//   - receptor rotor atoms (interaction.cpp:316-336): FP64 rotations of FP64 coordinates; their
//     terms and the explicit inter pairs in FP32, recomputed in FP64 from FP64 parameters
//     when the FP32 term exceeds 1 kcal/mol (FP32 carries ~1e-6 of a term, so a 1e6 clash
//     would be off by 1 kcal/mol; terms under 1 kcal/mol stay below 1e-6).
// Every per-lane sum runs in a fixed order and the warp sum is a fixed butterfly, so the
// value repeats bit for bit.
#pragma once

#include "device_eval.cuh"
#include "device_pairs.cuh"

namespace pxd {

struct D3 {
    double x, y, z;
};
__device__ __forceinline__ D3 d3_sub(D3 a, D3 b) { return D3{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ double d3_dot(D3 a, D3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ D3 d3_of(float3 v) {
    return D3{static_cast<double>(v.x), static_cast<double>(v.y), static_cast<double>(v.z)};
}

// Sum over the warp in FP64 (xor butterfly: every lane adds the same two values in the
// same order, so all lanes hold the same sum).
__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(kFull, v, off);
    return v;
}

constexpr double kCoulombD64 = 332.0637141491396;  // kCoulombFactor, system.h:83
constexpr float kPairFp64 = 1.f;                   // kcal/mol: larger FP32 terms are recomputed
constexpr float kPairTop = 1e4f;                   // kcal/mol: larger terms in pairs are FP64

// Pair energy A/r + C((S2/r^2)^6 - (S2/r^2)^3) from FP64 parameters and coordinates.
__device__ __forceinline__ double pair_energy64(double4 p, D3 xi, D3 xj) {
    const D3 r = d3_sub(xj, xi);
    const double r2 = d3_dot(r, r);
    const double x = p.z / r2;
    const double u6 = x * x * x;
    return p.x / sqrt(r2) + p.y * (u6 * u6 - u6);
}

// Energy of the receptor's rotor-touching terms (intra_molecular_interactions) with positions
// given in FP32 (P32) and FP64 (P64) by index.
template <class P32, class P64>
__device__ double topo_energy64(const DevTopo& t, const P32& pos32, const P64& pos64, int lane) {
    double e = 0.0;
    for (int s = lane; s < t.n_bond_slots; s += kWarp) {
        const int2 ij = __ldg(&t.bond_ij[s]);
        if (ij.x < 0) continue;
        const double2 p = __ldg(&t.bond_p64[s]);
        const D3 d = d3_sub(pos64(ij.y), pos64(ij.x));
        const double dr = sqrt(d3_dot(d, d)) - p.y;
        e += 0.5 * p.x * (dr * dr);
    }
    for (int s = lane; s < t.n_angle_slots; s += kWarp) {
        const int4 ijk = __ldg(&t.angle_ijk[s]);
        if (ijk.x < 0) continue;
        const float2 p = __ldg(&t.angle_p[s]);
        const float3 xi = pos32(ijk.x), xj = pos32(ijk.y), xk = pos32(ijk.z);
        const float3 v0 = sub3(xj, xi), v1 = sub3(xj, xk);
        const float3 c = cross3(v0, v1);
        const float theta = atan2f(sqrtf(dot3(c, c)), dot3(v0, v1) + kEpsF);
        const double delta = static_cast<double>(theta) - __ldg(&t.angle_p64[s]).y;
        e += 0.5 * static_cast<double>(p.x) * (delta * delta);
    }
    for (int s = lane; s < t.n_dih_slots; s += kWarp) {
        const int4 q = __ldg(&t.dih_ijkl[s]);
        if (q.x < 0) continue;
        const float3 pi = pos32(q.x), pj = pos32(q.y), pk = pos32(q.z), pl = pos32(q.w);
        const float3 rij = sub3(pj, pi), rkj = sub3(pj, pk), rkl = sub3(pl, pk);
        const float3 m = cross3(rij, rkj), n = cross3(rkj, rkl);
        const float3 w = cross3(m, n);
        const float phi = atan2f(sqrtf(dot3(w, w)), dot3(m, n) + kEpsF);
        const float theta = dot3(rij, n) < 0.f ? phi : -phi;
        const int2 tr = __ldg(&t.dih_terms[s]);
        for (int u = 0; u < tr.y; ++u) {
            const double4 term = t.dih_term64[tr.x + u];  // k, periodicity, phase
            const float delta = theta * static_cast<float>(term.y) - static_cast<float>(term.z);
            e += term.x * (1.0 + static_cast<double>(cosf(delta)));
        }
    }
    for (int s = lane; s < t.n_pair_slots; s += kWarp) {
        const int2 ij = __ldg(&t.pair_ij[s]);
        if (ij.x < 0) continue;
        const float3 xi = pos32(ij.x), xj = pos32(ij.y);
        const float4 p = __ldg(&t.pair_p[s]);
        const float3 rij = sub3(xj, xi);
        const float r2 = dot3(rij, rij);
        const float rinv = rsqrtf(r2);
        const float x = p.z * rinv * rinv;
        const float u6 = x * x * x;
        const float en = fmaf(p.y, u6 * u6 - u6, p.x * rinv);
        if (fabsf(en) <= kPairFp64)
            e += static_cast<double>(en);
        else  // also inf / NaN
            e += pair_energy64(t.pair_p64[s], pos64(ij.x), pos64(ij.y));
    }
    return e;
}

// Squared distances for which a bond or pair term stays in pairs; outside (coincident atoms, or
// atoms flung apart) it is FP64.
constexpr float kPairR2Min = 1e-2f, kPairR2Max = 1e30f;

__device__ __forceinline__ F2 atom_distance2(const float* x, int i, int j) {
    return pair_norm2(two_diff(x[3 * j], x[3 * i]), two_diff(x[3 * j + 1], x[3 * i + 1]),
                      two_diff(x[3 * j + 2], x[3 * i + 2]));
}

// Energy of the ligand's terms at FP32 coordinates x: terms in pairs added to `e`, FP64 terms to
// `e64`.
__device__ __forceinline__ void ligand_energy(const DevTopo& t, const float* x, F2& e, double& e64, int lane) {
    auto pos = [x](int i) { return make_float3(x[3 * i], x[3 * i + 1], x[3 * i + 2]); };
    auto pos64 = [x](int i) {
        return D3{static_cast<double>(x[3 * i]), static_cast<double>(x[3 * i + 1]), static_cast<double>(x[3 * i + 2])};
    };
    for (int s = lane; s < t.n_bond_slots; s += kWarp) {
        const int2 ij = __ldg(&t.bond_ij[s]);
        if (ij.x < 0) continue;
        const F2 r2 = atom_distance2(x, ij.x, ij.y);
        if (r2.h > kPairR2Min && r2.h < kPairR2Max) {
            const float2 p = __ldg(&t.bond_p[s]), pl = __ldg(&t.bond_lo[s]);
            F2 rinv, inv;
            pair_rsqrt(r2, rinv, inv);
            const F2 dr = pair_sub(pair_norm(pair_mul(r2, rinv)), {p.y, pl.y});
            const F2 en = pair_mul({0.5f * p.x, 0.5f * pl.x}, pair_square(pair_norm(dr)));
            if (en.h <= kPairTop) {
                pair_acc(e, en);
                continue;
            }
        }
        const double2 p = __ldg(&t.bond_p64[s]);
        const D3 d = d3_sub(pos64(ij.y), pos64(ij.x));
        const double dr = sqrt(d3_dot(d, d)) - p.y;
        e64 += 0.5 * p.x * (dr * dr);
    }
    for (int s = lane; s < t.n_angle_slots; s += kWarp) {
        const int4 ijk = __ldg(&t.angle_ijk[s]);
        if (ijk.x < 0) continue;
        const float2 p = __ldg(&t.angle_p[s]);
        const float3 xi = pos(ijk.x), xj = pos(ijk.y), xk = pos(ijk.z);
        const float3 v0 = sub3(xj, xi), v1 = sub3(xj, xk);
        const float3 c = cross3(v0, v1);
        const float theta = atan2f(sqrtf(dot3(c, c)), dot3(v0, v1) + kEpsF);
        const F2 delta = pair_sub({theta, 0.f}, {p.y, __ldg(&t.angle_lo[s])});
        pair_acc(e, pair_mul(pair_square(pair_norm(delta)), 0.5f * p.x));
    }
    for (int s = lane; s < t.n_dih_slots; s += kWarp) {
        const int4 q = __ldg(&t.dih_ijkl[s]);
        if (q.x < 0) continue;
        const float3 pi = pos(q.x), pj = pos(q.y), pk = pos(q.z), pl = pos(q.w);
        const float3 rij = sub3(pj, pi), rkj = sub3(pj, pk), rkl = sub3(pl, pk);
        const float3 m = cross3(rij, rkj), n = cross3(rkj, rkl);
        const float3 w = cross3(m, n);
        const float phi = atan2f(sqrtf(dot3(w, w)), dot3(m, n) + kEpsF);
        const float theta = dot3(rij, n) < 0.f ? phi : -phi;
        const int2 tr = __ldg(&t.dih_terms[s]);
        for (int u = 0; u < tr.y; ++u) {
            const float4 term = __ldg(&t.dih_term[tr.x + u]);  // k, periodicity, phase
            const float delta = theta * term.y - term.z;
            pair_acc(e, pair_mul({term.x, __ldg(&t.dih_lo[tr.x + u])}, two_diff(1.f, -cosf(delta))));
        }
    }
    for (int s = lane; s < t.n_pair_slots; s += kWarp) {
        const int2 ij = __ldg(&t.pair_ij[s]);
        if (ij.x < 0) continue;
        const float4 p = __ldg(&t.pair_p[s]);  // A, C, S2
        const float3 rij = sub3(pos(ij.y), pos(ij.x));
        const float d2 = dot3(rij, rij);
        const float d_1 = rsqrtf(d2);
        const float v = p.z * d_1 * d_1;
        const float v6 = v * v * v;
        const float en = fmaf(p.y, v6 * v6 - v6, p.x * d_1);
        if (fabsf(en) <= kPairFp64) {
            pair_acc(e, F2{en, 0.f});
            continue;
        }
        const F2 r2 = atom_distance2(x, ij.x, ij.y);
        if (fabsf(en) <= kPairTop && r2.h > kPairR2Min && r2.h < kPairR2Max) {  // not for an infinite or NaN term
            const float4 pl = __ldg(&t.pair_lo[s]);
            F2 rinv, inv;
            pair_rsqrt(r2, rinv, inv);
            const F2 u = pair_mul(inv, F2{p.z, pl.z});
            const F2 u6 = pair_mul(pair_square(u), u);
            pair_acc(e, pair_mul(pair_sub(pair_square(u6), u6), F2{p.y, pl.y}));
            pair_acc(e, pair_mul(rinv, F2{p.x, pl.x}));
        } else {
            e64 += pair_energy64(t.pair_p64[s], pos64(ij.x), pos64(ij.y));
        }
    }
}

// One axis of an atom's place in the maps (receptor_cache::get, grid.cpp:211-262): its cell and
// its fraction of the cell as a pair; -1 or 1 if it is below or above the box (the fraction is
// the face's), also for a coordinate that is not finite.
__device__ __forceinline__ int grid_place(const float* init, const DevGrid& g, int npts, float at, int& cell, F2& frac) {
    const int last = npts - 2;  // the last cell
    const float p = fmaxf(fminf(at, 1e9f), -1e9f);
    int c = static_cast<int>(floorf((p - init[0]) * g.spacing_inv));
    c = min(max(c, 0), last);
    // r = p - init - c spacing: the leading parts exactly, the small ones in a pair
    const F2 d = two_diff(p, init[0]);
    const F2 b = pair_mul({g.spacing_p[0], 0.f}, static_cast<float>(c));  // exact product
    F2 r = two_diff(d.h, b.h);
    F2 small{d.l, r.l};
    pair_acc(small.h, small.l, -b.l, 0.f);
    pair_acc(small.h, small.l, -init[1], -init[2]);
    const F2 b1 = pair_mul({g.spacing_p[1], 0.f}, static_cast<float>(c));
    pair_acc(small.h, small.l, -b1.h, -fmaf(g.spacing_p[2], static_cast<float>(c), b1.l));
    r.l = 0.f;
    pair_acc(r, small);
    r = pair_norm(r);
    const F2 sp{g.spacing_p[0], g.spacing_p[1]};
    // the cell's FP32 estimate can be one off next to a grid point
    if (r.h < 0.f && c > 0) {
        --c;
        pair_acc(r, sp);
    } else if (c < last && (r.h - sp.h) + (r.l - sp.l) >= 0.f) {
        ++c;
        r = pair_sub(r, sp);
    }
    r = pair_norm(r);
    const F2 over = pair_norm(pair_sub(r, sp));
    cell = c;
    if (c == 0 && r.h < 0.f) {
        frac = {0.f, 0.f};
        return -1;
    }
    if (c == last && over.h >= 0.f) {
        frac = {1.f, 0.f};
        return 1;
    }
    frac = pair_norm(pair_mul(r, F2{g.spacing_inv_p[0], g.spacing_inv_p[1]}));
    return 0;
}

// How far a coordinate lies outside the box on the given side, in cells.
__device__ __forceinline__ double grid_beyond(const DevGrid& g, double from_init, int side, int npts) {
    const double f = from_init * g.spacing_inv64;
    return side < 0 ? -f : f - (npts - 1);
}

// receptor_cache::get (grid.cpp:197-262) energy for an atom of charge q at p.
__device__ __forceinline__ void grid_energy(const DevGrid& g, int slot, F2 q, float3 p, F2& e, double& e64) {
    int cx, cy, cz;
    F2 x, y, z;
    const int ox = grid_place(g.init_p[0], g, g.npts.x, p.x, cx, x), oy = grid_place(g.init_p[1], g, g.npts.y, p.y, cy, y),
              oz = grid_place(g.init_p[2], g, g.npts.z, p.z, cz, z);
    if (ox | oy | oz) {
        double out = 0.0;
        if (ox) out += grid_beyond(g, p.x - g.init64.x, ox, g.npts.x);
        if (oy) out += grid_beyond(g, p.y - g.init64.y, oy, g.npts.y);
        if (oz) out += grid_beyond(g, p.z - g.init64.z, oz, g.npts.z);
        if (out > 0.0) e64 += out * g.spacing64 * g.slope64;
    }
    const F2 one{1.f, 0.f};
    const F2 mx = pair_norm(pair_sub(one, x)), my = pair_norm(pair_sub(one, y)), mz = pair_norm(pair_sub(one, z));
    const F2 xy[4] = {pair_mul(mx, my), pair_mul(x, my), pair_mul(mx, y), pair_mul(x, y)};
    const int sy = g.npts.z, sx = g.npts.y * g.npts.z;
    const int base = cx * sx + cy * sy + cz;
    const size_t P = static_cast<size_t>(g.P);
    F2 ec{0.f, 0.f}, ev{0.f, 0.f};
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const int off = base + (c & 1 ? sx : 0) + (c & 2 ? sy : 0) + (c & 4 ? 1 : 0);
        const F2 w = pair_mul(xy[c & 3], c & 4 ? z : mz);
        pair_acc(ec, pair_mul(w, F2{__ldg(&g.maps[off].x), __ldg(&g.e_lo[off])}));
        if (slot > 0) pair_acc(ev, pair_mul(w, F2{__ldg(&g.maps[slot * P + off].x), __ldg(&g.e_lo[slot * P + off])}));
    }
    pair_acc(ev, pair_mul(pair_norm(ec), q));
    if (fabsf(ev.h) <= kPairTop)
        pair_acc(e, ev);
    else
        e64 += static_cast<double>(ev.h) + static_cast<double>(ev.l);
}

// Reported energy of the pose x = [ligand xyz (3N) | receptor torsions] (shared memory, the
// optimiser's flat layout). b.loc_grad serves as scratch for the FP64 positions of the
// receptor's local atoms (24 of its 64 bytes per atom); the next evaluation clears it.
static __device__ __noinline__ double energy64(const EvalEnv& env, const DevLigand& L, const float* x,
                                               const PoseBufs& b, int lane) {
    const int N = L.n_atoms;
    const int n3 = 3 * N;
    const DevReceptor& R = env.rec;
    double* loc64 = reinterpret_cast<double*>(b.loc_grad);
    // receptor rotor atoms (receptor_torsion2xyz, interaction.cpp:316-336; the Rodrigues
    // matrix of math.cpp:62-94)
    for (int l = lane; l < R.n_local; l += kWarp) {
        const double4 v = R.local_xyz064[l];
        double px = v.x, py = v.y, pz = v.z;
        if (l < R.n_mov) {
            const int r = static_cast<int>(v.w);
            const double4 k = R.rotor_axis64[r];
            const double4 o = R.rotor_origin64[r];
            double st, ct;
            sincos(static_cast<double>(x[n3 + r]), &st, &ct);
            const double omc = 1.0 - ct;
            const double r00 = ct + k.x * k.x * omc, r01 = k.x * k.y * omc - k.z * st, r02 = k.x * k.z * omc + k.y * st;
            const double r10 = k.y * k.x * omc + k.z * st, r11 = ct + k.y * k.y * omc, r12 = k.y * k.z * omc - k.x * st;
            const double r20 = k.z * k.x * omc - k.y * st, r21 = k.z * k.y * omc + k.x * st, r22 = ct + k.z * k.z * omc;
            px = r00 * v.x + r01 * v.y + r02 * v.z + o.x;
            py = r10 * v.x + r11 * v.y + r12 * v.z + o.y;
            pz = r20 * v.x + r21 * v.y + r22 * v.z + o.z;
        }
        loc64[3 * l] = px;
        loc64[3 * l + 1] = py;
        loc64[3 * l + 2] = pz;
    }
    __syncwarp();
    auto lig32 = [x](int i) { return make_float3(x[3 * i], x[3 * i + 1], x[3 * i + 2]); };
    auto lig64 = [x](int i) {
        return D3{static_cast<double>(x[3 * i]), static_cast<double>(x[3 * i + 1]), static_cast<double>(x[3 * i + 2])};
    };
    auto loc64f = [loc64](int l) { return D3{loc64[3 * l], loc64[3 * l + 1], loc64[3 * l + 2]}; };
    auto loc32 = [loc64](int l) {
        return make_float3(static_cast<float>(loc64[3 * l]), static_cast<float>(loc64[3 * l + 1]),
                           static_cast<float>(loc64[3 * l + 2]));
    };
    F2 ep{0.f, 0.f};
    double e = 0.0;
    ligand_energy(L.topo, x, ep, e, lane);
    if (R.n_local > 0) e += topo_energy64(R.intra, loc32, loc64f, lane);
    if (env.grid.has_grid) {
        for (int a = lane; a < N; a += kWarp)
            grid_energy(env.grid, __ldg(&L.map_slot[a]), F2{__ldg(&L.charge[a]), __ldg(&L.charge_lo[a])}, lig32(a), ep, e);
    }
    // explicit inter pairs, one (ligand atom, receptor atom) pair per lane and step
    const int M = R.n_explicit;
    const int pairs = N * M;
    for (int k = lane; k < pairs; k += kWarp) {
        const int i = k / M, j = k - i * M;
        const int loc = __ldg(&R.ex_local[j]);
        const float4 rj = __ldg(&R.ex_xyzq[j]);
        const float3 xj = loc >= 0 ? loc32(loc) : xyz(rj);
        const float3 xi = lig32(i);
        const float2 sei = __ldg(&L.se[i]), sej = __ldg(&R.ex_se[j]);
        const float3 rij = sub3(xj, xi);
        const float rinv = rsqrtf(dot3(rij, rij));
        const float s = (sei.x + sej.x) * 0.5f;
        const float xx = s * s * rinv * rinv;
        const float u6 = xx * xx * xx;
        const float en = fmaf(sqrtf(sei.y * sej.y) * 4.f, u6 * u6 - u6, kCoulombF * __ldg(&L.charge[i]) * rj.w * rinv);
        if (fabsf(en) <= kPairFp64) {
            e += static_cast<double>(en);
        } else {
            const double4 r64 = R.ex_xyzq64[j];
            const double2 se64i = __ldg(&L.se64[i]), se64j = __ldg(&R.ex_se64[j]);
            const double sm = (se64i.x + se64j.x) * 0.5;
            const double4 p = make_double4(kCoulombD64 * __ldg(&L.charge64[i]) * r64.w,
                                           sqrt(se64i.y * se64j.y) * 4.0, sm * sm, 0.0);
            e += pair_energy64(p, lig64(i), loc >= 0 ? loc64f(loc) : D3{r64.x, r64.y, r64.z});
        }
    }
    // the pairs' warp sum in FP32 (two-sum), the FP64 terms' only where a lane has one
    const double pairs_sum = ds_warp_sum(DS{ep.h, ep.l});
    if (__any_sync(kFull, e != 0.0)) return pairs_sum + warp_sum_d(e) + R.e_const;
    return pairs_sum + R.e_const;
}

}  // namespace pxd
