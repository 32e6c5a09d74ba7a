// Warp-cooperative empirical score of one pose (pose selection / affinity): the device
// restatement of root_scorer::combine with its leaf scorers (scorer.cpp:53-724).
//
// Ligand coordinates come from the warp's shared-memory slice, receptor coordinates from
// the all-atom table with rotor atoms substituted from the slice. Receptor ring centroids
// and normals are precomputed on the host (ring atoms never sit on a rotor). Every term
// is summed per lane in a compensated FP32 pair and reduced over the warp.
#pragma once

#include "device_eval.cuh"

namespace pxd {

// get_reversed_linear_percent (math.h:196-215)
__device__ __forceinline__ float ramp_down(float v, float lo, float hi) {
    if (v < lo) return 1.f;
    if (v <= hi) return 1.f - (v - lo) / (hi - lo);
    return 0.f;
}
__device__ __forceinline__ float ramp_down_c(float v, float c, float lo, float hi) {
    return v < c ? ramp_down(c - v, lo, hi) : ramp_down(v - c, lo, hi);
}
__device__ __forceinline__ float dist3(float3 a, float3 b) {
    const float3 d = sub3(a, b);
    return sqrtf(dot3(d, d));
}

struct ScoreEnv {
    DevRecScore rs;
    const DevSf* sf;
    const float2* vdw;  // [99][rs.n_cls] mean sigma, 4 sqrt(eps eps) under sf (score_vdw_kernel)
};

// Position of a listed receptor atom (DevRecScore): its own, or its rotor's.
__device__ __forceinline__ float3 rec_pos(float4 v, const float4* loc_xyz) {
    const int l = __float_as_int(v.w);
    return l >= 0 ? xyz(loc_xyz[l]) : xyz(v);
}

__device__ __forceinline__ void lig_ring(const float4* X, const int* r, float3& c, float3& n) {
    int sz = 0;
    c = make_float3(0.f, 0.f, 0.f);
    for (int k = 0; k < 6; ++k) {
        const int a = __ldg(&r[k]);
        if (a < 0) break;
        c = add3(c, xyz(X[a]));
        ++sz;
    }
    c = mul3(c, 1.f / sz);
    const float3 p0 = xyz(X[__ldg(&r[0])]), p1 = xyz(X[__ldg(&r[1])]), p2 = xyz(X[__ldg(&r[2])]);
    n = cross3(sub3(p1, p0), sub3(p1, p2));
    n = mul3(n, 1.f / sqrtf(dot3(n, n)));
}

__device__ __forceinline__ float projected(float3 n1, float3 c1, float3 c2) {
    const float3 t = sub3(c2, c1);
    const float dp = dot3(n1, t);
    return sqrtf(dot3(t, t) - dp * dp);
}

// pi_stacking_batch::calculate (scorer.cpp:698-724) for one ring pair
__device__ __forceinline__ float stack_pair(float3 rc, float3 rn, float3 lc, float3 ln,
                                            const float* p, float center) {
    float d = dist3(rc, lc);
    if (d > p[1]) return 0.f;
    d = ramp_down(d, p[0], p[1]);
    const float s1 = projected(rn, rc, lc), s2 = projected(ln, lc, rc);
    float sg = s1 < s2 ? s1 : s2;
    if (sg > p[5]) return 0.f;
    sg = ramp_down(sg, p[4], p[5]);
    float th = acosf(fminf(fmaxf(dot3(rn, ln), -1.f), 1.f)) * (180.f / 3.14159265358979f);
    th = fminf(th, 180.f - th);
    th = ramp_down_c(th, center, p[2], p[3]);
    return -d * sg * th;
}

// hbond_interactions_ga_tuning_param::calculate, one (donor, acceptor) pair
__device__ __forceinline__ float hbond_pair(float3 dpos, float3 hpos, float3 apos, const float* p) {
    const float dd = ramp_down_c(dist3(hpos, apos), p[4], p[0], p[1]);
    if (dd < kEpsF) return 0.f;
    const float3 h2d = sub3(dpos, hpos), h2a = sub3(apos, hpos);
    const float ll = sqrtf(dot3(h2d, h2d)) * sqrtf(dot3(h2a, h2a));
    const float c = fminf(fmaxf(dot3(h2d, h2a) / (ll + kEpsF), -1.f), 1.f);
    const float ang = acosf(c) * (180.f / 3.14159265358979f);
    return -dd * ramp_down_c(ang, p[5], p[2], p[3]);
}

__device__ __forceinline__ float signed_dihedral(float3 pi, float3 pj, float3 pk, float3 pl) {
    const float3 rij = sub3(pj, pi), rkj = sub3(pj, pk), w0 = sub3(pl, pk);
    const float3 m = cross3(rij, rkj), n = cross3(rkj, w0);
    const float3 w = cross3(m, n);
    const float phi = atan2f(sqrtf(dot3(w, w)), dot3(m, n) + kEpsF);
    return dot3(rij, n) < 0.f ? phi : -phi;
}

// The Coulomb and LJ pairs and the hydrophobic contacts of the pose in X (ligand, smem) with
// receptor rotor atoms in loc_xyz (smem) are split into parts, the pairs by receptor atom, the
// contacts by ligand atom; a part's sums are compensated, per lane. The other terms are FP32
// sums of one warp each. The terms read the receptor lists by value, one record per atom:
// through index lists a contact was a chain of four loads, and a pose of 55 atoms in a pocket
// of 1,866 took one warp 460,000 cycles.

// Part `part` of `parts` of the Coulomb and clamped LJ terms over every ligand x receptor pair
// (scorer.cpp:222-276). Each lane takes receptor atoms and walks the ligand atoms (shared
// memory and L1-resident records, read by every lane at once): a receptor atom's records are
// loaded once per call instead of once per ligand atom. Mean sigma and 4 sqrt(eps eps) of a
// (type, class) come from a table; their square root per pair was a quarter of the loop.
static __device__ __forceinline__ void score_pairs(const ScoreEnv& env, const DevLigand& L, const float4* X,
                                                   const float4* loc_xyz, int lane, int part, int parts, DS& coul,
                                                   DS& vdw) {
    const DevRecScore& rs = env.rs;
    const DevSf& sf = *env.sf;
    if (sf.coef[PXD_TERM_COULOMB] == 0.f && sf.coef[PXD_TERM_VDW] == 0.f) return;
    const int N = L.n_atoms;
    const float cutoff = sf.vdw_cutoff;
    const float* const charge = L.charge;
    const int* const type = L.type;
    for (int j = lane + part * kWarp; j < rs.n_all; j += parts * kWarp) {
        const float4 rj = __ldg(&rs.all_xyzq[j]);
        const int2 lc = __ldg(&rs.all_lc[j]);
        const float3 xj = lc.x >= 0 ? xyz(loc_xyz[lc.x]) : xyz(rj);
        const float2* const row = env.vdw + lc.y;
        float ec = 0.f, ev = 0.f;
#pragma unroll 4
        for (int i = 0; i < N; ++i) {
            const float3 xi = xyz(X[i]);
            const float qi = __ldg(&charge[i]);
            const float2 sc = __ldg(&row[__ldg(&type[i]) * rs.n_cls]);
            const float d = dist3(xi, xj);
            const float rinv = 1.f / (d + kEpsF);
            ec = fmaf(qi * rj.w, rinv, ec);
            const float s = sc.x * rinv;
            const float s2 = s * s;
            const float u6 = s2 * s2 * s2;
            const float v = (u6 * u6 - u6) * sc.y;
            ev += fminf(fmaxf(v, -cutoff), cutoff);
        }
        ds_add(coul, ec * kCoulombF);
        ds_add(vdw, ev);
    }
}

// Part `part` of `parts` of the hydrophobic contacts (scorer.cpp:278-311).
static __device__ __forceinline__ void score_hydrophobic(const ScoreEnv& env, const DevLigand& L, const DevLigScore& ls,
                                                         const float4* X, const float4* loc_xyz, int lane, int part,
                                                         int parts, DS& acc) {
    const DevRecScore& rs = env.rs;
    const DevSf& sf = *env.sf;
    if (sf.coef[PXD_TERM_HYDROPHOBIC] == 0.f) return;
    const float hydro_factor = sf.hydro_factor, hydro_min = sf.hydro_min, hydro_max = sf.hydro_max;
    for (int a = part; a < ls.n_hyd; a += parts) {
        const int i = __ldg(&ls.hyd[a]);
        const float3 xi = xyz(X[i]);
        const float s1 = sf.vdw_sigma_raw[__ldg(&L.type[i])];
        float e = 0.f;
#pragma unroll 4
        for (int b = lane; b < rs.n_hyd; b += kWarp) {
            const float r1 = (s1 + __ldg(&rs.hyd_sigma[b])) * hydro_factor + hydro_min;
            e -= ramp_down(dist3(xi, rec_pos(__ldg(&rs.hyd[b]), loc_xyz)), r1, r1 + hydro_max);
        }
        ds_add(acc, e);
    }
}

// The other terms: the ionic, pi-cation and stacking terms (own_ion), hydrogen bonds and torsion
// strain (own_hb), added to acc.
static __device__ __forceinline__ void score_few(const ScoreEnv& env, const DevLigand& L, const DevLigScore& ls,
                                                 const float4* X, const float4* loc_xyz, int lane, bool own_ion,
                                                 bool own_hb, DS* acc) {
    const DevRecScore& rs = env.rs;
    const DevSf& sf = *env.sf;
    // ionic (scorer.cpp:313-368): ligand cations x receptor anions, receptor cations x ligand anions
    if (own_ion && sf.coef[PXD_TERM_IONIC] != 0.f) {
        float e = 0.f;
        for (int a = 0; a < ls.n_cat; ++a) {
            const float3 xi = xyz(X[__ldg(&ls.cat[a])]);
            for (int b = lane; b < rs.n_an; b += kWarp)
                e -= sf.ionic_coef[0] *
                     ramp_down(dist3(xi, rec_pos(__ldg(&rs.an[b]), loc_xyz)), sf.ionic[0][0], sf.ionic[0][1]);
        }
        for (int a = 0; a < ls.n_an; ++a) {
            const float3 xi = xyz(X[__ldg(&ls.an[a])]);
            for (int b = lane; b < rs.n_cat; b += kWarp)
                e -= sf.ionic_coef[1] *
                     ramp_down(dist3(rec_pos(__ldg(&rs.cat[b]), loc_xyz), xi), sf.ionic[1][0], sf.ionic[1][1]);
        }
        ds_add(acc[PXD_TERM_IONIC], e);
    }
    // cation-pi (scorer.cpp:370-462)
    if (own_ion && sf.coef[PXD_TERM_PI_CATION] != 0.f) {
        float e = 0.f;
        for (int a = 0; a < ls.n_cat; ++a) {
            const float3 xi = xyz(X[__ldg(&ls.cat[a])]);
            for (int b = lane; b < rs.n_r5; b += kWarp)
                e -= sf.picat_coef[0] * ramp_down(dist3(xyz(__ldg(&rs.r5c[b])), xi), sf.picat[0][0], sf.picat[0][1]);
            for (int b = lane; b < rs.n_r6; b += kWarp)
                e -= sf.picat_coef[1] * ramp_down(dist3(xyz(__ldg(&rs.r6c[b])), xi), sf.picat[1][0], sf.picat[1][1]);
        }
        for (int r = 0; r < ls.n_r5 + ls.n_r6; ++r) {
            const bool five = r < ls.n_r5;
            float3 c, n;
            lig_ring(X, five ? ls.r5 + 6 * r : ls.r6 + 6 * (r - ls.n_r5), c, n);
            const int k = five ? 2 : 3;
            for (int b = lane; b < rs.n_cat; b += kWarp)
                e -= sf.picat_coef[k] *
                     ramp_down(dist3(c, rec_pos(__ldg(&rs.cat[b]), loc_xyz)), sf.picat[k][0], sf.picat[k][1]);
        }
        ds_add(acc[PXD_TERM_PI_CATION], e);
    }
    // pi stacking, face-to-face (centre 0) and edge-to-face (centre 90) (scorer.cpp:638-724)
    for (int f = 0; f < 2; ++f) {
        if (!own_ion || sf.coef[PXD_TERM_F2F + f] == 0.f) continue;
        const float center = f == 0 ? 0.f : 90.f;
        float e = 0.f;
        for (int r = 0; r < ls.n_r5 + ls.n_r6; ++r) {
            const bool five = r < ls.n_r5;
            float3 lc, ln;
            lig_ring(X, five ? ls.r5 + 6 * r : ls.r6 + 6 * (r - ls.n_r5), lc, ln);
            // l5r5, l5r6, l6r5, l6r6 in the reference's argument order
            const int k5 = five ? 0 : 2, k6 = five ? 1 : 3;
            for (int b = lane; b < rs.n_r5; b += kWarp)
                e += sf.stack_coef[f][k5] * stack_pair(xyz(__ldg(&rs.r5c[b])), xyz(__ldg(&rs.r5n[b])), lc, ln,
                                                       sf.stack[f][k5], center);
            for (int b = lane; b < rs.n_r6; b += kWarp)
                e += sf.stack_coef[f][k6] * stack_pair(xyz(__ldg(&rs.r6c[b])), xyz(__ldg(&rs.r6n[b])), lc, ln,
                                                       sf.stack[f][k6], center);
        }
        ds_add(acc[PXD_TERM_F2F + f], e);
    }
    // hydrogen bonds, 8 donor/acceptor classes (scorer.cpp:464-577)
    if (own_hb && sf.coef[PXD_TERM_HBOND] != 0.f) {
        float e = 0.f;
        for (int c = 0; c < 2; ++c) {  // ligand donors (charged, neutral)
            const int nd = c == 0 ? ls.n_donc : ls.n_donn;
            const int2* dl = c == 0 ? ls.donc : ls.donn;
            for (int a = 0; a < nd; ++a) {
                const int2 dh = __ldg(&dl[a]);
                const float3 dp = xyz(X[dh.x]), hp = xyz(X[dh.y]);
                for (int u = 0; u < 2; ++u) {  // receptor acceptors (charged, neutral)
                    const int na = u == 0 ? rs.n_accc : rs.n_accn;
                    const float4* al = u == 0 ? rs.accc : rs.accn;
                    const int k = 2 * c + u;
                    float s = 0.f;
                    for (int b = lane; b < na; b += kWarp)
                        s += hbond_pair(dp, hp, rec_pos(__ldg(&al[b]), loc_xyz), sf.hbond[k]);
                    e += sf.hbond_coef[k] * s;
                }
            }
        }
        for (int u = 0; u < 2; ++u) {  // ligand acceptors (charged, neutral)
            const int na = u == 0 ? ls.n_accc : ls.n_accn;
            const int* al = u == 0 ? ls.accc : ls.accn;
            for (int a = 0; a < na; ++a) {
                const float3 ap = xyz(X[__ldg(&al[a])]);
                for (int c = 0; c < 2; ++c) {  // receptor donors (charged, neutral)
                    const int nd = c == 0 ? rs.n_donc : rs.n_donn;
                    const float4* const* dl = c == 0 ? rs.donc : rs.donn;
                    const int k = 4 + 2 * c + u;
                    float s = 0.f;
                    for (int b = lane; b < nd; b += kWarp)
                        s += hbond_pair(rec_pos(__ldg(&dl[0][b]), loc_xyz), rec_pos(__ldg(&dl[1][b]), loc_xyz), ap,
                                        sf.hbond[k]);
                    e += sf.hbond_coef[k] * s;
                }
            }
        }
        ds_add(acc[PXD_TERM_HBOND], e * sf.hbond_scale);
    }
    // torsion strain (scorer.cpp:579-613)
    if (own_hb && sf.coef[PXD_TERM_TSTRAIN] != 0.f) {
        for (int t = lane; t < ls.n_ts; t += kWarp) {
            const float4 co = __ldg(&ls.ts_coef[t]);
            const int2 rg = __ldg(&ls.ts_range[t]);
            float tmp = 0.f;
            int j = 0;
            for (; j < rg.y; ++j) {
                const int4 q = __ldg(&ls.ts_quad[rg.x + j]);
                if (q.x == q.y) break;
                const float th = signed_dihedral(xyz(X[q.x]), xyz(X[q.y]), xyz(X[q.z]), xyz(X[q.w]));
                tmp += (1.f + cosf(th)) * co.x + (1.f + cosf(2.f * th - 3.14159265358979f)) * co.y +
                       (1.f + cosf(3.f * th)) * co.z + (1.f + cosf(4.f * th - 3.14159265358979f)) * co.w;
            }
            if (j > 0) ds_add(acc[PXD_TERM_TSTRAIN], tmp / j);
        }
    }
}

// Completes the term values (scales, the constant rotatable term, GB/SA 0) and returns
// sum(coef * term) over the active terms except GB/SA.
static __device__ __forceinline__ double score_total(const DevSf& sf, const DevLigScore& ls, double* vals) {
    vals[PXD_TERM_VDW] *= sf.vdw_scale;
    vals[PXD_TERM_HYDROPHOBIC] *= sf.hydro_scale;
    vals[PXD_TERM_ROTATABLE] = sf.coef[PXD_TERM_ROTATABLE] != 0.f ? -1.0 / (2.620643 + ls.n_rot) : 0.0;
    vals[PXD_TERM_GBSA] = 0.0;
    double total = 0.0;
#pragma unroll
    for (int k = 0; k < PXD_NUM_TERMS; ++k) total += static_cast<double>(sf.coef[k]) * vals[k];
    return total;
}

// Score of the pose in X, by a team of warps of one block (or one warp, tn = 1): the
// members' partials are summed in member order, so every member returns the same score.
static __device__ __noinline__ double score_pose(const ScoreEnv& env, const DevLigand& L, const float4* X,
                                                 const float4* loc_xyz, int lane, int tw, int tn, TeamShared* ts) {
    DS acc[PXD_NUM_TERMS - 1];
#pragma unroll
    for (int k = 0; k < PXD_NUM_TERMS - 1; ++k) acc[k] = DS{0.f, 0.f};
    score_pairs(env, L, X, loc_xyz, lane, tw, tn, acc[PXD_TERM_COULOMB], acc[PXD_TERM_VDW]);
    const int hyd_warps = tn > 2 ? tn - 2 : tn;
    if (tw < hyd_warps)
        score_hydrophobic(env, L, L.score, X, loc_xyz, lane, tw, hyd_warps, acc[PXD_TERM_HYDROPHOBIC]);
    score_few(env, L, L.score, X, loc_xyz, lane, tw == max(tn - 2, 0), tw == tn - 1, acc);
    double vals[PXD_NUM_TERMS];
    if (tn > 1) {
#pragma unroll
        for (int k = 0; k < PXD_NUM_TERMS - 1; ++k) {
            const DS r = ds_warp_reduce(acc[k]);
            if (lane == 0) ts->terms[tw][k] = make_float2(r.hi, r.lo);
        }
        const bool ok = team_sync(ts, tn, lane);
#pragma unroll
        for (int k = 0; k < PXD_NUM_TERMS - 1; ++k) {
            DS t{ts->terms[0][k].x, ts->terms[0][k].y};
            for (int u = 1; u < tn; ++u) ds_add_ds(t, DS{ts->terms[u][k].x, ts->terms[u][k].y});
            vals[k] = static_cast<double>(t.hi) + static_cast<double>(t.lo);
        }
        // read by every member before any member writes its next partials; an aborted
        // team scores NaN
        if (!team_sync(ts, tn, lane) || !ok) return __longlong_as_double(0x7ff8000000000000LL);
    } else {
#pragma unroll
        for (int k = 0; k < PXD_NUM_TERMS - 1; ++k) vals[k] = ds_warp_sum(acc[k]);
    }
    return score_total(*env.sf, L.score, vals);
}

}  // namespace pxd
