// Empirical scores on the GPU: the pose-selection / affinity score kernel (a block per pose)
// and the FP64 generalised-Born / surface-area term, with their C ABI.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "../../include/pxdock_gb300_vdw.h"
#include "device_score.cuh"
#include "gb_exp.cuh"

namespace pxd {

// ------------------------------------------------------------------ uploads
struct Pack {
    std::vector<unsigned char> bytes;
    template <class T>
    size_t put(const std::vector<T>& v) {
        size_t off = (bytes.size() + 15) / 16 * 16;
        bytes.resize(off + v.size() * sizeof(T) + 16);
        if (!v.empty()) std::memcpy(bytes.data() + off, v.data(), v.size() * sizeof(T));
        return off;
    }
};

template <class T>
static const T* at(void* base, size_t off) {
    return reinterpret_cast<const T*>(static_cast<const unsigned char*>(base) + off);
}

static std::vector<int> ints(const int32_t* p, int n) {
    return n > 0 ? std::vector<int>(p, p + n) : std::vector<int>();
}

static std::vector<int2> pairs2(const int32_t* p, int n) {
    std::vector<int2> v;
    for (int i = 0; i < n; ++i) v.push_back(make_int2(p[2 * i], p[2 * i + 1]));
    return v;
}

// fill_atom_properties (scorer.cpp:737-753): GB radius by element, 1.3 for H bonded to N.
void gbsa_properties(const pxd_score_lists* l, int n, std::vector<double>& radius,
                     std::vector<double>& screen) {
    static const double kR[18] = {1.5, 1.2, 1.5, 1.5, 1.5, 1.5, 1.7, 1.55, 1.5,
                                  1.5, 1.5, 1.5, 1.5, 1.5, 2.1, 1.85, 1.8, 1.7};
    static const double kS[17] = {0.8, 0.85, 0.8, 0.8, 0.8, 0.8, 0.72, 0.79, 0.85,
                                  0.88, 0.8, 0.8, 0.8, 0.8, 0.8, 0.86, 0.96};
    radius.assign(n, -1.0);
    screen.assign(n, kS[0]);
    if (!l || !l->atomic_numbers) return;
    for (int b = 0; b < l->n_all_bonds; ++b) {
        const int i = l->all_bonds[2 * b], j = l->all_bonds[2 * b + 1];
        if (i < 0 || j < 0 || i >= n || j >= n) continue;
        const int ea = l->atomic_numbers[i], eb = l->atomic_numbers[j];
        if (ea == 1 && eb == 7) radius[i] = 1.3;
        else if (ea == 7 && eb == 1) radius[j] = 1.3;
    }
    for (int i = 0; i < n; ++i) {
        const int e = l->atomic_numbers[i];
        if (radius[i] < 0.0) radius[i] = (e >= 0 && e <= 17) ? kR[e] : kR[0];
        screen[i] = (e >= 0 && e <= 16) ? kS[e] : kS[0];
    }
}

// Pair-table class of an atom: ligand C N O S P F Cl other-heavy (0-7), receptor
// C N O other-heavy (0-3); hydrogens (and unknown elements, Z < 2) take none (-1).
int pair_class(int is_receptor, int z) {
    if (z < 2) return -1;
    switch (z) {
        case 6: return 0;
        case 7: return 1;
        case 8: return 2;
        default: break;
    }
    if (is_receptor) return 3;
    switch (z) {
        case 16: return 3;
        case 15: return 4;
        case 9: return 5;
        case 17: return 6;
        default: return 7;
    }
}

static float __int_as_float_host(int v) {
    float f;
    std::memcpy(&f, &v, sizeof(f));
    return f;
}

static std::vector<int> pair_classes(const pxd_score_lists* l, int n, int is_receptor) {
    std::vector<int> c;
    if (!l || !l->atomic_numbers) return c;
    c.resize(n);
    for (int i = 0; i < n; ++i) {
        const int k = pair_class(is_receptor, l->atomic_numbers[i]);
        c[i] = k < 0 ? -1 : (is_receptor ? k : 4 * k);
    }
    return c;
}

static bool ids_ok(const int32_t* p, int n, int limit) {
    for (int i = 0; i < n; ++i)
        if (p[i] < 0 || p[i] >= limit) return false;
    return true;
}

static bool lists_ok(const pxd_score_lists* l, int n_atoms) {
    if (!ids_ok(l->hydrophobic, l->n_hydrophobic, n_atoms) || !ids_ok(l->cation, l->n_cation, n_atoms) ||
        !ids_ok(l->anion, l->n_anion, n_atoms) || !ids_ok(l->don_charged, 2 * l->n_don_charged, n_atoms) ||
        !ids_ok(l->don_neutral, 2 * l->n_don_neutral, n_atoms) ||
        !ids_ok(l->acc_charged, l->n_acc_charged, n_atoms) || !ids_ok(l->acc_neutral, l->n_acc_neutral, n_atoms))
        return false;
    for (int k = 0; k < 2; ++k) {
        const int n = k ? l->n_ring6 : l->n_ring5;
        const int32_t* r = k ? l->ring6 : l->ring5;
        for (int i = 0; i < n; ++i) {
            int sz = 0;
            while (sz < 6 && r[6 * i + sz] >= 0) {
                if (r[6 * i + sz] >= n_atoms) return false;
                ++sz;
            }
            if (sz < 3) return false;
        }
    }
    for (int e = 0; e < l->n_tstrain; ++e) {
        if (l->tstrain_offsets[e] > l->tstrain_offsets[e + 1]) return false;
        for (int q = l->tstrain_offsets[e]; q < l->tstrain_offsets[e + 1]; ++q)
            if (!ids_ok(l->tstrain_quads + 4 * q, 4, n_atoms)) return false;
    }
    return true;
}

int upload_receptor_scoring(pxd_context* ctx, const pxd_score_lists* l, const std::vector<int>& local_of) {
    DevRecScore& d = ctx->rec_score;
    d = DevRecScore{};
    if (ctx->rec_score_mem) cudaFree(ctx->rec_score_mem);
    ctx->rec_score_mem = nullptr;
    const int M = ctx->n_rec;
    d.n_all = M;
    d.all_xyzq = at<float4>(ctx->rec_ex_all, ctx->ex_all_off[0]);
    d.all_se = at<float2>(ctx->rec_ex_all, ctx->ex_all_off[1]);
    gbsa_properties(l, M, ctx->rec_gb_radius, ctx->rec_gb_screen);
    if (l && !lists_ok(l, M)) return set_error(ctx, PXD_ERR_INVALID, "receptor interaction list atom out of range");
    // per-atom record of the differentiable score's pair loop: sigma, sqrt(epsilon),
    // pair-table class, rotor-atom local index (-1: fixed)
    const std::vector<int> pcls = pair_classes(l, M, 1);
    std::vector<float4> pairrec(M);
    for (int a = 0; a < M; ++a)
        pairrec[a] = make_float4(static_cast<float>(ctx->rec_sigma[a]),
                                 static_cast<float>(std::sqrt(ctx->rec_epsilon[a])),
                                 __int_as_float_host(pcls.empty() ? -1 : pcls[a]),
                                 __int_as_float_host(ctx->is_mov[a] ? local_of[a] : -1));
    std::vector<float2> cls;
    std::vector<int2> lc(M);
    {
        std::map<std::pair<int64_t, int64_t>, int> seen;
        for (int a = 0; a < M; ++a) {
            const float2 se = make_float2(static_cast<float>(ctx->rec_sigma[a]), static_cast<float>(ctx->rec_epsilon[a]));
            const auto it =
                seen.emplace(std::make_pair(number_bits(se.x), number_bits(se.y)), static_cast<int>(cls.size())).first;
            if (it->second == static_cast<int>(cls.size())) cls.push_back(se);
            lc[a] = make_int2(ctx->is_mov[a] ? local_of[a] : -1, it->second);
        }
    }
    Pack pk;
    const size_t o_pair = pk.put(pairrec), o_lc = pk.put(lc), o_cls = pk.put(cls);
    d.n_cls = static_cast<int>(cls.size());
    if (!l) {
        int rc0 = cuda_check(ctx, cudaMalloc(&ctx->rec_score_mem, pk.bytes.size()), "receptor score lists");
        if (rc0) return rc0;
        rc0 = upload(ctx, ctx->rec_score_mem, pk.bytes.data(), pk.bytes.size(), "receptor score lists copy");
        if (rc0) return rc0;
        d.pair_rec = at<float4>(ctx->rec_score_mem, o_pair);
        d.all_lc = at<int2>(ctx->rec_score_mem, o_lc);
        d.cls_se = at<float2>(ctx->rec_score_mem, o_cls);
        return PXD_OK;
    }
    // ring centroids and normals (to_ring_centroid / to_ring_normal, scorer.cpp:128-172)
    std::vector<float4> rc[2], rn[2];
    for (int k = 0; k < 2; ++k) {
        const int n = k ? l->n_ring6 : l->n_ring5;
        const int32_t* r = k ? l->ring6 : l->ring5;
        for (int i = 0; i < n; ++i) {
            double c[3] = {0, 0, 0};
            int sz = 0;
            while (sz < 6 && r[6 * i + sz] >= 0) {
                const int a = r[6 * i + sz];
                if (ctx->is_mov[a]) return set_error(ctx, PXD_ERR_INVALID, "receptor ring atom on a rotor");
                for (int u = 0; u < 3; ++u) c[u] += ctx->rec_xyz[3 * a + u];
                ++sz;
            }
            for (int u = 0; u < 3; ++u) c[u] /= sz;
            const double* p0 = &ctx->rec_xyz[3 * r[6 * i]];
            const double* p1 = &ctx->rec_xyz[3 * r[6 * i + 1]];
            const double* p2 = &ctx->rec_xyz[3 * r[6 * i + 2]];
            const double e1[3] = {p1[0] - p0[0], p1[1] - p0[1], p1[2] - p0[2]};
            const double e2[3] = {p1[0] - p2[0], p1[1] - p2[1], p1[2] - p2[2]};
            double nn[3] = {e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2],
                            e1[0] * e2[1] - e1[1] * e2[0]};
            const double len = std::sqrt(nn[0] * nn[0] + nn[1] * nn[1] + nn[2] * nn[2]);
            rc[k].push_back(make_float4(static_cast<float>(c[0]), static_cast<float>(c[1]),
                                        static_cast<float>(c[2]), 0.f));
            rn[k].push_back(make_float4(static_cast<float>(nn[0] / len), static_cast<float>(nn[1] / len),
                                        static_cast<float>(nn[2] / len), 0.f));
        }
    }
    // a list's atoms (every `step`-th index from `ids`) by value
    auto atoms = [&](const int32_t* ids, int n, int step = 1) {
        std::vector<float4> v;
        for (int i = 0; i < n; ++i) {
            const int a = ids[step * i];
            v.push_back(make_float4(static_cast<float>(ctx->rec_xyz[3 * a]), static_cast<float>(ctx->rec_xyz[3 * a + 1]),
                                    static_cast<float>(ctx->rec_xyz[3 * a + 2]), __int_as_float_host(lc[a].x)));
        }
        return v;
    };
    std::vector<float> hyd_sigma;
    for (int i = 0; i < l->n_hydrophobic; ++i) hyd_sigma.push_back(static_cast<float>(ctx->rec_sigma[l->hydrophobic[i]]));
    const size_t o_hyd = pk.put(atoms(l->hydrophobic, l->n_hydrophobic)), o_hyds = pk.put(hyd_sigma);
    const size_t o_cat = pk.put(atoms(l->cation, l->n_cation));
    const size_t o_an = pk.put(atoms(l->anion, l->n_anion));
    const size_t o_r5c = pk.put(rc[0]), o_r5n = pk.put(rn[0]), o_r6c = pk.put(rc[1]), o_r6n = pk.put(rn[1]);
    const size_t o_donc = pk.put(atoms(l->don_charged, l->n_don_charged, 2));
    const size_t o_donch = pk.put(atoms(l->don_charged + 1, l->n_don_charged, 2));
    const size_t o_donn = pk.put(atoms(l->don_neutral, l->n_don_neutral, 2));
    const size_t o_donnh = pk.put(atoms(l->don_neutral + 1, l->n_don_neutral, 2));
    const size_t o_accc = pk.put(atoms(l->acc_charged, l->n_acc_charged));
    const size_t o_accn = pk.put(atoms(l->acc_neutral, l->n_acc_neutral));
    const size_t o_pcl = pk.put(pcls);
    int rc_ = cuda_check(ctx, cudaMalloc(&ctx->rec_score_mem, pk.bytes.size()), "receptor score lists");
    if (rc_) return rc_;
    rc_ = upload(ctx, ctx->rec_score_mem, pk.bytes.data(), pk.bytes.size(), "receptor score lists copy");
    if (rc_) return rc_;
    void* b = ctx->rec_score_mem;
    d.has = 1;
    d.n_hyd = l->n_hydrophobic;
    d.n_cat = l->n_cation;
    d.n_an = l->n_anion;
    d.n_r5 = l->n_ring5;
    d.n_r6 = l->n_ring6;
    d.n_donc = l->n_don_charged;
    d.n_donn = l->n_don_neutral;
    d.n_accc = l->n_acc_charged;
    d.n_accn = l->n_acc_neutral;
    d.all_lc = at<int2>(b, o_lc);
    d.cls_se = at<float2>(b, o_cls);
    d.hyd = at<float4>(b, o_hyd);
    d.hyd_sigma = at<float>(b, o_hyds);
    d.cat = at<float4>(b, o_cat);
    d.an = at<float4>(b, o_an);
    d.r5c = at<float4>(b, o_r5c);
    d.r5n = at<float4>(b, o_r5n);
    d.r6c = at<float4>(b, o_r6c);
    d.r6n = at<float4>(b, o_r6n);
    d.donc[0] = at<float4>(b, o_donc);
    d.donc[1] = at<float4>(b, o_donch);
    d.donn[0] = at<float4>(b, o_donn);
    d.donn[1] = at<float4>(b, o_donnh);
    d.accc = at<float4>(b, o_accc);
    d.accn = at<float4>(b, o_accn);
    d.pclass = pcls.empty() ? nullptr : at<int>(b, o_pcl);
    d.pair_rec = at<float4>(b, o_pair);
    return PXD_OK;
}

// Appends the ligand's lists to its device allocation image is not possible after the
// fact, so the lists get their own allocation owned by the ligand entry.
int upload_ligand_scoring(pxd_context* ctx, LigandEntry& e, const pxd_score_lists* l) {
    DevLigScore& d = e.dev.score;
    d = DevLigScore{};
    gbsa_properties(l, e.n_atoms, e.gb_radius, e.gb_screen);
    if (!l) return PXD_OK;
    if (!lists_ok(l, e.n_atoms)) return set_error(ctx, PXD_ERR_INVALID, "ligand interaction list atom out of range");
    std::vector<int> r5(6 * static_cast<size_t>(l->n_ring5)), r6(6 * static_cast<size_t>(l->n_ring6));
    for (size_t i = 0; i < r5.size(); ++i) r5[i] = l->ring5[i];
    for (size_t i = 0; i < r6.size(); ++i) r6[i] = l->ring6[i];
    std::vector<float4> tsc;
    std::vector<int2> tsr;
    std::vector<int4> tsq;
    for (int t = 0; t < l->n_tstrain; ++t) {
        const double* c = l->tstrain_coefs + 4 * t;
        tsc.push_back(make_float4(static_cast<float>(c[0]), static_cast<float>(c[1]), static_cast<float>(c[2]),
                                  static_cast<float>(c[3])));
        tsr.push_back(make_int2(l->tstrain_offsets[t], l->tstrain_offsets[t + 1] - l->tstrain_offsets[t]));
    }
    const int nq = l->n_tstrain ? l->tstrain_offsets[l->n_tstrain] : 0;
    for (int q = 0; q < nq; ++q)
        tsq.push_back(make_int4(l->tstrain_quads[4 * q], l->tstrain_quads[4 * q + 1], l->tstrain_quads[4 * q + 2],
                                l->tstrain_quads[4 * q + 3]));
    Pack pk;
    const size_t o_hyd = pk.put(ints(l->hydrophobic, l->n_hydrophobic));
    const size_t o_cat = pk.put(ints(l->cation, l->n_cation));
    const size_t o_an = pk.put(ints(l->anion, l->n_anion));
    const size_t o_r5 = pk.put(r5), o_r6 = pk.put(r6);
    const size_t o_donc = pk.put(pairs2(l->don_charged, l->n_don_charged));
    const size_t o_donn = pk.put(pairs2(l->don_neutral, l->n_don_neutral));
    const size_t o_accc = pk.put(ints(l->acc_charged, l->n_acc_charged));
    const size_t o_accn = pk.put(ints(l->acc_neutral, l->n_acc_neutral));
    const size_t o_tsc = pk.put(tsc), o_tsr = pk.put(tsr), o_tsq = pk.put(tsq);
    const std::vector<int> pcls = pair_classes(l, e.n_atoms, 0);
    const size_t o_pcl = pk.put(pcls);
    void* b = nullptr;
    int rc = cuda_check(ctx, cudaMalloc(&b, pk.bytes.size()), "ligand score lists");
    if (rc) return rc;
    rc = upload(ctx, b, pk.bytes.data(), pk.bytes.size(), "ligand score lists copy");
    if (rc) {
        cudaFree(b);
        return rc;
    }
    e.score_mem = b;
    d.has = 1;
    d.n_hyd = l->n_hydrophobic;
    d.n_cat = l->n_cation;
    d.n_an = l->n_anion;
    d.n_r5 = l->n_ring5;
    d.n_r6 = l->n_ring6;
    d.n_donc = l->n_don_charged;
    d.n_donn = l->n_don_neutral;
    d.n_accc = l->n_acc_charged;
    d.n_accn = l->n_acc_neutral;
    d.n_ts = l->n_tstrain;
    d.n_rot = l->n_rotatable;
    d.hyd = at<int>(b, o_hyd);
    d.cat = at<int>(b, o_cat);
    d.an = at<int>(b, o_an);
    d.r5 = at<int>(b, o_r5);
    d.r6 = at<int>(b, o_r6);
    d.donc = at<int2>(b, o_donc);
    d.donn = at<int2>(b, o_donn);
    d.accc = at<int>(b, o_accc);
    d.accn = at<int>(b, o_accn);
    d.ts_coef = at<float4>(b, o_tsc);
    d.ts_range = at<int2>(b, o_tsr);
    d.ts_quad = at<int4>(b, o_tsq);
    d.pclass = pcls.empty() ? nullptr : at<int>(b, o_pcl);
    return PXD_OK;
}

// ------------------------------------------------------------------ kernels
// Mean sigma and 4 sqrt(eps eps) of every (ligand type, receptor class) under a scoring
// function, which the pair loop of score_terms would otherwise form per pair.
__global__ void score_vdw_kernel(const DevSf* sf, const float2* cls, int n_cls, float2* out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= PXD_NUM_VDW_TYPES * n_cls) return;
    const float2 ti = sf->vdw_type[k / n_cls], se = cls[k % n_cls];
    out[k] = make_float2((ti.x + se.x) * 0.5f, sqrtf(ti.y * se.y) * 4.f);
}

static int alloc_score_table(pxd_context* ctx, float2** out) {
    const size_t n = static_cast<size_t>(PXD_NUM_VDW_TYPES) * ctx->rec_score.n_cls;
    return cuda_check(ctx, cudaMalloc(out, sizeof(float2) * std::max<size_t>(n, 1)), "score tables");
}

static int fill_score_table(pxd_context* ctx, int w, float2* out) {
    const int n = PXD_NUM_VDW_TYPES * ctx->rec_score.n_cls;
    if (n > 0)
        score_vdw_kernel<<<(n + 127) / 128, 128, 0, ctx->stream>>>(ctx->d_sf[w], ctx->rec_score.cls_se,
                                                                   ctx->rec_score.n_cls, out);
    const int rc = cuda_check(ctx, cudaGetLastError(), "score_vdw_kernel launch");
    return rc ? rc : cuda_check(ctx, cudaStreamSynchronize(ctx->stream), "score tables");
}

// The tables of the installed scoring functions for a receptor that is being installed (they are
// freed with it). A context that has a receptor and a scoring function has their table: the
// callers set either only once it stands.
int build_score_tables(pxd_context* ctx) {
    for (int w = 0; w < 2; ++w) {
        if (!ctx->sf_set[w]) continue;
        int rc = alloc_score_table(ctx, &ctx->d_vdw[w]);
        if (!rc) rc = fill_score_table(ctx, w, ctx->d_vdw[w]);
        if (rc) return rc;
    }
    return PXD_OK;
}

constexpr int kMaxScoreWarps = 16;

struct EsArgs {
    ScoreEnv env;
    DevReceptor rec;
    const DevLigand* ligands;
    int n_ligands;
    const int* lig_ids;
    const float* xyz;
    const float* tors;
    int max_atoms;
    int n_poses;
    double* score;
    double* terms;
};

// One block per pose, its warps sharing the terms. The parts that a term is split into, and the
// order that they are added in, are the same for any number of warps (4 to 16), so a pose's
// score does not depend on its batch, bit for bit.
constexpr int kHydParts = kMaxScoreWarps - 2;

__global__ void __launch_bounds__(kMaxScoreWarps * kWarp) empirical_score_kernel(const __grid_constant__ EsArgs a) {
    extern __shared__ __align__(16) float smem[];
    __shared__ float2 s_part[3][kMaxScoreWarps][kWarp];  // Coulomb, LJ, hydrophobic
    __shared__ float2 s_term[PXD_NUM_TERMS - 1];
    const int lane = threadIdx.x & (kWarp - 1);
    const int w = threadIdx.x / kWarp, nw = blockDim.x / kWarp;
    float4* X = reinterpret_cast<float4*>(smem);
    float4* loc = X + a.max_atoms;
    const int R = a.rec.n_rotors;
    for (int pose = blockIdx.x; pose < a.n_poses; pose += gridDim.x) {
        const int lid = a.lig_ids[pose];
        if (lid < 0 || lid >= a.n_ligands || !a.ligands[lid].score.has ||
            a.ligands[lid].n_atoms > a.max_atoms) {
            if (threadIdx.x == 0) a.score[pose] = nan("");
            continue;
        }
        const DevLigand& L = a.ligands[lid];
        const float* px = a.xyz + static_cast<size_t>(pose) * a.max_atoms * 3;
        for (int i = threadIdx.x; i < L.n_atoms; i += blockDim.x)
            X[i] = make_float4(px[3 * i], px[3 * i + 1], px[3 * i + 2], 0.f);
        // rotor atom positions (torsional_receptor::apply_parameters)
        for (int l = threadIdx.x; l < a.rec.n_mov; l += blockDim.x) {
            const float4 v = __ldg(&a.rec.local_xyz0[l]);
            const int r = __float_as_int(v.w);
            Mat3 Rm, Jm;
            rotation_and_jacobian(xyz(__ldg(&a.rec.rotor_axis[r])), a.tors[static_cast<size_t>(pose) * R + r], Rm, Jm);
            const float3 p = add3(mat_apply(Rm, xyz(v)), xyz(__ldg(&a.rec.rotor_origin[r])));
            loc[l] = make_float4(p.x, p.y, p.z, 0.f);
        }
        __syncthreads();
        for (int v = w; v < kMaxScoreWarps; v += nw) {
            DS c{0.f, 0.f}, e{0.f, 0.f};
            score_pairs(a.env, L, X, loc, lane, v, kMaxScoreWarps, c, e);
            s_part[0][v][lane] = make_float2(c.hi, c.lo);
            s_part[1][v][lane] = make_float2(e.hi, e.lo);
        }
        if (w < nw - 2) {
            for (int v = w; v < kHydParts; v += nw - 2) {
                DS h{0.f, 0.f};
                score_hydrophobic(a.env, L, L.score, X, loc, lane, v, kHydParts, h);
                s_part[2][v][lane] = make_float2(h.hi, h.lo);
            }
        } else {
            DS acc[PXD_NUM_TERMS - 1];
#pragma unroll
            for (int k = 0; k < PXD_NUM_TERMS - 1; ++k) acc[k] = DS{0.f, 0.f};
            const bool ion = w == nw - 2;
            score_few(a.env, L, L.score, X, loc, lane, ion, !ion, acc);
#pragma unroll
            for (int k = 0; k < PXD_NUM_TERMS - 1; ++k) {
                if (k == PXD_TERM_COULOMB || k == PXD_TERM_VDW || k == PXD_TERM_HYDROPHOBIC) continue;
                if ((k == PXD_TERM_HBOND || k == PXD_TERM_TSTRAIN || k == PXD_TERM_ROTATABLE) == ion) continue;
                const DS r = ds_warp_reduce(acc[k]);
                if (lane == 0) s_term[k] = make_float2(r.hi, r.lo);
            }
        }
        __syncthreads();
        if (w < 3) {
            DS t{s_part[w][0][lane].x, s_part[w][0][lane].y};
            const int n = w < 2 ? kMaxScoreWarps : kHydParts;
            for (int v = 1; v < n; ++v) ds_add_ds(t, DS{s_part[w][v][lane].x, s_part[w][v][lane].y});
            t = ds_warp_reduce(t);
            const int k = w == 0 ? PXD_TERM_COULOMB : w == 1 ? PXD_TERM_VDW : PXD_TERM_HYDROPHOBIC;
            if (lane == 0) s_term[k] = make_float2(t.hi, t.lo);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double vals[PXD_NUM_TERMS];
#pragma unroll
            for (int k = 0; k < PXD_NUM_TERMS - 1; ++k)
                vals[k] = static_cast<double>(s_term[k].x) + static_cast<double>(s_term[k].y);
            a.score[pose] = score_total(*a.env.sf, L.score, vals);
            if (a.terms)
                for (int k = 0; k < PXD_NUM_TERMS; ++k) a.terms[static_cast<size_t>(pose) * PXD_NUM_TERMS + k] = vals[k];
        }
        // s_term, s_part and X are rewritten only after the next pose's first barrier has seen thread 0
        __syncthreads();
    }
}

// GB/SA (gbsa_total_energy::calculate, scorer.cpp:798-866) in FP64, for a batch of poses of
// one ligand: the complex, the ligand alone and the receptor alone. What bounds it is the
// FP64 pipe (about 1.7 operations a clock and SM), so the work is what is cut:
//   - the receptor-receptor Born sums are formed once per receptor conformation (once per
//     call without rotors) and serve the receptor alone and every complex;
//   - the pair energies run over i < j (the sum over ordered pairs is symmetric);
//   - r, 1/r and f, 1/f come from one rsqrt each.
// Every sum has a fixed order, so the energies repeat bit for bit. The work is split over
// warps (Born sums) and 64 x 64 tiles of atom pairs (energies), which fills the chip at one
// pose: 8 poses of 42 atoms in a pocket of 1,866 take 2.4 ms of kernel time; with one thread
// per atom and three systems per pose they took 186 ms.
constexpr double kGbOffset = 0.09;
constexpr int kGbTile = 64;
constexpr int kGbThreads = 128;
constexpr int kGbLanes = 8;       // lanes that share a receptor atom's sum over the ligand
constexpr int kGbPoses = 512;     // poses per batch of launches
constexpr size_t kGbBytes = size_t(64) << 20;  // workspace of a batch, or one pose's if that is more

struct GbArgs {
    int n_lig, n_rec, n_poses, n_conf;  // n_conf: receptor conformations, 1 or n_poses
    const double4* rec;      // [n_conf][n_rec] position, charge
    const double4* lig;      // [n_poses][n_lig]
    const double4* rec_p;    // [n_rec] radius, rho = radius - offset, rho * screen
    const double4* lig_p;    // [n_lig]
    double* sum_rr;          // [n_conf][n_rec] receptor-receptor Born sums
    double* ib_rec;          // [n_conf][n_rec] inverse Born radii, receptor alone
    double* ib_lig;          // [n_poses][n_lig] ligand alone
    double* ib_com;          // [n_poses][n_lig + n_rec] complex
    double* partial;         // [systems][n_tiles]
    int n_tiles;             // of the complex
    double* energy;          // [systems]: n_poses complexes, n_conf receptors, n_poses ligands
    GbExpTable exp2;
};

// One pair term of atom j's Born sum (scorer.cpp:806-821).
__device__ __forceinline__ double gb_born_term(double4 xi, double sr, double4 xj, double rho) {
    const double dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
    const double r2 = dx * dx + dy * dy + dz * dz;
    const double ri = rsqrt(r2);
    const double r = r2 > 0.0 ? r2 * ri : 0.0;
    const double U = r + sr;
    if (U < rho) return 0.0;
    const double L = fmax(rho, fabs(r - sr));
    // one division: 1/L - 1/U and 1/L + 1/U as (U -+ L) / (U L), which also keeps the digits that
    // the difference of two reciprocals loses
    const double i = 1.0 / (U * L), d = (U - L) * i;
    const double D = -0.25 * (r - sr * sr * ri) * (d * ((U + L) * i));
    return 0.5 * (D + (d + 0.5 * log(L * L * i + 1e-20) * ri));
}

__device__ __forceinline__ double gb_inverse_born(double sum, double4 p) {
    const double psi = sum * p.y;
    const double t = tanh(psi - 0.8 * psi * psi + 4.85 * psi * psi * psi);
    return 1.0 / p.y - t / p.x;
}

template <int kLanes>
__device__ __forceinline__ double gb_lane_sum(double v) {
#pragma unroll
    for (int off = kLanes / 2; off > 0; off >>= 1) v += __shfl_xor_sync(kFull, v, off);
    return v;
}

// Receptor alone: one warp per atom, the lanes over the other atoms.
__global__ void __launch_bounds__(kGbThreads) gb_receptor_kernel(const __grid_constant__ GbArgs a) {
    const int lane = threadIdx.x & (kWarp - 1);
    const int j = blockIdx.x * (kGbThreads / kWarp) + threadIdx.x / kWarp;
    if (j >= a.n_rec) return;
    const double4* x = a.rec + static_cast<size_t>(blockIdx.y) * a.n_rec;
    const double4 xj = x[j], pj = a.rec_p[j];
    double sum = 0.0;
    for (int i = lane; i < a.n_rec; i += kWarp)
        if (i != j) sum += gb_born_term(x[i], a.rec_p[i].z, xj, pj.y);
    sum = gb_lane_sum<kWarp>(sum);
    if (lane == 0) {
        const size_t o = static_cast<size_t>(blockIdx.y) * a.n_rec + j;
        a.sum_rr[o] = sum;
        a.ib_rec[o] = gb_inverse_born(sum, pj);
    }
}

// Complex and ligand alone: a warp per ligand atom (lanes over the receptor, then the
// ligand), then kGbLanes lanes per receptor atom (over the ligand, added to its receptor sum).
__global__ void __launch_bounds__(kGbThreads) gb_complex_kernel(const __grid_constant__ GbArgs a) {
    const int lane = threadIdx.x & (kWarp - 1);
    const int task = blockIdx.x * (kGbThreads / kWarp) + threadIdx.x / kWarp;
    const int p = blockIdx.y, c = a.n_conf > 1 ? p : 0;
    const double4* xl = a.lig + static_cast<size_t>(p) * a.n_lig;
    const double4* xr = a.rec + static_cast<size_t>(c) * a.n_rec;
    double* ib = a.ib_com + static_cast<size_t>(p) * (a.n_lig + a.n_rec);
    if (task < a.n_lig) {
        const double4 xj = xl[task], pj = a.lig_p[task];
        double own = 0.0, rec = 0.0;
        for (int i = lane; i < a.n_lig; i += kWarp)
            if (i != task) own += gb_born_term(xl[i], a.lig_p[i].z, xj, pj.y);
        for (int i = lane; i < a.n_rec; i += kWarp) rec += gb_born_term(xr[i], a.rec_p[i].z, xj, pj.y);
        own = gb_lane_sum<kWarp>(own);
        rec = gb_lane_sum<kWarp>(rec);
        if (lane == 0) {
            a.ib_lig[static_cast<size_t>(p) * a.n_lig + task] = gb_inverse_born(own, pj);
            ib[task] = gb_inverse_born(own + rec, pj);
        }
        return;
    }
    const int j = (task - a.n_lig) * (kWarp / kGbLanes) + lane / kGbLanes;
    const int jc = min(j, a.n_rec - 1);  // every lane of a warp that has an atom meets the shuffles
    if (jc < 0) return;
    const double4 xj = xr[jc], pj = a.rec_p[jc];
    double sum = 0.0;
    for (int i = lane % kGbLanes; i < a.n_lig; i += kGbLanes) sum += gb_born_term(xl[i], a.lig_p[i].z, xj, pj.y);
    sum = gb_lane_sum<kGbLanes>(sum);
    if (lane % kGbLanes == 0 && j < a.n_rec)
        ib[a.n_lig + j] = gb_inverse_born(a.sum_rr[static_cast<size_t>(c) * a.n_rec + j] + sum, pj);
}

// A system of the batch: its atoms and their inverse Born radii.
struct GbSystem {
    const double4 *lig, *rec;
    const double* ib;
    int n_lig, n;
    __device__ __forceinline__ double4 atom(int i) const { return i < n_lig ? lig[i] : rec[i - n_lig]; }
};

__device__ __forceinline__ GbSystem gb_system(const GbArgs& a, int s) {
    if (s < a.n_poses)
        return {a.lig + static_cast<size_t>(s) * a.n_lig, a.rec + (a.n_conf > 1 ? static_cast<size_t>(s) * a.n_rec : 0),
                a.ib_com + static_cast<size_t>(s) * (a.n_lig + a.n_rec), a.n_lig, a.n_lig + a.n_rec};
    s -= a.n_poses;
    if (s < a.n_conf)
        return {nullptr, a.rec + static_cast<size_t>(s) * a.n_rec, a.ib_rec + static_cast<size_t>(s) * a.n_rec, 0, a.n_rec};
    s -= a.n_conf;
    return {a.lig + static_cast<size_t>(s) * a.n_lig, nullptr, a.ib_lig + static_cast<size_t>(s) * a.n_lig, a.n_lig, a.n_lig};
}

constexpr double kGbKappa = 0.09293963686178248, kGbSolvent = 78.5, kGbProbe = 1.4, kGbSurface = 0.0678584012906;
constexpr double kGbCoulomb = 332.0637141491396;

__device__ __forceinline__ double gb_prefactor(double f) {
    return 0.5 * kGbCoulomb * (1.0 - exp(-kGbKappa * f) / kGbSolvent);
}

// Pair energies of one 64 x 64 tile (rows bi <= columns bj of the triangle i < j). The FP64 pipe
// bounds it (86 % busy), so the operations per pair are what counts: 66 with the library's exp
// and a division per pair, 45 with gb_exp, the division as a multiplication and the constant
// factors outside the loop (2.00 -> 1.35 ms for 8 poses in a pocket of 1,866 atoms).
__global__ void __launch_bounds__(kGbThreads) gb_pair_kernel(const __grid_constant__ GbArgs a) {
    __shared__ double4 s_x[kGbTile];
    __shared__ double s_ib[kGbTile], s_b[kGbTile];
    __shared__ double s_sum[kGbThreads / kWarp], s_exp[kExpTable];
    const GbSystem y = gb_system(a, blockIdx.y);
    const int nb = (y.n + kGbTile - 1) / kGbTile;
    int bi = 0, t = blockIdx.x;
    if (t >= nb * (nb + 1) / 2) return;
    while (t >= nb - bi) t -= nb - bi++;
    const int i0 = bi * kGbTile, j = (bi + t) * kGbTile + (threadIdx.x & (kGbTile - 1));
    const int ni = min(kGbTile, y.n - i0);
    for (int u = threadIdx.x; u < ni; u += kGbThreads) {
        s_x[u] = y.atom(i0 + u);
        const double ib = y.ib[i0 + u];
        s_ib[u] = -0.25 * ib;
        s_b[u] = 1.0 / ib;
    }
    for (int k = threadIdx.x; k < kExpTable; k += kGbThreads) s_exp[k] = a.exp2.v[k];
    __syncthreads();
    double e = 0.0;
    if (j < y.n) {
        const double4 xj = y.atom(j);
        const double ibj = y.ib[j], bj = 1.0 / ibj;
        const int last = min(ni, j - i0);  // i < j
        for (int u = threadIdx.x / kGbTile; u < last; u += kGbThreads / kGbTile) {
            const double4 xi = s_x[u];
            const double dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
            const double r2 = dx * dx + dy * dy + dz * dz;
            const double s = fma(s_b[u] * bj, gb_exp(r2 * (s_ib[u] * ibj), s_exp), r2) + 1e-20;
            const double fi = rsqrt(s);
            e = fma(xi.w * fi, fma(gb_exp(s * fi * -kGbKappa, s_exp), -1.0 / kGbSolvent, 1.0), e);
        }
        e *= xj.w * (0.5 * kGbCoulomb);
    }
    e = gb_lane_sum<kWarp>(e);
    if ((threadIdx.x & (kWarp - 1)) == 0) s_sum[threadIdx.x / kWarp] = e;
    __syncthreads();
    if (threadIdx.x == 0) {
        double v = 0.0;
        for (int w = 0; w < kGbThreads / kWarp; ++w) v += s_sum[w];
        a.partial[static_cast<size_t>(blockIdx.y) * a.n_tiles + blockIdx.x] = -2.0 * v;
    }
}

// A system's total: its tiles' pair energies, and per atom the self energy and the surface term.
__global__ void __launch_bounds__(kGbThreads) gb_total_kernel(const __grid_constant__ GbArgs a) {
    __shared__ double s_sum[kGbThreads / kWarp];
    const GbSystem y = gb_system(a, blockIdx.x);
    const int nb = (y.n + kGbTile - 1) / kGbTile;
    double e = 0.0;
    for (int t = threadIdx.x; t < nb * (nb + 1) / 2; t += kGbThreads)
        e += a.partial[static_cast<size_t>(blockIdx.x) * a.n_tiles + t];
    for (int i = threadIdx.x; i < y.n; i += kGbThreads) {
        const double q = y.atom(i).w, ib = y.ib[i];
        const double radius = i < y.n_lig ? a.lig_p[i].x : a.rec_p[i - y.n_lig].x;
        const double rr = radius + kGbProbe, x2 = radius * ib * (radius * ib);
        e += rr * rr * (x2 * x2 * x2) * kGbSurface - q * q * ib * gb_prefactor(1.0 / ib);
    }
    e = gb_lane_sum<kWarp>(e);
    if ((threadIdx.x & (kWarp - 1)) == 0) s_sum[threadIdx.x / kWarp] = e;
    __syncthreads();
    if (threadIdx.x == 0) {
        double v = 0.0;
        for (int w = 0; w < kGbThreads / kWarp; ++w) v += s_sum[w];
        a.energy[blockIdx.x] = v;
    }
}

static std::vector<double4> gb_properties4(const std::vector<double>& radius, const std::vector<double>& screen) {
    std::vector<double4> v;
    for (size_t i = 0; i < radius.size(); ++i) {
        const double rho = radius[i] - kGbOffset;
        v.push_back(make_double4(radius[i], rho, rho * screen[i], 0.0));
    }
    return v;
}

// Receptor coordinates for torsions t in FP64 (torsional_receptor::apply_parameters).
static std::vector<double> receptor_coords(pxd_context* ctx, const double* t) {
    std::vector<double> x = ctx->rec_xyz;
    for (int r = 0; r < ctx->rec.n_rotors; ++r) {
        const double* k = &ctx->rotor_axis[3 * r];
        const double* o = &ctx->rotor_origin[3 * r];
        const double st = std::sin(t[r]), ct = std::cos(t[r]), omc = 1 - ct;
        const double m[9] = {ct + k[0] * k[0] * omc,        k[0] * k[1] * omc - k[2] * st,
                             k[1] * st + k[0] * k[2] * omc, k[2] * st + k[0] * k[1] * omc,
                             ct + k[1] * k[1] * omc,        k[1] * k[2] * omc - k[0] * st,
                             k[0] * k[2] * omc - k[1] * st, k[0] * st + k[1] * k[2] * omc,
                             ct + k[2] * k[2] * omc};
        for (int u = ctx->rotor_mov_off[r]; u < ctx->rotor_mov_off[r + 1]; ++u) {
            double* p = &x[3 * static_cast<size_t>(ctx->mov_atoms[u])];
            const double v[3] = {p[0] - o[0], p[1] - o[1], p[2] - o[2]};
            for (int d = 0; d < 3; ++d) p[d] = m[3 * d] * v[0] + m[3 * d + 1] * v[1] + m[3 * d + 2] * v[2] + o[d];
        }
    }
    return x;
}

// Poses per batch of gbsa_batch: a pose's tile sums grow with the square of its atoms (1.2 MB at
// 20,000), and with rotors each has a receptor of its own.
static int gb_batch_poses(const pxd_context* ctx, const LigandEntry& e) {
    const size_t nr = ctx->n_rec, nl = e.n_atoms, nb = (nl + nr + kGbTile - 1) / kGbTile;
    const bool own = ctx->rec.n_rotors > 0;
    const size_t pose = sizeof(double) * ((own ? 3 : 2) * (nb * (nb + 1) / 2) + nr + 2 * nl + (own ? 2 * nr : 0)) +
                        sizeof(double4) * (nl + (own ? nr : 0));
    return static_cast<int>(std::min<size_t>(std::max<size_t>(kGbBytes / pose, 1), kGbPoses));
}

// GB/SA energies of n poses of one ligand (lig_xyz [n][N][3], rec_tors [n][R]):
// complex, ligand and receptor energies of pose k in parts[3 k .. 3 k + 2].
static int gbsa_batch(pxd_context* ctx, const LigandEntry& e, int n, const double* lig_xyz, const double* rec_tors,
                      double* parts) {
    const int nl = e.n_atoms, nr = ctx->n_rec, R = ctx->rec.n_rotors;
    const int nc = R > 0 ? n : 1;
    std::vector<double4> rec, lig;
    for (int c = 0; c < nc; ++c) {
        const std::vector<double> x = receptor_coords(ctx, R > 0 ? rec_tors + static_cast<size_t>(c) * R : nullptr);
        for (int i = 0; i < nr; ++i) rec.push_back(make_double4(x[3 * i], x[3 * i + 1], x[3 * i + 2], ctx->rec_charge[i]));
    }
    for (int p = 0; p < n; ++p)
        for (int i = 0; i < nl; ++i) {
            const double* x = lig_xyz + 3 * (static_cast<size_t>(p) * nl + i);
            lig.push_back(make_double4(x[0], x[1], x[2], e.charge[i]));
        }
    Pack pk;
    const size_t o_rec = pk.put(rec), o_lig = pk.put(lig);
    const size_t o_rp = pk.put(gb_properties4(ctx->rec_gb_radius, ctx->rec_gb_screen));
    const size_t o_lp = pk.put(gb_properties4(e.gb_radius, e.gb_screen));
    const int nb = (nl + nr + kGbTile - 1) / kGbTile, systems = 2 * n + nc;
    GbArgs a{};
    static const GbExpTable exp2 = gb_exp_table();
    a.exp2 = exp2;
    a.n_lig = nl;
    a.n_rec = nr;
    a.n_poses = n;
    a.n_conf = nc;
    a.n_tiles = nb * (nb + 1) / 2;
    const size_t in_bytes = (pk.bytes.size() + 15) / 16 * 16;
    const size_t rec_n = static_cast<size_t>(nc) * nr, lig_n = static_cast<size_t>(n) * nl;
    const size_t doubles = 2 * rec_n + lig_n + lig_n + static_cast<size_t>(n) * nr +
                           static_cast<size_t>(systems) * a.n_tiles + systems;
    void* mem = nullptr;
    int rc = cuda_check(ctx, cudaMallocAsync(&mem, in_bytes + sizeof(double) * doubles, ctx->stream), "gbsa buffers");
    if (rc) return rc;
    a.rec = at<double4>(mem, o_rec);
    a.lig = at<double4>(mem, o_lig);
    a.rec_p = at<double4>(mem, o_rp);
    a.lig_p = at<double4>(mem, o_lp);
    a.sum_rr = reinterpret_cast<double*>(static_cast<char*>(mem) + in_bytes);
    a.ib_rec = a.sum_rr + rec_n;
    a.ib_lig = a.ib_rec + rec_n;
    a.ib_com = a.ib_lig + lig_n;
    a.partial = a.ib_com + lig_n + static_cast<size_t>(n) * nr;
    a.energy = a.partial + static_cast<size_t>(systems) * a.n_tiles;
    queue_copy(ctx, &rc, mem, pk.bytes.data(), pk.bytes.size(), cudaMemcpyHostToDevice, ctx->stream, "gbsa inputs");
    if (!rc) {
        constexpr int warps = kGbThreads / kWarp;
        if (nr > 0) gb_receptor_kernel<<<dim3((nr + warps - 1) / warps, nc), kGbThreads, 0, ctx->stream>>>(a);
        constexpr int per = kWarp / kGbLanes;
        const int tasks = nl + (nr + per - 1) / per;
        gb_complex_kernel<<<dim3((tasks + warps - 1) / warps, n), kGbThreads, 0, ctx->stream>>>(a);
        gb_pair_kernel<<<dim3(a.n_tiles, systems), kGbThreads, 0, ctx->stream>>>(a);
        gb_total_kernel<<<systems, kGbThreads, 0, ctx->stream>>>(a);
        rc = cuda_check(ctx, cudaGetLastError(), "gbsa kernels launch");
    }
    std::vector<double> out(systems);
    queue_copy(ctx, &rc, out.data(), a.energy, sizeof(double) * systems, cudaMemcpyDeviceToHost, ctx->stream, "gbsa sums");
    cudaFreeAsync(mem, ctx->stream);
    rc = sync_copies(ctx, rc, ctx->stream, "gbsa");
    if (rc) return rc;
    for (int p = 0; p < n; ++p) {
        parts[3 * p] = out[p];
        parts[3 * p + 1] = out[n + nc + p];
        parts[3 * p + 2] = out[n + (nc > 1 ? p : 0)];
    }
    return PXD_OK;
}

}  // namespace pxd

using namespace pxd;

extern "C" {

int pxd_set_scoring_function(pxd_context* ctx, int32_t which, const pxd_sf_params* p) {
    if (!ctx || !p || which < 0 || which > 1) return PXD_ERR_INVALID;
    cudaSetDevice(ctx->device);
    DevSf h{};
    for (int k = 0; k < PXD_NUM_TERMS; ++k) h.coef[k] = static_cast<float>(p->coef[k]);
    h.vdw_scale = static_cast<float>(p->vdw_scale);
    h.vdw_cutoff = static_cast<float>(p->vdw_cutoff);
    for (int t = 0; t < PXD_NUM_VDW_TYPES; ++t) {
        // mm_interaction_vdw_energy constructor (scorer.cpp:207-220)
        h.vdw_type[t] = make_float2(static_cast<float>(PXD_VDW_SIGMA[t] * p->vdw_sigma_scale[t]),
                                    static_cast<float>(PXD_VDW_EPSILON[t] * p->vdw_epsilon_scale[t]));
        h.vdw_sigma_raw[t] = static_cast<float>(PXD_VDW_SIGMA[t]);
    }
    for (int k = 0; k < 2; ++k) {
        h.ionic_coef[k] = static_cast<float>(p->ionic_coef[k]);
        for (int u = 0; u < 2; ++u) h.ionic[k][u] = static_cast<float>(p->ionic[k][u]);
    }
    for (int k = 0; k < 4; ++k) {
        h.picat_coef[k] = static_cast<float>(p->picat_coef[k]);
        for (int u = 0; u < 2; ++u) h.picat[k][u] = static_cast<float>(p->picat[k][u]);
    }
    for (int w = 0; w < 2; ++w)
        for (int k = 0; k < 4; ++k) {
            h.stack_coef[w][k] = static_cast<float>(p->stack_coef[w][k]);
            for (int u = 0; u < 6; ++u) h.stack[w][k][u] = static_cast<float>(p->stack[w][k][u]);
        }
    h.hbond_scale = static_cast<float>(p->hbond_scale);
    for (int k = 0; k < 8; ++k) {
        h.hbond_coef[k] = static_cast<float>(p->hbond_coef[k]);
        for (int u = 0; u < 6; ++u) h.hbond[k][u] = static_cast<float>(p->hbond[k][u]);
    }
    h.hydro_scale = static_cast<float>(p->hydro_scale);
    h.hydro_min = static_cast<float>(p->hydro_dist_min);
    h.hydro_max = static_cast<float>(p->hydro_dist_max);
    h.hydro_factor = static_cast<float>(p->hydro_scale_factor);
    if (!ctx->d_sf[which]) {
        int rc = cuda_check(ctx, cudaMalloc(&ctx->d_sf[which], sizeof(DevSf)), "scoring function");
        if (rc) return rc;
    }
    // the new table's memory first: without it, the function and table that were there stay
    float2* table = nullptr;
    int rc = ctx->has_receptor ? alloc_score_table(ctx, &table) : PXD_OK;
    if (rc) return rc;
    ctx->sf_set[which] = false;
    rc = upload(ctx, ctx->d_sf[which], &h, sizeof(DevSf), "scoring function copy");
    if (!rc && table) rc = fill_score_table(ctx, which, table);
    if (rc) {
        if (table) cudaFree(table);
        return rc;
    }
    if (ctx->d_vdw[which]) cudaFree(ctx->d_vdw[which]);
    ctx->d_vdw[which] = table;
    ctx->sf_host[which] = *p;
    ctx->sf_set[which] = true;
    return PXD_OK;
}

int pxd_score_dev(pxd_context* ctx, int32_t which, int32_t n_poses, int32_t max_atoms, const int32_t* ids,
                  const float* xyz, const float* tors, double* score, double* terms, void* stream) {
    if (!ctx) return PXD_ERR_INVALID;
    if (which < 0 || which > 1 || n_poses < 0 || max_atoms <= 0 || max_atoms > PXD_MAX_LIGAND_ATOMS)
        return set_error(ctx, PXD_ERR_INVALID, "bad score batch");
    if (!ctx->has_receptor) return set_error(ctx, PXD_ERR_STATE, "set a receptor first");
    if (!ctx->sf_set[which]) return set_error(ctx, PXD_ERR_STATE, "set the scoring function first");
    if (ctx->rec.n_rotors > 0 && !tors) return set_error(ctx, PXD_ERR_INVALID, "receptor torsion buffer required");
    cudaSetDevice(ctx->device);
    if (n_poses == 0) return PXD_OK;
    int rc = sync_ligand_table(ctx);
    if (rc) return rc;
    EsArgs a{};
    a.env.rs = ctx->rec_score;
    a.env.sf = ctx->d_sf[which];
    a.env.vdw = ctx->d_vdw[which];
    a.rec = ctx->rec;
    a.ligands = ctx->d_ligands;
    a.n_ligands = static_cast<int>(ctx->ligands.size());
    a.lig_ids = ids;
    a.xyz = xyz;
    a.tors = tors;
    a.max_atoms = max_atoms;
    a.n_poses = n_poses;
    a.score = score;
    a.terms = terms;
    const size_t smem = sizeof(float4) * (max_atoms + ctx->rec.n_mov + 1);
    if (smem > 32 * 1024) {  // with the kernel's own 12.1 KB, towards the 48 KB of an unasked launch
        rc = raise_smem_limit(ctx, reinterpret_cast<const void*>(empirical_score_kernel), smem, "score smem");
        if (rc) return rc;
    }
    // enough warps to fill the chip: four per pose (the kernel's least) once the poses do, up to 16
    // for a few poses
    int warps = 4;
    while (warps < kMaxScoreWarps && static_cast<long long>(n_poses) * warps < 16LL * ctx->n_sm) warps *= 2;
    const int blocks = std::min(n_poses, ctx->n_sm * 64);
    cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : ctx->stream;
    empirical_score_kernel<<<blocks, warps * kWarp, smem, s>>>(a);
    return cuda_check(ctx, cudaGetLastError(), "empirical_score_kernel launch");
}

int pxd_score_gbsa(pxd_context* ctx, int32_t lig, const double* lig_xyz, const double* rec_tors, double* delta,
                   double* parts) {
    if (!ctx || !lig_xyz || !delta) return PXD_ERR_INVALID;
    if (!ctx->has_receptor) return set_error(ctx, PXD_ERR_STATE, "set a receptor first");
    if (lig < 0 || lig >= static_cast<int>(ctx->ligands.size())) return set_error(ctx, PXD_ERR_INVALID, "ligand id");
    if (ctx->rec.n_rotors > 0 && !rec_tors) return set_error(ctx, PXD_ERR_INVALID, "receptor torsions required");
    cudaSetDevice(ctx->device);
    double out[3];
    const int rc = gbsa_batch(ctx, ctx->ligands[lig], 1, lig_xyz, rec_tors, out);
    if (rc) return rc;
    *delta = out[0] - out[1] - out[2];
    if (parts)
        for (int k = 0; k < 3; ++k) parts[k] = out[k];
    return PXD_OK;
}

int pxd_score(pxd_context* ctx, int32_t which, int32_t lig, int32_t n_poses, const double* xyz, const double* tors,
              double* score, double* terms) {
    if (!ctx) return PXD_ERR_INVALID;
    if (lig < 0 || lig >= static_cast<int>(ctx->ligands.size()) || n_poses < 0 || which < 0 || which > 1)
        return set_error(ctx, PXD_ERR_INVALID, "ligand id / batch");
    if (!ctx->has_receptor) return set_error(ctx, PXD_ERR_STATE, "set a receptor first");
    cudaSetDevice(ctx->device);
    const int N = ctx->ligands[lig].n_atoms, R = ctx->rec.n_rotors;
    const size_t nx = static_cast<size_t>(n_poses) * N * 3, nt = static_cast<size_t>(n_poses) * R;
    std::vector<float> hx(nx), ht(nt);
    for (size_t i = 0; i < nx; ++i) hx[i] = static_cast<float>(xyz[i]);
    for (size_t i = 0; i < nt; ++i) ht[i] = static_cast<float>(tors[i]);
    std::vector<int> ids(n_poses, lig);
    void* mem = nullptr;
    const size_t bytes = 4 * (nx + nt + n_poses) + 8 * (n_poses + static_cast<size_t>(n_poses) * PXD_NUM_TERMS) + 64;
    int rc = cuda_check(ctx, cudaMallocAsync(&mem, bytes, ctx->stream), "score staging");
    if (rc) return rc;
    double* d_s = static_cast<double*>(mem);
    double* d_t = d_s + n_poses;
    float* d_x = reinterpret_cast<float*>(d_t + static_cast<size_t>(n_poses) * PXD_NUM_TERMS);
    float* d_r = d_x + nx;
    int* d_i = reinterpret_cast<int*>(d_r + nt + 1);
    queue_copy(ctx, &rc, d_x, hx.data(), 4 * nx, cudaMemcpyHostToDevice, ctx->stream, "score coordinates");
    if (nt) queue_copy(ctx, &rc, d_r, ht.data(), 4 * nt, cudaMemcpyHostToDevice, ctx->stream, "score torsions");
    queue_copy(ctx, &rc, d_i, ids.data(), 4 * static_cast<size_t>(n_poses), cudaMemcpyHostToDevice, ctx->stream,
               "score ligand ids");
    if (!rc) rc = pxd_score_dev(ctx, which, n_poses, N, d_i, d_x, d_r, d_s, d_t, ctx->stream);
    std::vector<double> ht2(static_cast<size_t>(n_poses) * PXD_NUM_TERMS);
    queue_copy(ctx, &rc, score, d_s, 8 * static_cast<size_t>(n_poses), cudaMemcpyDeviceToHost, ctx->stream,
               "scores");
    queue_copy(ctx, &rc, ht2.data(), d_t, 8 * ht2.size(), cudaMemcpyDeviceToHost, ctx->stream, "score terms");
    cudaFreeAsync(mem, ctx->stream);
    rc = sync_copies(ctx, rc, ctx->stream, "score");
    if (rc) return rc;
    const double gcoef = ctx->sf_host[which].coef[PXD_TERM_GBSA];
    if (gcoef > 1e-5 || gcoef < -1e-5) {
        if (R > 0 && !tors) return set_error(ctx, PXD_ERR_INVALID, "receptor torsions required");
        int batch = std::min(n_poses, gb_batch_poses(ctx, ctx->ligands[lig]));
        std::vector<double> parts(3 * static_cast<size_t>(batch));
        for (int p0 = 0, n; p0 < n_poses; p0 += n) {
            for (;; batch = n / 2) {  // smaller where the device is short of memory
                n = std::min(batch, n_poses - p0);
                rc = gbsa_batch(ctx, ctx->ligands[lig], n, xyz + 3 * static_cast<size_t>(N) * p0,
                                R > 0 ? tors + static_cast<size_t>(R) * p0 : nullptr, parts.data());
                if (rc != PXD_ERR_NOMEM || n <= 1) break;
                cudaGetLastError();
            }
            if (rc) return rc;
            for (int p = 0; p < n; ++p) {
                const double g = parts[3 * p] - parts[3 * p + 1] - parts[3 * p + 2];
                ht2[static_cast<size_t>(p0 + p) * PXD_NUM_TERMS + PXD_TERM_GBSA] = g;
                score[p0 + p] += gcoef * g;
            }
        }
    }
    for (int p = 0; p < n_poses; ++p) {
        if (terms)
            for (int k = 0; k < PXD_NUM_TERMS; ++k)
                terms[static_cast<size_t>(p) * PXD_NUM_TERMS + k] = ht2[static_cast<size_t>(p) * PXD_NUM_TERMS + k];
    }
    return PXD_OK;
}

}  // extern "C"
