"""The work that a user of pxdock_gb300 has it do, as cases that can be timed and checked.

A case is a dict of plain values; its "kind" names the call. `prepare` makes what a program
has in hand before the call (contexts with a receptor, ligands and maps; poses), `run` makes
the call through the package's public entry points and returns its outputs, `work` counts the
bytes and operations that the call cannot do without, and `exact` gives the outputs in FP64
from plain torch where they are not the end of an iteration that amplifies rounding (the
optimiser and the search: their iterates part after a few dozen evaluations).

Molecules are the package's seeded synthetic complexes (the shapes of its benchmark and
tests): pockets of 300-2,500 heavy atoms with polar hydrogens, ligands of 8-60 heavy atoms.
The optimiser and search cases load their maps from records in hand, as a program that keeps
a map cache does; the other cases build them.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

_HERE = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(os.getcwd(), "protenix-dock_gb300") not in sys.path:
    sys.path.insert(0, os.path.join(os.getcwd(), "protenix-dock_gb300"))

from pxdock_gb300 import abi, autograd, model, native, synth, unroll  # noqa: E402

SLOPE = 1e6      # the engine's default out-of-box slope
SPACING = 0.375  # the engine's default map spacing


# ------------------------------------------------------------------------------- the cases
def listed():
    return [
        # a new pocket: the maps of the ligand's vdW types over a 30 A box, read back for a cache
        dict(name="maps_81", kind="maps", heavy=1500, lig=24, rot=5, box=30.0, box_y=30.0, box_z=30.0,
             spacing=SPACING),
        # the engine's start: maps of all 99 ligand types over a 20 A box, then the first poses scored
        dict(name="maps_all_types", kind="engine_start", heavy=1500, lig=24, rot=5, box=20.0, box_y=18.0,
             box_z=19.1, spacing=SPACING, poses=37),
        # one pose's energy and gradient from host arrays: a script that steps a pose itself
        dict(name="energy_one_pose", kind="energy_host", heavy=1500, lig=24, rot=5, box=20.0, poses=1),
        # energies and gradients of a large batch on the device: rescoring, a gradient-based sampler
        dict(name="energy_batch", kind="energy", heavy=1500, lig=24, rot=5, box=30.0, poses=65536),
        # the pose-selection score of the poses of a docking run
        dict(name="pose_scores", kind="score", heavy=1500, lig=31, rot=7, which=0, poses=2049),
        # the affinity score (with GB/SA) of the poses kept for one ligand
        dict(name="affinity_scores", kind="score", heavy=1500, lig=24, rot=5, which=1, poses=8),
        # one training step on fixed poses: score and docking energy, gradients to the pose
        # variables, the 36 weights and the pair tables
        dict(name="train_fixed_poses", kind="train", heavy=1500, lig=30, rot=5, box=20.0, complexes=16, poses=256),
        # the second-order products of a training step through the optimiser
        dict(name="train_second_order", kind="second", heavy=600, lig=32, rot=6, complexes=32, poses=64),
        # batched pose optimisation at the benchmark's size
        dict(name="optimize_batch", kind="optimize", heavy=1500, lig=24, rot=5, box=30.0, poses=65536, rotors=0,
             history=8, iters=300, tol=1e-3),
        # the poses of one ligand file with the engine's own constants and movable receptor hydroxyls
        dict(name="optimize_one_ligand", kind="optimize", heavy=1500, lig=24, rot=5, box=20.0, poses=48, rotors=4,
             history=100, iters=240, tol=0.5),
        # screening: ligands of uneven size in one launch
        dict(name="optimize_screen", kind="screen", heavy=1500, ligands=24, poses=96, box=22.5, history=8, iters=300,
             tol=1e-3),
        # the docking search of one complex at the engine's exhaustiveness
        dict(name="search", kind="search", heavy=1500, lig=24, rot=5, box=20.0, walkers=64, steps=24, relax=40),
    ]


def draw(rng):
    """One more case of the ranges that the listed ones stand for."""
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    lig = log(8, 45)
    rot = rng.randint(0, min(8, lig // 3))
    heavy = log(300, 2500)
    kind = rng.choice(["maps", "engine_start", "energy_host", "energy", "score", "score", "train", "second",
                       "optimize", "screen", "search"])
    side = lambda lo, hi: round(rng.uniform(lo, hi), 2)  # noqa: E731
    if kind in ("maps", "engine_start"):
        hi = 26.0 if kind == "maps" else 16.0
        c = dict(kind=kind, heavy=min(heavy, 1900), lig=lig, rot=rot, box=side(9, hi), box_y=side(9, hi),
                 box_z=side(9, hi), spacing=rng.choice([0.375, 0.375, 0.5, 0.42]))
        return dict(c, poses=log(1, 300)) if kind == "engine_start" else c
    if kind == "energy_host":
        return dict(kind=kind, heavy=heavy, lig=lig, rot=rot, box=side(15, 25), poses=log(1, 200))
    if kind == "energy":
        return dict(kind=kind, heavy=heavy, lig=min(lig, 30), rot=min(rot, 10), box=side(15, 30), poses=log(100, 60000))
    if kind == "score":
        which = rng.randint(0, 1)
        return dict(kind=kind, heavy=heavy, lig=lig, rot=rot, which=which, poses=log(1, 24) if which else log(1, 8000))
    if kind == "train":
        return dict(kind=kind, heavy=min(heavy, 1500), lig=min(lig, 32), rot=min(rot, 8), box=side(15, 20),
                    complexes=log(1, 16), poses=log(16, 256))
    if kind == "second":
        return dict(kind=kind, heavy=min(heavy, 700), lig=lig, rot=rot, complexes=log(1, 32), poses=log(16, 64))
    if kind == "optimize":
        rotors = rng.choice([0, 0, 3, 8])
        ref = rng.random() < 0.5
        return dict(kind=kind, heavy=min(max(heavy, 600), 1600), lig=min(lig, 24), rot=min(rot, 8), box=side(15, 24),
                    poses=log(1, 300) if ref else log(300, 20000), rotors=rotors, history=100 if ref else 8,
                    iters=240 if ref else 300, tol=0.5 if ref else 1e-3)
    if kind == "screen":
        return dict(kind=kind, heavy=min(heavy, 1600), ligands=log(4, 24), poses=log(16, 96), box=side(15, 24), history=8,
                    iters=300, tol=1e-3)
    return dict(kind="search", heavy=min(heavy, 1600), lig=min(lig, 28), rot=min(rot, 8), box=side(14, 22),
                walkers=log(8, 300), steps=log(4, 24), relax=rng.choice([20, 40]))


# ----------------------------------------------------------------------- molecules and inputs
@functools.lru_cache(maxsize=96)
def _receptor(seed, heavy, rotors=0):
    cube = 26.0 * (heavy / 1500.0) ** (1.0 / 3.0)
    cavity = 7.0 * (heavy / 1500.0) ** (1.0 / 3.0)
    return model.Receptor.from_json(synth.make_receptor(seed=seed, n_heavy=heavy, cube=cube, cavity=cavity,
                                                        n_rotors=rotors))


@functools.lru_cache(maxsize=256)
def _ligand(seed, heavy, rot):
    for k in range(60):  # some draws of the generator cannot be embedded: try others, a little smaller
        h = max(8, heavy - k // 2)
        try:
            lj = synth.make_ligand(seed=seed + 7919 * k, n_heavy=h, n_rot=min(max(rot, h // 6), h // 3),
                                   n_n=max(1, round(0.12 * h)), n_o=max(1, round(0.15 * h)),
                                   n_other=round(0.03 * h), max_tries=15)
        except RuntimeError:
            continue
        lig = model.Ligand.from_json(lj)
        if lig.n_atoms <= 256 and lig.n_torsions <= 32 and lig.tree.n_frags <= 64:
            return lig
    raise RuntimeError("no ligand of %d heavy atoms" % heavy)


@functools.lru_cache(maxsize=1)
def _scoring():
    return model.load_scoring_function(os.path.join(os.path.dirname(os.path.abspath(model.__file__)), "data",
                                                    "scoring_function.json"))


def _types(*ligands):
    return sorted(set(int(t) for lig in ligands for t in lig.vdw_type))


def _box(case):
    b = case["box"]
    return model.make_box((0.0, 0.0, 0.0), (b, case.get("box_y", b), case.get("box_z", b)),
                          case.get("spacing", SPACING))


def _corners(box):
    lo = np.array(box.init_xyz)
    return lo, lo + (np.array(box.npoints) - 1) * box.spacing


def _complex(case, seed):
    """The case's ligand in one of five pockets."""
    return _receptor(seed % 5, case["heavy"], case.get("rotors", 0)), _ligand(1, case["lig"], case["rot"])


def _context(rec, ligands, sf=False):
    ctx = native.Context(0)
    ctx.set_receptor(rec)
    ctx.set_slope(SLOPE)
    if sf:
        for which in (0, 1):
            ctx.set_scoring_function(which, _scoring()[which])
    return ctx, [ctx.add_ligand(lig) for lig in ligands]


@functools.lru_cache(maxsize=6)
def _cache_records(rec, dims, types):
    """The map records {E, dE/dx, dE/dy, dE/dz} of a box as a map cache holds them (FP32)."""
    box = model.make_box((0.0, 0.0, 0.0), dims, SPACING)
    return {t: m.to(torch.float32).cpu().numpy() for t, m in _maps64(rec, box, types).items()}


def _load_maps(ctx, rec, dims, types):
    box = model.make_box((0.0, 0.0, 0.0), dims, SPACING)
    for t, m in _cache_records(rec, dims, tuple(types)).items():
        ctx.write_map(box, t, m)
    return box


def _cuda(a, dtype):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype).cuda()


def _stream():
    return torch.cuda.current_stream().cuda_stream or 1


def _pocket_poses(lig, n, seed, scale=2.5):
    """Poses as a docking run leaves them: near the pocket's centre, any orientation and torsions."""
    return synth.random_poses(lig, [-scale] * 3, [scale] * 3, n, seed)


def _dofs(lig_of, D, seed):
    rng = np.random.default_rng(seed)
    q = unroll.random_dofs(rng, [lig.n_torsions for lig in lig_of], D, centre_scale=2.5)
    return q.astype(np.float32)


def _train_set(case, seed):
    """Complexes of a training set: receptors, ligands, and per pose its complex and variables."""
    n, P = case["complexes"], case["poses"]
    recs = [_receptor(100 + c + 50 * (seed % 3), case["heavy"]) for c in range(n)]
    sizes = [max(8, case["lig"] - 7 + 13 * c % 15) for c in range(n)]
    ligs = [_ligand(5000 + c, h, min(case["rot"], h // 3)) for c, h in enumerate(sizes)]
    cplx = np.repeat(np.arange(n), P)
    A = max(lig.n_atoms for lig in ligs)
    D = 7 + max(lig.n_torsions for lig in ligs)
    ref = np.zeros((n * P, A, 3), np.float32)
    for c, lig in enumerate(ligs):
        ref[c * P:(c + 1) * P, : lig.n_atoms] = lig.poses[0] - lig.poses[0].mean(axis=0)
    return recs, ligs, cplx, A, D, ref, _dofs([ligs[c] for c in cplx], D, seed)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("train", "second"):
        recs, ligs, cplx, A, D, ref, q = _train_set(case, seed)
        made = [_context(rec, [lig], sf=True) for rec, lig in zip(recs, ligs)]
        ctxs = [m[0] for m in made]
        s = dict(kind=kind, ctxs=ctxs, ctx_ids=_cuda(cplx, torch.int32),
                 lig_ids=_cuda([made[c][1][0] for c in cplx], torch.int32), ref=_cuda(ref, torch.float32),
                 q=_cuda(q, torch.float32), w=_cuda(abi.sf_weights(_scoring()[0]), torch.float64),
                 t=_cuda(abi.smooth_pair_tables(1), torch.float32))
        if kind == "train":
            box = _box(case)
            for ctx, lig in zip(ctxs, ligs):
                ctx.build_grid(box, _types(lig))
        else:
            s["backend"] = unroll.KernelBackend(ctxs, s["ctx_ids"], s["lig_ids"], s["ref"], D)
            s["u"] = _cuda(np.random.default_rng(seed + 1).normal(size=q.shape) * (np.abs(q) > 0), torch.float64)
        return s
    if kind == "screen":
        rec = _receptor(seed % 5, case["heavy"])
        ligs = [_ligand(1000 + k, 10 + 37 * k % 40, k % 9) for k in range(case["ligands"])]
        ctx, ids = _context(rec, ligs)
        box = _load_maps(ctx, rec, (case["box"],) * 3, _types(*ligs))
        P, A = case["poses"], max(lig.n_atoms for lig in ligs)
        xyz = np.zeros((P * len(ligs), A, 3))
        for k, lig in enumerate(ligs):
            xyz[k * P:(k + 1) * P, : lig.n_atoms] = synth.random_poses(lig, *_corners(box), P, seed + k)
        order = np.random.default_rng(seed).permutation(len(xyz))
        p = native.lbfgs_params(max_iter=case["iters"], history=case["history"], tolerance_grad=case["tol"])
        return dict(kind=kind, ctx=ctx, params=p, ids=np.repeat(np.array(ids, np.int32), P)[order], xyz=xyz[order])
    rec, lig = _complex(case, seed)
    ctx, (lid,) = _context(rec, [lig], sf=kind in ("score", "search"))
    s = dict(kind=kind, ctx=ctx, lid=lid)
    if kind == "maps":
        rng = np.random.default_rng(seed)
        s["box"] = model.make_box(tuple(rng.uniform(-1.0, 1.0, 3)), (case["box"], case["box_y"], case["box_z"]),
                                  case["spacing"])
        return dict(s, types=_types(lig))
    if kind == "score":
        return dict(s, which=case["which"], xyz=_pocket_poses(lig, case["poses"], seed))
    if kind in ("optimize", "search"):
        box = _load_maps(ctx, rec, (case["box"],) * 3, _types(lig))
    else:
        box = _box(case)
        if kind != "engine_start":
            ctx.build_grid(box, _types(lig))
    if kind == "search":
        lo, hi = _corners(box)
        s["params"] = native.mc_params(lo, hi, seed=seed % 100000, max_nsteps=case["steps"], relax_nsteps=case["relax"])
        s["starts"] = np.repeat(lig.poses[0][None], case["walkers"], axis=0)
        return dict(s, walkers=np.arange(case["walkers"]))
    n = case["poses"]
    xyz = synth.random_poses(lig, *_corners(box), n, seed)
    if kind == "optimize":
        s["params"] = native.lbfgs_params(max_iter=case["iters"], history=case["history"], tolerance_grad=case["tol"])
        s["tors"] = np.random.default_rng(seed).uniform(-math.pi, math.pi, size=(n, rec.n_rotors))
        if n <= 300:  # a ligand file's poses: host arrays
            return dict(s, xyz=xyz)
    if kind in ("energy_host", "engine_start"):
        return dict(s, xyz=xyz, box=box)
    s.update(start=_cuda(xyz, torch.float32), ids=torch.full((n,), lid, dtype=torch.int32, device="cuda"))
    if kind == "optimize":
        s["start_tors"] = _cuda(s.pop("tors") if rec.n_rotors else np.zeros((n, 1)), torch.float32)
    return s


# ------------------------------------------------------------------------------- the calls
def run(s):
    return _RUN[s["kind"]](s)


def _run_maps(s):
    s["ctx"].build_grid(s["box"], s["types"])
    return {"coulomb": s["ctx"].read_map(abi.COULOMB_MAP), "vdw": [s["ctx"].read_map(t) for t in s["types"]]}


def _run_engine_start(s):
    s["ctx"].build_grid(s["box"])
    e, g, _ = s["ctx"].score_grad(s["lid"], s["xyz"])
    return {"energy": e, "grad": g}


def _run_energy_host(s):
    e, g, _ = s["ctx"].score_grad(s["lid"], s["xyz"])
    return {"energy": e, "grad": g}


def _run_energy(s):
    x = s["start"]
    e = torch.empty(x.shape[0], dtype=torch.float64, device=x.device)
    g = torch.empty_like(x)
    s["ctx"].score_grad_dev(x.shape[0], x.shape[1], s["ids"].data_ptr(), x.data_ptr(), None, e.data_ptr(),
                            g.data_ptr(), None, stream=_stream())
    return {"energy": e, "grad": g}


def _run_score(s):
    score, terms = s["ctx"].score(s["which"], s["lid"], s["xyz"])
    return {"score": score, "terms": terms}


def _run_train(s):
    q, w, t = (s[k].detach().requires_grad_(True) for k in ("q", "w", "t"))
    xyz = autograd.ligand_pose_multi(s["ctxs"], s["ctx_ids"], s["lig_ids"], s["ref"], q)
    score = autograd.empirical_score(s["ctxs"], s["lig_ids"], xyz, w, t, ctx_ids=s["ctx_ids"])
    energy = autograd.docking_energy(s["ctxs"], s["lig_ids"], xyz, ctx_ids=s["ctx_ids"])
    (score + energy).mean().backward()
    return {"score": score.detach(), "energy": energy.detach(), "dq": q.grad, "dw": w.grad, "dt": t.grad}


def _run_second(s):
    b = s["backend"]
    g, x, gx = b.grad(s["q"], s["w"], s["t"])
    hu, dw, dt = b.hvp(s["q"], s["u"], x, gx, s["w"], s["t"])
    return {"g": g, "x": x, "gx": gx, "hu": hu, "dw": dw, "dt": dt}


def _run_optimize(s):
    if "xyz" in s:
        return s["ctx"].lbfgs(s["params"], s["lid"], s["xyz"], s["tors"])
    x, tors = s["start"].clone(), s["start_tors"].clone()
    n = x.shape[0]
    e = torch.empty(n, dtype=torch.float64, device=x.device)
    nev, st = (torch.empty(n, dtype=torch.int32, device=x.device) for _ in range(2))
    s["ctx"].lbfgs_dev(s["params"], n, x.shape[1], s["ids"].data_ptr(), x.data_ptr(), tors.data_ptr(), e.data_ptr(),
                       nev.data_ptr(), st.data_ptr(), stream=_stream())
    return {"xyz": x, "torsions": tors, "energy": e, "nevals": nev, "status": st}


def _run_screen(s):
    return s["ctx"].lbfgs_multi(s["params"], s["ids"], s["xyz"])


def _run_search(s):
    return s["ctx"].mc_search(s["params"], s["lid"], s["starts"], s["walkers"])


_RUN = {"maps": _run_maps, "engine_start": _run_engine_start, "energy_host": _run_energy_host, "energy": _run_energy,
        "score": _run_score, "train": _run_train, "second": _run_second, "optimize": _run_optimize,
        "screen": _run_screen, "search": _run_search}


# ------------------------------------------------------------------------------- the work
EVALS = {"optimize": 160, "screen": 220}  # evaluations per pose at 300 iterations (measured means)


def _evaluation(N):
    """Bytes and operations of one energy and gradient: two maps x 8 corners x 16 bytes per atom
    and the pose in and out; ~25 operations per atom pair, ~250 per atom for the bonded terms
    and the lookups."""
    return 256 * N + 24 * N, 25 * N * N / 2 + 250 * N


def work(case):
    kind = case["kind"]
    M = 1.25 * case["heavy"]  # receptor atoms with polar hydrogens
    N = 1.8 * case.get("lig", 34)
    if kind in ("maps", "engine_start"):
        P = 1
        for k in ("box", "box_y", "box_z"):
            nv = math.ceil(case[k] / case["spacing"])
            P *= nv + nv % 2 + 1
        T = 9 if kind == "maps" else 99
        # per point and receptor atom: distance and its powers (~16), Coulomb with gradient (8), and per
        # vdW type an energy and a gradient from them (4 per distinct receptor type, ~6 of them, per point)
        flops = P * M * 24 + P * T * 6 * 8
        return {"bytes": 20.0 * P * (T + 1) + 40 * M, "flops": float(flops)}
    if kind in ("energy", "energy_host"):
        b, f = _evaluation(N)
        return {"bytes": float(case["poses"] * 24 * N + min(case["poses"] * 256 * N, 16 * 10 * (case["box"] / SPACING) ** 3)),
                "flops": float(case["poses"] * f)}
    if kind == "score":
        pairs = N * M * case["poses"]
        flops = 18 * pairs
        if case["which"]:
            flops += case["poses"] * 35 * ((M + N) ** 2 + M ** 2)
        return {"bytes": float(case["poses"] * (12 * N + 96) + 24 * M), "flops": float(flops)}
    if kind == "train":
        n = case["complexes"] * case["poses"]
        return {"bytes": float(n * (12 * 4 * N + 300) + case["complexes"] * 28 * M), "flops": float(n * N * M * 30)}
    if kind == "second":
        n = case["complexes"] * case["poses"]
        return {"bytes": float(n * (12 * 6 * N + 200) + case["complexes"] * 28 * M), "flops": float(n * N * M * 90)}
    b, f = _evaluation(N)
    if kind == "search":
        evals = case["walkers"] * (250 + case["steps"] * case["relax"] * 0.8)
        score = case["walkers"] * case["steps"] * 18 * N * M
        return {"bytes": float(case["walkers"] * 24 * N * 2), "flops": float(evals * f + score)}
    poses = case["poses"] * case.get("ligands", 1)
    evals = poses * EVALS[kind]
    return {"bytes": float(poses * (24 * N + 16) + 16 * 10 * (case["box"] / SPACING) ** 3), "flops": float(evals * f)}


# ---------------------------------------------------------------------------- FP64 outputs
COULOMB = 332.0637141491396


def _d(a):
    return torch.as_tensor(np.asarray(a), dtype=torch.float64, device="cuda")


def _i(a):
    return torch.as_tensor(np.asarray(a), dtype=torch.int64, device="cuda")


def _maps64(rec, box, types):
    """{type or COULOMB_MAP: [P][4] records} in FP64: sums of inverse powers per receptor type."""
    keep = np.setdiff1d(np.arange(rec.n_atoms), rec.movable_atoms())
    kinds, cls = np.unique(np.stack([rec.ff.sigma[keep], rec.ff.epsilon[keep]], 1), axis=0, return_inverse=True)
    xyz, q = _d(rec.xyz[keep]), _d(rec.ff.charge[keep])
    one = torch.cat([torch.ones_like(xyz[:, :1]), xyz], 1)  # columns 1, x, y, z of every atom
    of = torch.nn.functional.one_hot(_i(cls.reshape(-1)), len(kinds)).double()
    cols = (of[:, :, None] * one[:, None, :]).flatten(1)    # the same, per receptor type
    sig, eps = model.vdw_table()
    axes = [_d(box.init_xyz[d] + box.spacing * np.arange(box.npoints[d])) for d in range(3)]
    pts = torch.stack(torch.meshgrid(*axes, indexing="ij"), -1).reshape(-1, 3)
    out = {t: torch.zeros((len(pts), 4), dtype=torch.float64, device="cuda") for t in [abi.COULOMB_MAP, *types]}
    for i in range(0, len(pts), 65536):
        p = pts[i:i + 65536]
        r2 = sum((p[:, d, None] - xyz[None, :, d]) ** 2 for d in range(3))
        inv = 1.0 / r2.clamp_min(1e-4)
        # sum of w (1, atom - point) from the sums of w (1, atom)
        moved = lambda s: torch.cat([s[..., :1], s[..., 1:] - p.view(-1, *[1] * (s.dim() - 2), 3) * s[..., :1]], -1)  # noqa: E731
        qr = q * inv.sqrt() * COULOMB
        out[abi.COULOMB_MAP][i:i + 65536, 0] = qr.sum(1)
        out[abi.COULOMB_MAP][i:i + 65536, 1:] = moved((qr * inv) @ one)[:, 1:]
        i6 = inv * inv * inv
        m6, m12 = i6 @ of, (i6 * i6) @ of
        v8 = moved(((i6 * inv) @ cols).view(len(p), -1, 4))[..., 1:]
        v14 = moved(((i6 * i6 * inv) @ cols).view(len(p), -1, 4))[..., 1:]
        for t in types:
            s6 = _d(((sig[t] + kinds[:, 0]) * 0.5) ** 6)
            C = _d(4.0 * np.sqrt(eps[t] * kinds[:, 1]))
            out[t][i:i + 65536, 0] = m12 @ (C * s6 * s6) - m6 @ (C * s6)
            out[t][i:i + 65536, 1:] = ((12.0 * C * s6 * s6)[:, None] * v14 - (6.0 * C * s6)[:, None] * v8).sum(1)
    return {t: m.clamp(-1e30, 1e30) for t, m in out.items()}


def _cross_angle(u, v):
    """(|u x v|, u . v) along the last axis."""
    c = torch.linalg.cross(u, v)
    return (c * c).sum(-1).clamp_min(1e-60).sqrt(), (u * v).sum(-1)


def _dihedral(x, a):
    rij, rkj, rkl = x[:, a[:, 1]] - x[:, a[:, 0]], x[:, a[:, 1]] - x[:, a[:, 2]], x[:, a[:, 3]] - x[:, a[:, 2]]
    m, n = torch.linalg.cross(rij, rkj), torch.linalg.cross(rkj, rkl)
    w, d = _cross_angle(m, n)
    phi = torch.atan2(w, d + 1e-20)
    return torch.where((rij * n).sum(-1) < 0, phi, -phi)


def _intra64(ff, x):
    """Force-field energy of poses x [B][N][3]."""
    e = x.new_zeros(x.shape[0])
    if len(ff.bonds):
        b = _i(ff.bonds)
        r = (x[:, b[:, 1]] - x[:, b[:, 0]]).norm(dim=-1)
        e = e + (0.5 * _d(ff.bond_k) * (r - _d(ff.bond_length)) ** 2).sum(1)
    if len(ff.angles):
        a = _i(ff.angles)
        w, d = _cross_angle(x[:, a[:, 1]] - x[:, a[:, 0]], x[:, a[:, 1]] - x[:, a[:, 2]])
        e = e + (0.5 * _d(ff.angle_k) * (torch.atan2(w, d + 1e-20) - _d(ff.angle_radian)) ** 2).sum(1)
    for atoms, per, phase, k in (ff.impropers, ff.propers):
        if len(atoms):
            on = np.cumprod(np.asarray(per) != 0, axis=1)
            th = _dihedral(x, _i(atoms))[..., None]
            e = e + (_d(k * on) * (1 + torch.cos(th * _d(per) - _d(phase)))).sum((1, 2))
    for pairs, sc, sv in ((ff.pairs14, 0.833333333, 0.5), (ff.pairs, 1.0, 1.0)):
        if len(pairs):
            i, j = np.asarray(pairs).T
            r2 = ((x[:, _i(j)] - x[:, _i(i)]) ** 2).sum(-1)
            u6 = (_d(((ff.sigma[i] + ff.sigma[j]) * 0.5) ** 2) / r2) ** 3
            e = e + (_d(ff.charge[i] * ff.charge[j] * sc * COULOMB) / r2.sqrt()).sum(1)
            e = e + (_d(np.sqrt(ff.epsilon[i] * ff.epsilon[j]) * sv * 4.0) * (u6 * u6 - u6)).sum(1)
    return e


def _lookup64(maps, box, lig, x):
    """Interpolated map energy [B] and gradient [B][N][3] of poses x, with the out-of-box penalty."""
    npt = _d(box.npoints) - 1
    f = (x - _d(box.init_xyz)) / box.spacing
    below, above = (-f).clamp_min(0), (f - npt).clamp_min(0)
    g = torch.minimum(f.clamp_min(0), npt)
    lo = torch.minimum(g.floor(), npt - 1)
    fr = g - lo
    lo = lo.long()
    ny, nz = box.npoints[1], box.npoints[2]
    q = _d(lig.ff.charge)
    rec = x.new_zeros(x.shape[:2] + (4,))
    for c in range(8):
        o = [(c >> d) & 1 for d in range(3)]
        w = torch.ones_like(fr[..., 0])
        for d in range(3):
            w = w * (fr[..., d] if o[d] else 1 - fr[..., d])
        at = ((lo[..., 0] + o[0]) * ny + lo[..., 1] + o[1]) * nz + lo[..., 2] + o[2]
        rec = rec + w[..., None] * q[:, None] * maps[abi.COULOMB_MAP][at]
        for t in _types(lig):
            own = _i(np.where(np.asarray(lig.vdw_type) == t)[0])
            rec[:, own] = rec[:, own] + w[:, own, None] * maps[t][at[:, own]]
    out = (below + above).sum(-1)
    grad = torch.where((out > 0)[..., None], SLOPE * ((above > 0).double() - (below > 0).double()), rec[..., 1:])
    return (rec[..., 0] + out * box.spacing * SLOPE).sum(1), grad


def _docking64(maps, box, lig, x):
    """Docking energy [B] of poses x and its gradient."""
    x = x.detach().requires_grad_(True)
    e = _intra64(lig.ff, x)
    (g,) = torch.autograd.grad(e.sum(), x)
    em, gm = _lookup64(maps, box, lig, x.detach())
    return e.detach() + em, g + gm


def _energy64(case, seed):
    rec, lig = _complex(case, seed)
    box = _box(case)
    maps = _maps64(rec, box, _types(lig))
    xyz = _d(synth.random_poses(lig, *_corners(box), case["poses"], seed)).float().double()
    both = [_docking64(maps, box, lig, xyz[i:i + 8192]) for i in range(0, len(xyz), 8192)]
    return {"energy": torch.cat([b[0] for b in both]), "grad": torch.cat([b[1] for b in both])}


def _ramp(v, lo, hi):
    return (1 - (v - lo) / (hi - lo)).clamp(0, 1)


def _acos_deg(c):
    return torch.acos(c.clamp(-1 + 1e-13, 1 - 1e-13)) * (180.0 / math.pi)


def _dist(a, b):
    """[B][n][m] distances between points a [B][n][3] and b [m][3] or [B][m][3]."""
    b = b if b.dim() == 3 else b[None]
    return sum((a[:, :, None, k] - b[:, None, :, k]) ** 2 for k in range(3)).clamp_min(1e-40).sqrt()


def _rings(x, rings):
    """Centroids and unit normals [B][r][3] of rings of poses x [B][n][3]."""
    c, n = [], []
    for r in rings:
        a = [int(k) for k in r if k >= 0]
        c.append(x[:, a].mean(1))
        v = torch.linalg.cross(x[:, a[1]] - x[:, a[0]], x[:, a[1]] - x[:, a[2]])
        n.append(v / v.norm(dim=-1, keepdim=True))
    z = x.new_zeros((x.shape[0], 0, 3))
    return (torch.stack(c, 1), torch.stack(n, 1)) if c else (z, z)


def _stack(rc, rn, lc, ln, p, centre):
    d = _dist(lc, rc)
    t = rc[:, None] - lc[:, :, None]
    proj = lambda n: ((t * t).sum(-1) - (n * t).sum(-1) ** 2).clamp_min(1e-40).sqrt()  # noqa: E731
    sg = torch.minimum(proj(rn[:, None]), proj(ln[:, :, None]))
    th = _acos_deg((rn[:, None] * ln[:, :, None]).sum(-1))
    th = torch.minimum(th, 180 - th)
    on = (d <= p[1]) & (sg <= p[5])
    v = _ramp(d, p[0], p[1]) * _ramp(sg, p[4], p[5]) * _ramp((th - centre).abs(), p[2], p[3])
    return -torch.where(on, v, torch.zeros_like(v)).sum((1, 2))


def _hbond(dpos, hpos, apos, p):
    """Donors (dpos, hpos) [B|1][d][3] x acceptors apos [B|1][a][3]."""
    h2d = (dpos - hpos)[:, :, None]
    h2a = apos[:, None] - hpos[:, :, None]
    r = (h2a * h2a).sum(-1).clamp_min(1e-40).sqrt()
    ang = _acos_deg((h2d * h2a).sum(-1) / (h2d.norm(dim=-1) * r + 1e-20))
    return -(_ramp((r - p[4]).abs(), p[0], p[1]) * _ramp((ang - p[5]).abs(), p[2], p[3])).sum((1, 2))


def _features64(rec, lig, sf, x, tables=None):
    """The 28 unweighted sums of the empirical score [B][28] at poses x [B][N][3]."""
    R, L = rec.lists, lig.lists
    B = x.shape[0]
    rx = _d(rec.xyz)
    zero = x.new_zeros(B)
    f = [zero] * 28
    sig, eps = model.vdw_table()
    ty = np.asarray(lig.vdw_type)
    d = _dist(x, rx)
    f[0] = ((_d(lig.ff.charge)[:, None] * _d(rec.ff.charge)) / d).sum((1, 2)) * COULOMB
    s = _d((sig[ty] * np.array(sf.vdw_sigma_scale)[ty])[:, None] + rec.ff.sigma) * 0.5
    C = _d(np.sqrt((eps[ty] * np.array(sf.vdw_epsilon_scale)[ty])[:, None] * rec.ff.epsilon) * 4.0)
    s2 = (s / d) * (s / d)
    u6 = s2 * s2 * s2
    f[1] = ((u6 * u6 - u6) * C).clamp(-sf.vdw_cutoff, sf.vdw_cutoff).sum((1, 2))
    if tables is not None:
        ligc = {6: 0, 7: 1, 8: 2, 16: 3, 15: 4, 9: 5, 17: 6}
        lc = np.array([ligc.get(int(z), 7) if z >= 2 else -1 for z in L.atomic_numbers])
        rc = np.array([{6: 0, 7: 1, 8: 2}.get(int(z), 3) if z >= 2 else -1 for z in R.atomic_numbers])
        on = _i((lc[:, None] >= 0) & (rc[None] >= 0)).bool()
        t = d / abi.PAIR_BIN_WIDTH
        on = on & (t < abi.PAIR_BINS - 1)
        b = t.detach().floor().clamp(0, abi.PAIR_BINS - 2)
        at = _i((4 * lc[:, None] + rc[None]).clip(0) * abi.PAIR_BINS) + b.long()
        flat, fr = tables.reshape(-1), t - b
        pick = lambda k: flat.index_select(0, k.reshape(-1)).view_as(k)  # noqa: E731
        v = pick(at) * (1 - fr) + pick(at + 1) * fr
        f[27] = torch.where(on, v, torch.zeros_like(v)).sum((1, 2))
    h, rh = np.asarray(L.hydrophobic), np.asarray(R.hydrophobic)
    if len(h) and len(rh) and sf.hydro_dist_max:
        r1 = _d((sig[ty[h]][:, None] + rec.ff.sigma[rh]) * sf.hydro_scale_factor + sf.hydro_dist_min)
        f[24] = -_ramp(d.index_select(1, _i(h)).index_select(2, _i(rh)), r1, r1 + sf.hydro_dist_max).sum((1, 2))
    for k, (a, b) in enumerate(((L.cation, R.anion), (L.anion, R.cation))):
        if len(a) and len(b) and sf.ionic[k][1]:
            f[2 + k] = -_ramp(d.index_select(1, _i(a)).index_select(2, _i(b)), *sf.ionic[k]).sum((1, 2))
    lr = [_rings(x, L.ring5), _rings(x, L.ring6)]
    rr = [_rings(rx[None], R.ring5), _rings(rx[None], R.ring6)]
    for k in range(2):
        if len(L.cation) and sf.picat[k][1]:
            f[4 + k] = -_ramp(_dist(x[:, _i(L.cation)], rr[k][0][0]), *sf.picat[k]).sum((1, 2))
        if len(R.cation) and sf.picat[2 + k][1]:
            f[6 + k] = -_ramp(_dist(lr[k][0], rx[_i(R.cation)]), *sf.picat[2 + k]).sum((1, 2))
    for w in range(2):
        for k in range(4):
            (lc, ln), (rc, rn), p = lr[k // 2], rr[k % 2], list(sf.stack[w][k])
            if lc.shape[1] and rc.shape[1] and p[1]:
                f[8 + 4 * w + k] = _stack(rc, rn, lc, ln, p, 0.0 if w == 0 else 90.0)
    rx1 = rx[None]
    for k in range(8):
        dl = (L, R)[k // 4]
        al = (R, L)[k // 4]
        don = (dl.don_charged, dl.don_neutral)[(k % 4) // 2]
        acc = (al.acc_charged, al.acc_neutral)[k % 2]
        if len(don) and len(acc) and sf.hbond[k][1]:
            dx, ax = (x, rx1) if k < 4 else (rx1, x)
            don = _i(don)
            f[16 + k] = _hbond(dx[:, don[:, 0]], dx[:, don[:, 1]], ax[:, _i(acc)], list(sf.hbond[k]))
    for e, co in enumerate(L.tstrain_coefs):
        quads = np.asarray(L.tstrain_quads[L.tstrain_offsets[e]:L.tstrain_offsets[e + 1]])
        stop = [j for j, q in enumerate(quads) if q[0] == q[1]]
        quads = quads[: stop[0]] if stop else quads
        if len(quads):
            th = _dihedral(x, _i(quads))
            v = sum(float(c) * (1 + torch.cos((k + 1) * th - (math.pi if k % 2 else 0.0))) for k, c in enumerate(co))
            f[25] = f[25] + v.mean(1)
    f[26] = zero - 1.0 / (2.620643 + L.n_rotatable)
    return torch.stack(f, 1)


def _combine64(w, f):
    """S [B] from the 36 weights and the features."""
    term = [f[:, 0], w[11] * f[:, 1], f[:, 2:4] @ w[14:16], f[:, 4:8] @ w[16:20], f[:, 8:12] @ w[20:24],
            f[:, 12:16] @ w[24:28], w[13] * (f[:, 16:24] @ w[28:36]), w[12] * f[:, 24], f[:, 25], f[:, 26]]
    return sum(w[k] * v for k, v in enumerate(term)) + f[:, 27]


def _gb_system(x, q, radius, screen):
    """Generalised-Born + surface energy of one system."""
    rho = radius - 0.09
    sr = rho * screen
    eye = torch.eye(len(x), dtype=torch.bool, device=x.device)
    r = torch.cdist(x, x, compute_mode="donot_use_mm_for_euclid_dist").masked_fill(eye, 1.0)
    U, D = r + sr[None], (r - sr[None]).abs()
    Lb = torch.maximum(rho[:, None], D)
    t = 0.25 * (r - sr[None] ** 2 / r) * (U ** -2 - Lb ** -2) + (1 / Lb - 1 / U) + 0.5 * torch.log(Lb / U) / r
    psi = 0.5 * t.masked_fill(eye | (U < rho[:, None]), 0.0).sum(1) * rho
    born = 1 / (1 / rho - torch.tanh(psi - 0.8 * psi ** 2 + 4.85 * psi ** 3) / radius)
    bp = born[:, None] * born[None]
    f = (r * r + bp * torch.exp(-0.25 * r * r / bp)).sqrt()
    f = torch.where(eye, born[:, None].expand_as(f), f)
    pref = 0.5 * COULOMB * (1.0 - torch.exp(-0.09293963686178248 * f) / 78.5)
    surface = ((radius + 1.4) ** 2 * (radius / born) ** 6 * 0.0678584012906).sum()
    return -(q[:, None] * q[None] / f * pref).sum() + surface


def _gb_properties(lists, n):
    R = [1.5, 1.2, 1.5, 1.5, 1.5, 1.5, 1.7, 1.55, 1.5, 1.5, 1.5, 1.5, 1.5, 1.5, 2.1, 1.85, 1.8, 1.7]
    S = [0.8, 0.85, 0.8, 0.8, 0.8, 0.8, 0.72, 0.79, 0.85, 0.88, 0.8, 0.8, 0.8, 0.8, 0.8, 0.86, 0.96]
    z = np.asarray(lists.atomic_numbers)
    radius = np.array([R[k] if k < 18 else 1.5 for k in z])
    screen = np.array([S[k] if k < 17 else 0.8 for k in z])
    for i, j in lists.all_bonds:  # hydrogens on nitrogen
        for a, b in ((i, j), (j, i)):
            if z[a] == 1 and z[b] == 7:
                radius[a] = 1.3
    return _d(radius), _d(screen)


def _gbsa64(rec, lig, x):
    gr, gl = _gb_properties(rec.lists, rec.n_atoms), _gb_properties(lig.lists, lig.n_atoms)
    rx, rq, lq = _d(rec.xyz), _d(rec.ff.charge), _d(lig.ff.charge)
    pro = _gb_system(rx, rq, *gr)
    cat = [torch.cat(v) for v in ((lq, rq), (gl[0], gr[0]), (gl[1], gr[1]))]
    return torch.stack([_gb_system(torch.cat((p, rx)), *cat) - _gb_system(p, lq, *gl) - pro for p in x])


def _score64(case, seed):
    rec, lig = _complex(case, seed)
    sf = _scoring()[case["which"]]
    xyz = _d(_pocket_poses(lig, case["poses"], seed))
    step = max(1, int(3e7 // (lig.n_atoms * rec.n_atoms)))
    x32 = xyz.float().double()
    f = torch.cat([_features64(rec, lig, sf, x32[i:i + step]) for i in range(0, len(xyz), step)])
    w = _d(abi.sf_weights(sf))
    coef = np.array(sf.coef)
    terms = [f[:, 0], w[11] * f[:, 1], f[:, 2:4] @ w[14:16], f[:, 4:8] @ w[16:20], f[:, 8:12] @ w[20:24],
             f[:, 12:16] @ w[24:28], w[13] * (f[:, 16:24] @ w[28:36]), w[12] * f[:, 24], f[:, 25], f[:, 26],
             _gbsa64(rec, lig, xyz) if coef[10] else 0 * f[:, 0]]
    terms = torch.stack([t * float(c != 0) for t, c in zip(terms, coef)], 1)
    return {"score": terms @ _d(coef), "terms": terms}


def _place64(lig, ref, q):
    """Poses [B][N][3] of the variables q [B][7 + T]: the torsion tree from its reference pose."""
    tree, B = lig.tree, q.shape[0]
    perm = np.asarray(tree.perm)
    c = ref[_i(perm)]
    centre = c.mean(0)
    mine, parent, theta = {}, {}, {}
    for k in range(tree.n_torsions):
        f = int(tree.tors_frag[k])
        mine[f], parent[f], theta[f] = int(tree.tors_mine_atom[k]), int(tree.tors_parent[k]), 7 + k
    u = q[:, 3:7] / q[:, 3:7].norm(dim=1, keepdim=True)
    a, b, cc, d = u.unbind(1)
    rot = torch.stack([a * a + b * b - cc * cc - d * d, 2 * (b * cc - a * d), 2 * (a * cc + b * d),
                       2 * (a * d + b * cc), a * a - b * b + cc * cc - d * d, 2 * (cc * d - a * b),
                       2 * (b * d - a * cc), 2 * (a * b + cc * d), a * a - b * b - cc * cc + d * d], 1).view(B, 3, 3)
    frame = {int(r): (rot, q[:, :3]) for r in tree.roots}
    out = [None] * len(perm)
    for f in [int(r) for r in tree.roots] + [int(t) for t in tree.tors_frag]:
        anchor = centre
        if f in mine:
            pf = parent[f]
            k = theta[f] - 7
            axis = c[mine[f]] - c[int(tree.tors_parent_atom[k])]
            pr, po = frame[pf]
            ax = pr @ (axis / axis.norm())
            org = pr @ (c[mine[f]] - (c[mine[pf]] if pf in mine else centre)) + po
            K = torch.stack([torch.zeros_like(ax[:, 0]), -ax[:, 2], ax[:, 1], ax[:, 2], torch.zeros_like(ax[:, 0]),
                             -ax[:, 0], -ax[:, 1], ax[:, 0], torch.zeros_like(ax[:, 0])], 1).view(B, 3, 3)
            th = q[:, theta[f], None, None]
            turn = torch.eye(3, dtype=q.dtype, device=q.device) + torch.sin(th) * K + (1 - torch.cos(th)) * (K @ K)
            frame[f] = (turn @ pr, org)
            anchor = c[mine[f]]
        fr, fo = frame[f]
        for p in range(int(tree.frag_start[f]), int(tree.frag_end[f])):
            out[p] = fo if p == mine.get(f) else fr @ (c[p] - anchor) + fo
    inv = np.argsort(perm)
    return torch.stack([out[p] for p in inv], 1)


def _train_parts(case, seed):
    """Per complex: receptor, ligand, rows, chunks of rows small enough for autograd."""
    recs, ligs, cplx, A, D, ref, q = _train_set(case, seed)
    for c, (rec, lig) in enumerate(zip(recs, ligs)):
        rows = np.where(cplx == c)[0]
        step = max(1, int(1.6e7 // (lig.n_atoms * rec.n_atoms)))
        yield (rec, lig, _d(ref[rows[0], : lig.n_atoms]), A,
               [(rows[i:i + step], _d(q[rows[i:i + step]])) for i in range(0, len(rows), step)])


def _train64(case, seed):
    sf, box = _scoring()[0], _box(case)
    n = case["complexes"] * case["poses"]
    w = _d(abi.sf_weights(sf)).requires_grad_(True)
    t = _d(abi.smooth_pair_tables(1)).requires_grad_(True)
    score, energy, dq, dw, dt = [], [], [], torch.zeros_like(w), torch.zeros_like(t)
    for rec, lig, ref, _, chunks in _train_parts(case, seed):
        maps = _maps64(rec, box, _types(lig))
        for _, q in chunks:
            q.requires_grad_(True)
            x = _place64(lig, ref, q)
            S = _combine64(w, _features64(rec, lig, sf, x, t))
            e, g = _docking64(maps, box, lig, x)
            gq, gw, gt = torch.autograd.grad(S.sum() + (g * x).sum(), (q, w, t))
            score.append(S.detach())
            energy.append(e)
            dq.append(gq / n)
            dw, dt = dw + gw / n, dt + gt / n
    return {"score": torch.cat(score), "energy": torch.cat(energy), "dq": torch.cat(dq), "dw": dw, "dt": dt}


def _second64(case, seed):
    sf = _scoring()[0]
    w = _d(abi.sf_weights(sf)).requires_grad_(True)
    t = _d(abi.smooth_pair_tables(1)).requires_grad_(True)
    q_all = _train_set(case, seed)[6]
    u_all = _d(np.random.default_rng(seed + 1).normal(size=q_all.shape) * (np.abs(q_all) > 0))
    out = {"g": [], "x": [], "gx": [], "hu": []}
    dw, dt = torch.zeros_like(w), torch.zeros(t.numel(), dtype=torch.float64, device="cuda")
    for rec, lig, ref, A, chunks in _train_parts(case, seed):
        for rows, q in chunks:
            q.requires_grad_(True)
            x = _place64(lig, ref, q)
            S = _combine64(w, _features64(rec, lig, sf, x, t)).sum()
            g, gx = torch.autograd.grad(S, (q, x), create_graph=True)
            hu, gw, gt = torch.autograd.grad((g * u_all[_i(rows)]).sum(), (q, w, t), allow_unused=True)
            out["g"].append(g.detach())
            out["hu"].append(hu)
            for k, v in (("x", x), ("gx", gx)):
                out[k].append(torch.nn.functional.pad(v.detach(), (0, 0, 0, A - v.shape[1])))
            dw, dt = dw + gw, dt + gt.reshape(-1)
    return {**{k: torch.cat(v) for k, v in out.items()}, "dw": dw, "dt": dt}


def exact(case, seed):
    kind = case["kind"]
    if kind == "maps":
        rec, lig = _complex(case, seed)
        rng = np.random.default_rng(seed)
        box = model.make_box(tuple(rng.uniform(-1.0, 1.0, 3)), (case["box"], case["box_y"], case["box_z"]),
                             case["spacing"])
        maps = _maps64(rec, box, _types(lig))
        return {"coulomb": maps[abi.COULOMB_MAP], "vdw": [maps[t] for t in _types(lig)]}
    if kind in ("energy", "energy_host", "engine_start"):
        return _energy64(case, seed)
    if kind == "score":
        return _score64(case, seed)
    if kind == "train":
        return _train64(case, seed)
    if kind == "second":
        return _second64(case, seed)
    return None  # the optimiser and the search amplify rounding over their iterations
