"""The reported energy (FP32 pairs) against the FP64 port at the places where its branches
meet: atoms on and next to grid points and box faces, atoms outside the box, coincident and
nearly coincident atoms, atoms flung apart, and ligands of one atom to several rounds."""
import os

import numpy as np
import pytest

import oracle
from pxdock_gb300 import model, native, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[(8, 0), (12, 2), (30, 4)])
def system(request):
    native.load(auto_build=True)
    heavy, rot = request.param
    rec = model.Receptor.from_json(synth.make_receptor(seed=0, n_heavy=300, cube=16.0, cavity=5.0))
    lig = model.Ligand.from_json(synth.make_ligand(seed=2, n_heavy=heavy, n_rot=rot))
    box = model.make_box((0.1, -0.2, 0.05), (9.0, 8.2, 7.0), 0.375)
    types = sorted(set(int(t) for t in lig.vdw_type))
    ctx = native.Context(0)
    ctx.set_receptor(rec)
    ctx.build_grid(box, types)
    ctx.set_slope(1e6)
    lid = ctx.add_ligand(lig)
    port = oracle.PortSystem(rec, lig)
    port.build_grid(box, types, nthreads=os.cpu_count() or 1)
    port.set_slope(1e6)
    yield ctx, lid, lig, box, port
    ctx.close()


def places(lig, box, rng):
    lo = np.array(box.init_xyz)
    n = np.array(box.npoints)
    base = lig.poses[0] - lig.poses[0].mean(axis=0)
    out = {"inside": base + lo + 0.5 * (n - 1) * box.spacing}
    for name, node in (("node", n // 2), ("low face", n * 0), ("high face", n - 1)):
        for eps in (0.0, 3e-8, -3e-8, 1e-5, -1e-5):
            out["%s %g" % (name, eps)] = base - base[0] + lo + node * box.spacing + eps
    out["outside"] = base + lo - 40.0
    out["far"] = base + 1e5
    x = out["inside"].copy()
    x[3] = x[0] + 1e-3
    out["clash"] = x
    x = out["inside"].copy()
    x[3] = x[0] + np.array([0.02, 0.03, 0.05])
    out["near clash"] = x
    x = out["inside"].copy()
    x[2] += 3e9
    out["flung atom"] = x
    for k in range(4):
        out["random %d" % k] = out["inside"] + rng.normal(scale=0.5, size=base.shape)
    return out


def test_energy_at_the_edges(system):
    ctx, lid, lig, box, port = system
    cases = places(lig, box, np.random.default_rng(1))
    xyz = np.stack(list(cases.values())).astype(np.float32).astype(np.float64)
    e, _, _ = ctx.score_grad(lid, xyz)
    for name, x, got in zip(cases, xyz, e):
        ref = port.score_grad([], x)[0]
        # FP32 angles move a term by k |theta - theta0| 1e-7 (1e-5 kcal/mol each, some dozens of
        # terms); the rest is FP32 pairs or FP64, 1e-12 of itself
        assert abs(got - ref) <= 1e-3 + 1e-9 * abs(ref), name
