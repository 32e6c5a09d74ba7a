"""Receptors with 32 and more movable atoms, some of them listed by their rotor more than once: the
torsion gradient stays the derivative of the energy, which counts an atom as often as it is
listed."""
import numpy as np
import pytest

from pxdock_gb300 import model, native, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("repeat", [1, 2, 3])
def test_torsion_gradient(repeat):
    native.load(auto_build=True)
    js = synth.make_receptor(seed=4, n_heavy=300, cube=16.0, cavity=4.0, n_rotors=8)
    rec = model.Receptor.from_json(js)
    lig = model.Ligand.from_json(synth.make_ligand(seed=1, n_heavy=9, n_rot=2))
    rng = np.random.default_rng(0)
    # more movable atoms for the first rotor (any atoms away from its axis), then the repeats
    own = set(a for g in rec.rotor_groups for a in g) | set(rec.rotor_axis.ravel().tolist())
    far = [a for a in np.argsort(-np.linalg.norm(rec.xyz - rec.xyz[rec.rotor_axis[0, 1]], axis=1)) if a not in own][:30]
    groups = [list(g) for g in rec.rotor_groups]
    groups[0] += [int(a) for a in far]
    groups[1] = groups[1] * repeat
    groups[2] = groups[2] * repeat
    rec = model.Receptor(rec.xyz, rec.ff, rotor_axis=rec.rotor_axis, rotor_atoms=groups, raw=js)
    box = model.make_box((0.0, 0.0, 0.0), (9.0, 9.0, 9.0), 0.5)
    xyz = np.repeat(lig.poses[:1] - lig.poses[:1].mean(axis=1, keepdims=True), 3, axis=0)
    with native.Context(0) as ctx:
        ctx.set_receptor(rec)
        ctx.build_grid(box, sorted(set(int(t) for t in lig.vdw_type)))
        lid = ctx.add_ligand(lig)
        t0 = rng.uniform(-0.3, 0.3, size=rec.n_rotors)
        h = 1e-3
        _, gx, gt = ctx.score_grad(lid, xyz[:1], t0[None])
        for r in (1, 2):
            t = np.repeat(t0[None], 2, axis=0)
            t[0, r] -= h
            t[1, r] += h
            e, _, _ = ctx.score_grad(lid, xyz[:2], t)
            slope = (e[1] - e[0]) / (t[1, r].astype(np.float32).astype(float) - t[0, r].astype(np.float32).astype(float))
            assert abs(gt[0, r] - slope) <= 1e-2 + 1e-3 * abs(slope), (r, gt[0, r], slope)
