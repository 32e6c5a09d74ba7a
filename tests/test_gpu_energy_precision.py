"""The reported energy where terms are large. Intra-ligand energies of clashing poses against
sums in extended precision, map lookups of atoms outside the box, and an atom at infinity."""
import numpy as np
import pytest

import oracle
from pxdock_gb300 import model, native, synth

pytestmark = pytest.mark.gpu
COULOMB = 332.0637141491396


def strip(ff, keep_pairs):
    for names in (("bonds", "bond_k", "bond_length"), ("angles", "angle_k", "angle_radian")):
        for n in names:
            setattr(ff, n, getattr(ff, n)[:0])
    ff.impropers = tuple(a[:0] for a in ff.impropers)
    ff.propers = tuple(a[:0] for a in ff.propers)
    if not keep_pairs:
        ff.pairs14, ff.pairs = ff.pairs14[:0], ff.pairs[:0]


def test_clashing_pairs():
    """Non-bonded terms alone, atoms drawn into a small ball: the energy is a few terms of 1e7 to
    1e17 kcal/mol, each FP64 (a dozen operations), summed in FP64: 1e-14 of the sum of sizes;
    FP32 terms of up to 1 kcal/mol leave 1e-6 of themselves."""
    native.load(auto_build=True)
    lig = model.Ligand.from_json(synth.make_ligand(seed=2, n_heavy=12, n_rot=2))
    strip(lig.ff, True)
    rng = np.random.default_rng(0)
    base = lig.poses[0] - lig.poses[0].mean(axis=0)
    xyz = np.stack([base * s + rng.normal(scale=0.05, size=base.shape) for s in np.linspace(0.08, 0.3, 64)])
    xyz = xyz.astype(np.float32).astype(np.float64)
    with native.Context(0) as ctx:
        js = synth.make_receptor(seed=0, n_heavy=20, cube=14.0, cavity=2.0)
        js["xyz"] = [[a + 1e5 for a in x] for x in js["xyz"]]
        rec = model.Receptor.from_json(js)
        rec.ff.charge[:] = 0.0
        ctx.set_receptor(rec)
        e, _, _ = ctx.score_grad(ctx.add_ligand(lig), xyz)
        const, _, _ = ctx.score_grad(0, (base + 1e4)[None].astype(np.float32))  # the receptor's own, and FP32 terms
    ff, big = lig.ff, np.longdouble
    ref, size = np.zeros(len(xyz), big), np.zeros(len(xyz), big)
    own, at = big(0), (base + 1e4).astype(np.float32).astype(big)[None]
    for pairs, sc, sv in ((ff.pairs14, 0.833333333, 0.5), (ff.pairs, 1.0, 1.0)):
        i, j = np.asarray(pairs).T
        A = big(COULOMB) * ff.charge[i].astype(big) * ff.charge[j] * sc
        C, S2 = 4 * np.sqrt((ff.epsilon[i] * ff.epsilon[j]).astype(big)) * sv, ((ff.sigma[i] + ff.sigma[j]).astype(big) / 2) ** 2
        for x, out in ((xyz.astype(big), ref), (at, None)):
            r2 = ((x[:, j] - x[:, i]) ** 2).sum(-1)
            u6 = (S2 / r2) ** 3
            t = A / np.sqrt(r2) + C * (u6 * u6 - u6)
            if out is None:
                own += t.sum()
            else:
                out += t.sum(1)
                size += np.abs(t).sum(1)
    err = np.abs(e - (ref + (const[0] - own)))
    assert float(np.median(size)) > 1e6
    assert np.all(err <= 1e-4 + 1e-14 * size), float((err / size).max())


def test_far_outside_and_infinite():
    """Map lookups alone. Outside the box the penalty is FP64 as the port's; an atom at infinity
    gives an infinite energy, and one that is not a number the lookup on a face."""
    native.load(auto_build=True)
    lig = model.Ligand.from_json(synth.make_ligand(seed=1, n_heavy=9, n_rot=1))
    strip(lig.ff, False)
    rec = model.Receptor.from_json(synth.make_receptor(seed=0, n_heavy=120, cube=16.0, cavity=5.0))
    box = model.make_box((0.1, -0.2, 0.05), (9.0, 8.2, 7.0), 0.375)
    port = oracle.PortSystem(rec, lig)
    types = sorted(set(int(t) for t in lig.vdw_type))
    port.build_grid(box, types, nthreads=4)
    port.set_slope(1e6)
    base = lig.poses[0] - lig.poses[0].mean(axis=0)
    out = np.stack([base + d for d in (40.0, -300.0, 1e5, 1e12)]).astype(np.float32).astype(np.float64)
    bad = np.repeat(base[None], 3, axis=0)
    bad[0, 2, 0], bad[1, 3, 2], bad[2, 4, 1] = np.inf, -np.inf, np.nan
    with native.Context(0) as ctx:
        ctx.set_receptor(rec)
        ctx.build_grid(box, types)
        ctx.set_slope(1e6)
        lid = ctx.add_ligand(lig)
        e, _, _ = ctx.score_grad(lid, out)
        eb, _, _ = ctx.score_grad(lid, bad)
    ref = np.array([port.score_grad([], x)[0] for x in out])
    np.testing.assert_allclose(e, ref, rtol=4e-15)  # 17 atoms added up in another order, a few roundings each
    assert np.isposinf(eb[:2]).all() and np.isfinite(eb[2])
