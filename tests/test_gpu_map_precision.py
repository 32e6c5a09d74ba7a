"""The Coulomb energies of a built map (FP32 record + remainder) against sums in extended
precision, with all atoms near the box, with one 190 A away (the same coordinate grids,
coarser), and with one 900 A away (the wide split).

Charges are multiples of 2^-12 and coordinates of 2^-40 A about a box centred at 0, so that
neither is rounded on its way. What is left: a term q/r in FP32 triples (2^-55 of itself, 2^-51
allowed), their FP64 total, and its storage as two floats (2^-49 of it, 2^-48 allowed)."""
import ctypes as C

import numpy as np
import pytest

from pxdock_gb300 import abi, model, native, synth

pytestmark = pytest.mark.gpu
COULOMB = 332.0637141491396


@pytest.mark.parametrize("far", [None, (188.0, -31.0, 20.0), (900.0, -700.0, 650.0)])
def test_coulomb_energies(far):
    native.load(auto_build=True)
    js = synth.make_receptor(seed=5, n_heavy=300, cube=16.0, cavity=3.0)
    if far:
        js["xyz"][0] = list(far)
    rec = model.Receptor.from_json(js)
    rec.xyz[:] = np.round(rec.xyz * 2.0 ** 40) / 2.0 ** 40
    rec.ff.charge[:] = np.round(rec.ff.charge * 4096) / 4096
    box = model.make_box((0.0, 0.0, 0.0), (9.0, 7.5, 6.0), 0.375)
    with native.Context(0) as ctx:
        ctx.set_receptor(rec)
        ctx.build_grid(box, [3])
        P = int(np.prod(list(box.npoints)))
        got = np.zeros((P, 4))
        ctx._check(ctx.lib.pxd_grid_read_map64(ctx.h, abi.COULOMB_MAP, got.ctypes.data_as(C.POINTER(C.c_double))))
    axes = [box.init_xyz[d] + box.spacing * np.arange(box.npoints[d]) for d in range(3)]
    pts = np.stack(np.meshgrid(*axes, indexing="ij"), -1).reshape(-1, 3)
    at = np.random.default_rng(0).choice(P, 600, replace=False)
    d = rec.xyz[None].astype(np.longdouble) - pts[at, None].astype(np.longdouble)
    r = np.sqrt((d * d).sum(-1))
    assert r.min() > 0.01
    q = rec.ff.charge.astype(np.longdouble) / r * np.longdouble(COULOMB)
    ref = q.sum(1)
    err = np.abs(got[at, 0].astype(np.longdouble) - ref)
    assert np.all(err <= 2.0 ** -51 * np.abs(q).sum(1) + 2.0 ** -48 * np.abs(ref)), float(err.max())
    # the gradient: FP32 roundings of sums in pairs
    g = (q[..., None] * d / (r * r)[..., None]).sum(1)
    np.testing.assert_allclose(got[at, 1:], g.astype(np.float64), rtol=2.0 ** -23, atol=1e-9)


@pytest.mark.parametrize("where", [1e16, 1e22])
def test_atom_out_of_fp32(where):
    """An atom so far that FP32 does not hold its squared distance adds next to nothing: the maps
    are those of the receptor with its charge and well depth at zero (q / r <= 2e-14 kcal/mol)."""
    native.load(auto_build=True)
    js = synth.make_receptor(seed=5, n_heavy=120, cube=14.0, cavity=3.0)
    js["xyz"][0] = [where, -0.5 * where, 0.25 * where]
    box = model.make_box((0.0, 0.0, 0.0), (5.0, 4.0, 3.0), 0.375)
    maps = []
    for off in (False, True):
        rec = model.Receptor.from_json(js)
        if off:
            rec.ff.charge[0] = rec.ff.epsilon[0] = 0.0
        with native.Context(0) as ctx:
            ctx.set_receptor(rec)
            ctx.build_grid(box, [3, 7])
            maps.append([ctx.read_map(m) for m in (abi.COULOMB_MAP, 3, 7)])
    for got, want in zip(*maps):
        assert np.isfinite(want).all()
        np.testing.assert_allclose(got, want, rtol=2.0 ** -23, atol=1e-12)
