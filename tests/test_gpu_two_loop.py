"""The optimiser's two-loop recursion at variable counts on both sides of its register rows (32
elements each, two to eight), against the FP64 port.

Four iterations with three kept pairs from a slightly displaced pose. A change of 1e-6 A of the
start, an FP32 coordinate's rounding, moves the port's own descent by up to 2e-5 A and 1e-5 of
the energy; fifty times that is allowed, and ten times for the energy."""
import numpy as np
import pytest

import oracle
from pxdock_gb300 import abi, model, native, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heavy,seed,atoms", [(7, 2, 13), (9, 1, 21), (10, 2, 23), (16, 2, 32), (24, 1, 42), (25, 2, 45),
                                              (28, 2, 53), (28, 3, 54), (30, 1, 68), (37, 1, 81)])
def test_rows(heavy, seed, atoms):
    native.load(auto_build=True)
    rec = model.Receptor.from_json(synth.make_receptor(seed=2, n_heavy=40, cube=16.0, cavity=5.0, n_rotors=1))
    lig = model.Ligand.from_json(synth.make_ligand(seed=seed, n_heavy=heavy, n_rot=min(3, heavy // 6)))
    assert lig.n_atoms == atoms and rec.n_rotors == 1  # 3 atoms + 1 variables
    ctx = native.Context(0)
    ctx.set_receptor(rec)
    lid = ctx.add_ligand(lig)
    port = oracle.PortSystem(rec, lig)
    rng = np.random.default_rng(heavy)
    x0 = (lig.poses[0] + rng.normal(scale=0.02, size=(3, lig.n_atoms, 3))).astype(np.float32).astype(np.float64)
    out = ctx.lbfgs(native.lbfgs_params(max_iter=4, history=3), lid, x0)
    for k in range(3):
        want = port.lbfgs(abi.lbfgs_params(max_iter=4, history=3), np.zeros(rec.n_rotors), x0[k])
        assert abs(out["energy"][k] - want["energy"]) <= 1e-3 + 1e-4 * abs(want["energy"])
        np.testing.assert_allclose(out["xyz"][k], want["xyz"], rtol=0, atol=1e-3)
    ctx.close()


def test_register_budgets_agree():
    """A launch's register budget follows its pose count: the same poses end bit for bit the same
    in launches on both sides of each limit."""
    torch = pytest.importorskip("torch")
    native.load(auto_build=True)
    n_sm = torch.cuda.get_device_properties(0).multi_processor_count
    rec = model.Receptor.from_json(synth.make_receptor(seed=2, n_heavy=60, cube=16.0, cavity=5.0, n_rotors=1))
    lig = model.Ligand.from_json(synth.make_ligand(seed=1, n_heavy=9, n_rot=1))
    ctx = native.Context(0)
    ctx.set_receptor(rec)
    ctx.build_grid(model.make_box((0.0, 0.0, 0.0), (12.0, 12.0, 12.0), 0.5), sorted(set(int(t) for t in lig.vdw_type)))
    lid = ctx.add_ligand(lig)
    x = lig.poses[0] + np.random.default_rng(0).normal(scale=0.1, size=(12 * n_sm + 1, lig.n_atoms, 3))
    p = native.lbfgs_params(max_iter=30, history=8)
    want = ctx.lbfgs(p, lid, x[:5])
    for n in (8 * n_sm, 8 * n_sm + 1, 12 * n_sm, 12 * n_sm + 1):
        got = ctx.lbfgs(p, lid, x[:n])
        for key in ("energy", "nevals", "status", "xyz", "torsions"):
            np.testing.assert_array_equal(got[key][:5], want[key], err_msg=key)
    ctx.close()
