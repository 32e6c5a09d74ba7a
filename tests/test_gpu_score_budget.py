"""Scoring launches run under a register budget chosen by their pose count and their block's
shared memory: the same poses get the same energies and gradients, bit for bit, from a launch of
a few and from one that fills the device, for ligands of each budget."""
import numpy as np
import pytest

from pxdock_gb300 import model, native, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heavy,rot", [(9, 1), (30, 4), (37, 5)])
def test_budgets_agree(heavy, rot):
    torch = pytest.importorskip("torch")
    native.load(auto_build=True)
    n = 16 * torch.cuda.get_device_properties(0).multi_processor_count + 1
    rec = model.Receptor.from_json(synth.make_receptor(seed=2, n_heavy=60, cube=16.0, cavity=5.0, n_rotors=1))
    lig = model.Ligand.from_json(synth.make_ligand(seed=1, n_heavy=heavy, n_rot=rot))
    ctx = native.Context(0)
    ctx.set_receptor(rec)
    ctx.build_grid(model.make_box((0.0, 0.0, 0.0), (16.0, 16.0, 16.0), 0.5), sorted(set(int(t) for t in lig.vdw_type)))
    lid = ctx.add_ligand(lig)
    rng = np.random.default_rng(heavy)
    x = lig.poses[0] + rng.normal(scale=0.2, size=(n, lig.n_atoms, 3))
    tors = rng.uniform(-3, 3, size=(n, 1))
    many, few = ctx.score_grad(lid, x, tors), ctx.score_grad(lid, x[-7:], tors[-7:])
    for a, b in zip(many, few):
        np.testing.assert_array_equal(np.asarray(a)[-7:], np.asarray(b))
    ctx.close()
