"""A pose's score and terms do not depend on the poses that it is scored with: bit for bit the
same from launches of each number of warps per pose, for poses at either end of the batch."""
import os

import numpy as np
import pytest

from pxdock_gb300 import model, native, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", [0, 1])
@pytest.mark.parametrize("heavy,lig_heavy,rotors", [(25, 8, 0), (400, 31, 2)])
def test_any_batch(which, heavy, lig_heavy, rotors):
    native.load(auto_build=True)
    rec = model.Receptor.from_json(synth.make_receptor(seed=2, n_heavy=heavy, cube=16.0, cavity=4.0, n_rotors=rotors))
    lig = model.Ligand.from_json(synth.make_ligand(seed=1, n_heavy=lig_heavy, n_rot=min(4, lig_heavy // 6)))
    sf = model.load_scoring_function(os.path.join(os.path.dirname(model.__file__), "data", "scoring_function.json"))
    n = 153 if which else 700  # 16, 8 and 4 warps: up to 152, 304 and more poses on 152 SMs
    rng = np.random.default_rng(heavy)
    xyz = lig.poses[0] + rng.normal(scale=0.4, size=(n, lig.n_atoms, 3))
    tors = rng.uniform(-3, 3, size=(n, rotors))
    with native.Context(0) as ctx:
        ctx.set_receptor(rec)
        ctx.set_scoring_function(which, sf[which])
        lid = ctx.add_ligand(lig)
        score, terms = ctx.score(which, lid, xyz, tors)
        for a, b in ((0, 1), (n - 1, n), (3, 155), (n - 290, n), (0, 400)):
            if 0 <= a < b <= n:
                s, t = ctx.score(which, lid, xyz[a:b], tors[a:b])
                np.testing.assert_array_equal(s, score[a:b])
                np.testing.assert_array_equal(t, terms[a:b])
    assert np.isfinite(score).all()
