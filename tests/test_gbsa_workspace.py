"""The GB/SA term's device memory for receptors of several thousand atoms, on a runtime of host
memory: batches of poses within 64 MB, and smaller ones, not an error, where that is not to be
had."""
import os

import numpy as np
import pytest

import fake_runtime
from pxdock_gb300 import model, native, synth


@pytest.mark.parametrize("heavy,rotors,poses", [(300, 0, 600), (4000, 0, 600), (4000, 3, 600)])
def test_batches(tmp_path, heavy, rotors, poses):
    cube = 26.0 * (heavy / 1500.0) ** (1 / 3)
    rec = model.Receptor.from_json(synth.make_receptor(seed=3, n_heavy=heavy, cube=cube, n_rotors=rotors))
    lig = model.Ligand.from_json(synth.make_ligand(seed=1, n_heavy=9, n_rot=2))
    sf = model.load_scoring_function(os.path.join(os.path.dirname(model.__file__), "data", "scoring_function.json"))[1]
    with fake_runtime.loaded(tmp_path) as fake, native.Context(0) as ctx:
        ctx.set_scoring_function(1, sf)
        ctx.set_receptor(rec)
        lid = ctx.add_ligand(lig)
        xyz, tors = np.repeat(lig.poses[:1], poses, axis=0), np.zeros((poses, rec.n_rotors))
        ctx.score(1, lid, xyz[:1], tors[:1])  # the ligand table, once
        fake.reset()
        ctx.score(1, lid, xyz, tors)
        last = fake.lib.fake_mallocs() - 1  # the last batch's workspace
        counts = []
        for fail in (-1, last):
            fake.reset()
            fake.lib.fake_fail_at(fail)
            ctx.score(1, lid, xyz, tors)
            fake.lib.fake_fail_at(-1)
            assert fake.lib.fake_largest() <= (64 << 20) + (1 << 20)  # and what the batch shares
            systems = [g[0] for name, g in fake.launches() if "gb_total" in name]
            assert sum(systems) == 2 * poses + (poses if rotors else len(systems))
            counts.append(len(systems))
        assert counts[1] > counts[0]
        assert fake.violations == ""
