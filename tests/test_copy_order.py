"""What a context uploads is on the device before a kernel reads it: the context's stream does
not wait for the legacy stream, so no copy or memset may be left pending there. On a runtime of
host memory, over the calls that install something and the first launches after each."""
import os

import numpy as np
import pytest

import fake_runtime
from pxdock_gb300 import abi, model, native, synth


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    with fake_runtime.loaded(tmp_path_factory.mktemp("fake")) as f:
        yield f


def test_uploads_precede_launches(fake):
    rec = model.Receptor.from_json(synth.make_receptor(seed=0, n_heavy=60, cube=16.0, cavity=4.0, n_rotors=1))
    lig = model.Ligand.from_json(synth.make_ligand(seed=1, n_heavy=9, n_rot=2))
    sf = model.load_scoring_function(os.path.join(os.path.dirname(model.__file__), "data", "scoring_function.json"))
    types = sorted(set(int(t) for t in lig.vdw_type))
    box = model.make_box((0.0, 0.0, 0.0), (6.0, 6.0, 6.0), 0.5)
    records = np.zeros((int(np.prod(list(box.npoints))), 4), np.float32)
    fake.reset()
    with native.Context(0) as ctx:
        for which in (0, 1):
            ctx.set_scoring_function(which, sf[which])
        for _ in range(2):  # the first receptor, and another in its place
            ctx.set_receptor(rec)
            ctx.set_scoring_function(0, sf[0])
            lid = ctx.add_ligand(lig)
            ctx.score_grad(lid, lig.poses[:1], np.zeros((1, 1)))
            ctx.score(1, lid, lig.poses[:1], np.zeros((1, 1)))
            ctx.build_grid(box, types)
            ctx.score_grad(lid, lig.poses[:1], np.zeros((1, 1)))
            ctx.write_map(box, abi.COULOMB_MAP, records)
            ctx.score_grad(lid, lig.poses[:1], np.zeros((1, 1)))
            ctx.write_map(model.make_box((0.0, 0.0, 0.0), (6.5, 6.0, 6.0), 0.5), types[0],
                          np.zeros((int(np.prod(list(model.make_box((0.0, 0.0, 0.0), (6.5, 6.0, 6.0), 0.5).npoints))), 4),
                                   np.float32))
            ctx.lbfgs(native.lbfgs_params(max_iter=1, history=2), lid, lig.poses[:1], np.zeros((1, 1)))
    assert len(fake.launches()) > 10
    assert fake.violations == ""
