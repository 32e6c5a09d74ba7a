"""The search's descent (the two-loop recursion with passes loaded two ahead, whole rows of 32
elements, FP32 coefficients) where it is not yet chaotic: the start's relaxation of walker 0,
which makes no moves, against the FP64 port's. Variable counts on both sides of the rows, two
to eight iterations with three kept pairs (counts of one to three, then the ring's wraps) and
with eight; a walker alone (its block's warps as a team) and one of many (a warp each); without
maps, and with maps and movable receptor atoms.

A change of 1e-6 A of the start, an FP32 coordinate's rounding, moves the port's own descent of up
to eight iterations by at most 5e-6 A and 7e-5 of the energy, of moves of 0.01 to 0.8 A; fifty
times the first and ten times the second are allowed."""
import os

import numpy as np
import pytest

import oracle
from pxdock_gb300 import abi, model, native, synth

pytestmark = pytest.mark.gpu
SF = os.path.join(os.path.dirname(model.__file__), "data", "scoring_function.json")


@pytest.mark.parametrize("maps", [False, True])
@pytest.mark.parametrize("heavy,seed", [(7, 2), (9, 1), (10, 2), (16, 2), (24, 1), (25, 2), (28, 2), (28, 3), (30, 1),
                                        (37, 1)])
def test_descent(heavy, seed, maps):
    native.load(auto_build=True)
    rec = model.Receptor.from_json(synth.make_receptor(seed=2, n_heavy=40, cube=16.0, cavity=5.0, n_rotors=1))
    lig = model.Ligand.from_json(synth.make_ligand(seed=seed, n_heavy=heavy, n_rot=min(3, heavy // 6)))
    sf = model.load_scoring_function(SF)[0]
    port = oracle.PortSystem(rec, lig)
    x0 = lig.poses[0] + np.random.default_rng(heavy).normal(scale=0.02, size=lig.poses[0].shape)
    x0 = x0.astype(np.float32).astype(np.float64)
    with native.Context(0) as ctx:
        ctx.set_receptor(rec)
        ctx.set_scoring_function(0, sf)
        if maps:
            box = model.make_box((0.0, 0.0, 0.0), (22.0, 22.0, 22.0), 0.5)
            types = sorted(set(int(t) for t in lig.vdw_type))
            ctx.build_grid(box, types)
            port.build_grid(box, types, nthreads=os.cpu_count() or 1)
        lid = ctx.add_ligand(lig)
        for history, steps in ((3, 2), (3, 3), (3, 4), (3, 5), (3, 6), (3, 8), (8, 7)):
            want = port.lbfgs(abi.lbfgs_params(max_iter=steps, history=history), np.zeros(rec.n_rotors), x0)
            for walkers in (1, 200):
                p = native.mc_params([-20.0] * 3, [20.0] * 3, max_nsteps=0, full_nsteps=steps, lbfgs=dict(history=history))
                out = ctx.mc_search(p, lid, np.repeat(x0[None], walkers, axis=0), np.zeros(walkers, np.int32))
                for k in {0, walkers - 1}:
                    name = (history, steps, walkers)
                    np.testing.assert_allclose(out["xyz"][k], want["xyz"], rtol=0, atol=2.5e-4, err_msg=str(name))
                    assert abs(out["energy"][k] - want["energy"]) <= 7e-4 * abs(want["energy"]) + 1e-3, name
