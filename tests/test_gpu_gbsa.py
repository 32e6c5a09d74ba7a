"""The batched GB/SA term against the FP64 port: batches with and without receptor rotors
(one receptor conformation per call, or one per pose), atom counts off the kernels' tile and
lane sizes, and a batch longer than one set of launches."""
import os

import numpy as np
import pytest

import oracle
from pxdock_gb300 import abi, model, native, synth

pytestmark = pytest.mark.gpu
GBSA = abi.TERM_NAMES.index("Gbsa_Com_Energy-Gbsa_Lig_Energy-Gbsa_Pro_Energy")


@pytest.mark.parametrize("heavy,lig_heavy,rotors,n", [(40, 8, 0, 1), (40, 8, 0, 513), (90, 12, 3, 5), (230, 24, 0, 3),
                                                      (230, 24, 2, 2)])
def test_batched_gbsa(heavy, lig_heavy, rotors, n):
    native.load(auto_build=True)
    rec = model.Receptor.from_json(synth.make_receptor(seed=3, n_heavy=heavy, cube=16.0, cavity=4.0, n_rotors=rotors))
    lig = model.Ligand.from_json(synth.make_ligand(seed=1, n_heavy=lig_heavy, n_rot=min(3, lig_heavy // 4)))
    sf = model.load_scoring_function(os.path.join(os.path.dirname(model.__file__), "data", "scoring_function.json"))[1]
    ctx = native.Context(0)
    ctx.set_receptor(rec)
    ctx.set_scoring_function(1, sf)
    lid = ctx.add_ligand(lig)
    port = oracle.PortSystem(rec, lig)
    rng = np.random.default_rng(n)
    poses = lig.poses[0][None] + rng.normal(scale=0.3, size=(n, lig.n_atoms, 3))
    tors = rng.uniform(-3, 3, size=(n, rec.n_rotors))
    score, terms = ctx.score(1, lid, poses, tors)
    for p in sorted({0, n // 2, n - 1}):
        rx = port.receptor_apply(tors[p]) if rotors else rec.xyz
        ref, tref = port.score(sf, rx, poses[p])
        # FP64 on both sides: the difference of energies of some 1e4 kcal/mol, each a sum of
        # ~1e5 terms rounded at 1e-16
        assert abs(terms[p][GBSA] - tref[10]) <= 1e-7
        delta, parts = ctx.gbsa(lid, poses[p], tors[p])
        assert delta == terms[p][GBSA]  # a batch gives each pose what a call of its own gives
        assert delta == parts[0] - parts[1] - parts[2]
    ctx.close()
