"""A receptor atom whose sigma or well depth is not a number is a kind of its own: it spoils the
vdW maps and scores that it takes part in, and is not taken for another atom's kind. The Coulomb
map stays."""
import os

import numpy as np
import pytest

from pxdock_gb300 import abi, model, native, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", [True, False])
@pytest.mark.parametrize("what", ["sigma", "epsilon"])
def test_nan_parameter(first, what):
    native.load(auto_build=True)
    rec = model.Receptor.from_json(synth.make_receptor(seed=5, n_heavy=60, cube=14.0, cavity=3.0))
    lig = model.Ligand.from_json(synth.make_ligand(seed=1, n_heavy=9, n_rot=2))
    sf = model.load_scoring_function(os.path.join(os.path.dirname(model.__file__), "data", "scoring_function.json"))[0]
    box = model.make_box((0.0, 0.0, 0.0), (4.0, 3.0, 3.0), 0.5)
    heavy = np.where(rec.ff.epsilon > 0)[0]
    out = []
    for bad in (False, True):
        if bad:
            getattr(rec.ff, what)[heavy[0 if first else -1]] = np.nan
        with native.Context(0) as ctx:
            ctx.set_scoring_function(0, sf)
            ctx.set_receptor(rec)
            ctx.build_grid(box, [3])
            with native.Context(0) as plain:  # the score reads no maps, whose types are not the ligand's here
                plain.set_scoring_function(0, sf)
                plain.set_receptor(rec)
                score, terms = plain.score(0, plain.add_ligand(lig), lig.poses[:1])
            out.append((ctx.read_map(abi.COULOMB_MAP), ctx.read_map(3), terms[0]))
    (coulomb, vdw, terms), (coulomb_n, vdw_n, terms_n) = out
    np.testing.assert_allclose(coulomb_n, coulomb, rtol=2.0 ** -22, atol=1e-9)
    # clamped to the records' range, as every sum that is not a number was
    assert np.all(vdw_n == np.float32(-1e30))
    assert np.all(np.abs(vdw) <= 1e30) and not np.any(vdw[:, 0] == np.float32(-1e30))
    # each of its pairs in a score is clamped to the cutoff
    v = abi.TERM_NAMES.index("InteractionVDW_Energy")
    assert terms_n[v] < terms[v] - 0.5 * sf.vdw_scale * sf.vdw_cutoff * lig.n_atoms
    np.testing.assert_array_equal(np.delete(terms_n, v), np.delete(terms, v))
