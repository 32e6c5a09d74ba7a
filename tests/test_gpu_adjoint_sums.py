"""The sums over poses of the adjoint launch - weight gradient from the blocks' weighted
features, pair-table gradient from its partials - at pose counts on both sides of a warp's, a
block's and the reductions' sizes, for value (adjoint) and tangent launches.

The weight gradient is FP64 throughout: it equals the one of the summed features within 1e-12
of the sum of magnitudes. A table bin is an FP32 sum of up to a few thousand terms of one sign
in a partial: 1e-4 of the largest bin against the sum of launches of eight poses."""
import os

import numpy as np
import pytest

from pxdock_gb300 import abi, model, native, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 9, 300, 4871])
@pytest.mark.parametrize("tangent", [False, True])
def test_sums_over_poses(n, tangent):
    torch = pytest.importorskip("torch")
    native.load(auto_build=True)
    rec = model.Receptor.from_json(synth.make_receptor(seed=0, n_heavy=120, cube=16.0, cavity=4.0, n_rotors=1))
    lig = model.Ligand.from_json(synth.make_ligand(seed=1, n_heavy=9, n_rot=2))
    sf = model.load_scoring_function(os.path.join(os.path.dirname(model.__file__), "data", "scoring_function.json"))[0]
    ctx = native.Context(0)
    ctx.set_receptor(rec)
    ctx.set_scoring_function(0, sf)
    lid = ctx.add_ligand(lig)
    rng = np.random.default_rng(n)
    A, dev = lig.n_atoms, torch.device("cuda", 0)
    cuda = lambda a, t: torch.tensor(a, dtype=t, device=dev)
    x = cuda(lig.poses[0] + rng.normal(scale=0.3, size=(n, A, 3)), torch.float32)
    xd = cuda(rng.normal(size=(n, A, 3)), torch.float32)
    tors = cuda(rng.uniform(-3, 3, size=(n, 1)), torch.float32)
    g = cuda(rng.uniform(0.5, 1.5, size=n), torch.float64)
    wn = abi.sf_weights(sf) * rng.uniform(0.5, 1.5, size=abi.NUM_SF_WEIGHTS)
    w, tab = cuda(wn, torch.float64), cuda(abi.smooth_pair_tables(1), torch.float32)
    ids, zero = cuda(np.full(n, lid), torch.int32), cuda(np.zeros(n), torch.int32)
    feats = torch.zeros((n, abi.NUM_SCORE_FEATURES), dtype=torch.float64, device=dev)
    gx = torch.empty_like(x)
    p = lambda t, a=0: t[a:].data_ptr()

    def launch(a, b):
        dw = torch.zeros(abi.NUM_SF_WEIGHTS, dtype=torch.float64, device=dev)
        dt = torch.zeros(abi.PAIR_TYPES * abi.PAIR_BINS, dtype=torch.float64, device=dev)
        if tangent:
            native.score_hvp_multi_dev([ctx], 0, b - a, A, p(zero, a), p(ids, a), p(x, a), p(xd, a), p(tors, a), p(w),
                                       p(tab), p(g, a), p(feats, a), p(gx, a), p(dw), p(dt), None)
        else:
            native.score_adjoint_multi_dev([ctx], 0, b - a, A, p(zero, a), p(ids, a), p(x, a), p(tors, a), p(w), p(tab),
                                           p(g, a), None, p(feats, a), p(gx, a), p(dw), p(dt), None)
        torch.cuda.synchronize()
        return dw.cpu().numpy(), dt.cpu().numpy()

    torch.cuda.synchronize()
    dw, dt = launch(0, n)
    f = feats.cpu().numpy() * g.cpu().numpy()[:, None]
    want = abi.weights_grad(wn, f.sum(0))
    np.testing.assert_allclose(dw, want, rtol=0, atol=1e-12 * np.max(abi.weights_grad(np.abs(wn), np.abs(f).sum(0))))
    parts = sum(launch(a, min(a + 8, n))[1] for a in range(0, n, 8))
    np.testing.assert_allclose(dt, parts, rtol=0, atol=1e-4 * np.max(np.abs(parts)))
    ctx.close()


@pytest.mark.parametrize("n", [0, 1, 33, 8192, 20001])
def test_weight_grad_of_features(n):
    """The same map from given features (FP64 sums: 1e-12 of the sum of magnitudes), added to
    what the output holds; no pose leaves it as it is."""
    torch = pytest.importorskip("torch")
    native.load(auto_build=True)
    rng = np.random.default_rng(n)
    f, g = rng.normal(size=(n, abi.NUM_SCORE_FEATURES)), rng.normal(size=n)
    w, before = rng.normal(size=abi.NUM_SF_WEIGHTS), rng.normal(size=abi.NUM_SF_WEIGHTS)
    fd, gd, wd, dw = (torch.tensor(a, device="cuda") for a in (np.vstack([f, f[:1] * 0 if n else np.zeros((1, 28))]),
                                                               np.append(g, 7.0), w, before))
    ctx = native.Context(0)
    torch.cuda.synchronize()
    ctx.score_weight_grad_dev(n, fd.data_ptr(), gd.data_ptr(), wd.data_ptr(), dw.data_ptr())
    torch.cuda.synchronize()
    want = before + abi.weights_grad(w, (f * g[:, None]).sum(0))
    size = np.abs(before) + abi.weights_grad(np.abs(w), np.abs(f * g[:, None]).sum(0))
    assert np.all(np.abs(dw.cpu().numpy() - want) <= 1e-12 * size)
    ctx.close()
