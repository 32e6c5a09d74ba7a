"""The differentiable score of no poses: its gradients are zeros, as for any batch's missing
poses. The host's part on a runtime of host memory; the whole call on the GPU."""
import os

import pytest

import fake_runtime
from pxdock_gb300 import abi, autograd, model, native, synth


def test_weight_grad_of_no_address(tmp_path):
    with fake_runtime.loaded(tmp_path) as fake, native.Context(0) as ctx:
        fake.reset()
        ctx.score_weight_grad_dev(0, None, None, None, None)
        assert fake.launches() == []
        with pytest.raises(native.NativeError):
            ctx.score_weight_grad_dev(1, None, None, None, None)


@pytest.mark.gpu
def test_backward_of_no_poses():
    torch = pytest.importorskip("torch")
    native.load(auto_build=True)
    rec = model.Receptor.from_json(synth.make_receptor(seed=0, n_heavy=60, cube=16.0, cavity=4.0))
    lig = model.Ligand.from_json(synth.make_ligand(seed=1, n_heavy=9, n_rot=2))
    sf = model.load_scoring_function(os.path.join(os.path.dirname(model.__file__), "data", "scoring_function.json"))[0]
    ctx = native.Context(0)
    ctx.set_receptor(rec)
    ctx.set_scoring_function(0, sf)
    ctx.add_ligand(lig)
    x = torch.zeros((0, lig.n_atoms, 3), device="cuda", requires_grad=True)
    w = torch.tensor(abi.sf_weights(sf), device="cuda", requires_grad=True)
    ids = torch.zeros(0, dtype=torch.int32, device="cuda")
    autograd.empirical_score(ctx, ids, x, w).sum().backward()
    assert x.grad.shape == x.shape
    assert torch.equal(w.grad, torch.zeros_like(w))
    ctx.close()
