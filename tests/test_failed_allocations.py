"""An installation whose allocation fails: the call reports it, and the context is in a state that
it knows - without a receptor, or with the scoring function that was there - so that no kernel
is launched on what is missing. On a runtime of host memory."""
import os

import numpy as np
import pytest

import fake_runtime
from pxdock_gb300 import model, native, synth


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    with fake_runtime.loaded(tmp_path_factory.mktemp("fake")) as f:
        yield f


@pytest.fixture()
def parts():
    rec = model.Receptor.from_json(synth.make_receptor(seed=0, n_heavy=60, cube=16.0, cavity=4.0))
    lig = model.Ligand.from_json(synth.make_ligand(seed=1, n_heavy=9, n_rot=2))
    sf = model.load_scoring_function(os.path.join(os.path.dirname(model.__file__), "data", "scoring_function.json"))
    return rec, lig, sf


def allocations(fake, call):
    fake.lib.fake_fail_at(-1)
    call()
    return fake.lib.fake_mallocs()


def fails(fake, k, call):
    fake.lib.fake_fail_at(k)
    with pytest.raises(native.NativeError):
        call()
    fake.lib.fake_fail_at(-1)
    fake.reset()


def test_receptor(fake, parts):
    rec, lig, sf = parts
    with native.Context(0) as ctx:
        ctx.set_scoring_function(0, sf[0])
        lid = ctx.add_ligand(lig)
        n = allocations(fake, lambda: ctx.set_receptor(rec))
        assert n >= 5
        for k in range(n):
            fails(fake, k, lambda: ctx.set_receptor(rec))
            for call in (lambda: ctx.score(0, lid, lig.poses[:1]),
                         lambda: ctx.mc_search(native.mc_params([-1] * 3, [1] * 3), lid, lig.poses[:1], np.arange(1))):
                with pytest.raises(native.NativeError) as e:
                    call()
                assert e.value.code == 2
            assert fake.launches() == []
            ctx.set_receptor(rec)
            ctx.score(0, lid, lig.poses[:1])
        assert fake.violations == ""


def test_scoring_function(fake, parts):
    rec, lig, sf = parts
    with native.Context(0) as ctx:
        ctx.set_receptor(rec)
        lid = ctx.add_ligand(lig)
        n = 2  # a first installation: the function and its table
        for k in range(n):
            fails(fake, k, lambda: ctx.set_scoring_function(1, sf[1]))
            with pytest.raises(native.NativeError):
                ctx.score(1, lid, lig.poses[:1])
            assert fake.launches() == []
            if k == 0:
                assert allocations(fake, lambda: native.Context.set_scoring_function(ctx, 0, sf[0])) == n
        ctx.set_scoring_function(1, sf[1])
        # another in its place: the one that was there stays
        fails(fake, 0, lambda: ctx.set_scoring_function(1, sf[0]))
        ctx.score(1, lid, lig.poses[:1])
        assert fake.violations == ""
