"""The map build's chunks of points, by the number of receptor atom kinds: the launches of a box on
a runtime of host memory, and the maps of a box of several chunks against the FP64 port."""
import ctypes as C
import os

import numpy as np
import pytest

import fake_runtime
import oracle
from pxdock_gb300 import abi, model, native, synth


def own_kinds(n_heavy, spread=1e-3):
    """A receptor whose atoms all have a sigma of their own."""
    rec = model.Receptor.from_json(synth.make_receptor(seed=5, n_heavy=n_heavy, cube=18.0, cavity=3.0))
    rec.ff.sigma[:] = rec.ff.sigma + spread * np.arange(rec.n_atoms) / rec.n_atoms
    return rec


def test_launches(tmp_path):
    """Whatever the number of kinds, a launch has three blocks per SM (152 here) while points are
    left, the workspace is at most 2 GB, and less memory makes smaller chunks, not an error."""
    box = model.make_box((0.0, 0.0, 0.0), (25.0, 25.0, 25.0), 0.375)
    P = int(np.prod(list(box.npoints)))
    with fake_runtime.loaded(tmp_path) as fake, native.Context(0) as ctx:
        for rec in (model.Receptor.from_json(synth.make_receptor(seed=5, n_heavy=300)), own_kinds(300), own_kinds(1500)):
            ctx.set_receptor(rec)
            for short in (False, True):
                fake.reset()
                fake.lib.fake_fail_at(1 if short else -1)  # the maps, then the workspace
                ctx.build_grid(box, [3, 5])
                fake.lib.fake_fail_at(-1)
                blocks = [g[0] for name, g in fake.launches() if "grid_moment" in name]
                assert sum(blocks) >= (P + 127) // 128 and (sum(blocks) - len(blocks)) * 128 < P
                if not short:
                    assert min(blocks[:-1], default=456) >= 456
                    full = len(blocks)
                else:
                    assert full <= len(blocks) <= 2 * full
                assert fake.lib.fake_largest() <= (2 << 30) + (1 << 22)


@pytest.mark.gpu
def test_maps_of_several_chunks():
    """Tolerances as for one chunk (test_gpu_grid_build)."""
    native.load(auto_build=True)
    rec = own_kinds(320)
    types = [3, 4, 11]
    box = model.make_box((0.11, -0.2, 0.3), (16.0, 15.0, 17.0), 0.375)
    P = int(np.prod(list(box.npoints)))
    assert P > 2 * 152 * 256  # three chunks
    port = oracle.PortSystem(rec, model.Ligand.from_json(synth.make_ligand(seed=1)))
    port.build_grid(box, types, nthreads=os.cpu_count() or 1)
    rec64 = np.zeros((P, 4))
    with native.Context(0) as ctx:
        ctx.set_receptor(rec)
        ctx.build_grid(box, types)
        for m in [abi.COULOMB_MAP] + types:
            ref = port.grid_map(m, box)
            big = np.max(np.abs(ref), axis=1)
            assert np.all(np.abs(ctx.read_map(m).astype(np.float64) - ref).max(axis=1) <= 2e-5 * big + 1e-6), m
            ctx._check(ctx.lib.pxd_grid_read_map64(ctx.h, m, rec64.ctypes.data_as(C.POINTER(C.c_double))))
            assert np.all(np.abs(rec64[:, 0] - ref[:, 0]) <= 1e-8 + 1e-9 * np.abs(ref[:, 0])), m
