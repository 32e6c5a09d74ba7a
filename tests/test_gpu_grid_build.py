"""The map build against the FP64 port's maps, where its plan can go wrong: type counts off the
groups a thread takes, point counts off the block size, atom counts off the tiles, rotor
atoms left out, a receptor with an outlying atom (the wide coordinate split), and the FP64
energies beside the records."""
import ctypes as C
import os

import numpy as np
import pytest

import oracle
from pxdock_gb300 import abi, model, native, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heavy,rotors,types,size,outlier", [
    (30, 0, [3], (2.0, 1.0, 0.9), False),
    (210, 0, [3, 4, 5], (3.1, 4.0, 2.2), False),
    (260, 2, list(range(9)), (4.0, 3.0, 3.0), False),
    (120, 0, list(range(12, 29)), (3.0, 3.0, 3.0), True),
])
def test_maps_match_the_port(heavy, rotors, types, size, outlier):
    native.load(auto_build=True)
    js = synth.make_receptor(seed=5, n_heavy=heavy, cube=14.0, cavity=2.5, n_rotors=rotors)
    if outlier:
        js["xyz"][0] = [900.0, -700.0, 650.0]
    rec = model.Receptor.from_json(js)
    box = model.make_box((0.11, -0.2, 0.3), size, 0.375)
    ctx = native.Context(0)
    ctx.set_receptor(rec)
    ctx.build_grid(box, types)
    port = oracle.PortSystem(rec, model.Ligand.from_json(synth.make_ligand(seed=1)))
    port.build_grid(box, types, nthreads=os.cpu_count() or 1)
    P = int(np.prod(list(box.npoints)))
    rec64 = np.zeros((P, 4))
    for m in [abi.COULOMB_MAP] + types:
        ref = port.grid_map(m, box)
        gpu = ctx.read_map(m).astype(np.float64)
        # FP32 records: the energy rounded once (6e-8), the LJ gradient a sum of FP32 terms whose
        # attraction and repulsion cancel (1e-5 of the record's largest component)
        big = np.max(np.abs(ref), axis=1)
        assert np.all(np.abs(gpu - ref).max(axis=1) <= 2e-5 * big + 1e-6), m
        ctx._check(ctx.lib.pxd_grid_read_map64(ctx.h, m, rec64.ctypes.data_as(C.POINTER(C.c_double))))
        # FP64 energies: pairs of ~47 bits over sums of at most ~1e4 kcal/mol (the r^-12 terms
        # in FP64), kept as FP32 record + FP32 remainder (2^-48)
        assert np.all(np.abs(rec64[:, 0] - ref[:, 0]) <= 1e-8 + 1e-9 * np.abs(ref[:, 0])), m
    ctx.close()
