"""A mixed-precision context whose box changes from call to call (pressure
coupling): energies, gradients and the virial of every call against the FP64
oracle at that box and against a new context there -- over small changes, a
change of the neighbour cells' count and of the cell shape, grids of the own
transform and of the library's.

Against the oracle: the parity tests' tolerances of the mixed path (energies
1e-6, virial 1e-5 of its largest element).  Against a new context: the two run
the same kernels, whose FP32 atomic adds come in another order, so the spread is
that of FP32 rounding (2^-24 = 6e-8) in the largest terms of an output; 16 of
them (1e-6) for the scalars and the virial, whose single large structure factors
round one way or the other, and 1e-5 for the norm of the gradients, where
neighbours' forces cancel to a tenth."""
import dataclasses

import numpy as np
import pytest

from oracle import oracle
from polmdqc_b200 import abi, systems
from polmdqc_b200.engine import Engine, Settings

pytestmark = pytest.mark.gpu
FLAGS = abi.DO_ENERGY | abi.DO_GRADIENT | abi.DO_VIRIAL
BOX = 18.643


@pytest.mark.parametrize("nfft", [(24, 24, 24), (24, 28, 25)])
def test_changed_box_in_mixed_precision(nfft):
    s = systems.water_box(216, BOX, seed=8)
    st = Settings(nfft=nfft, cutoff=6.1, precision=abi.PREC_MIXED, poleps=1e-6)
    ref = Settings(nfft=nfft, cutoff=6.1, precision=abi.PREC_FP64)
    edges = [(BOX, BOX, BOX, 90.0), (BOX * 1.001, BOX * 1.001, BOX * 1.001, 90.0), (18.0, BOX, BOX, 90.0),
             (BOX, BOX, BOX, 90.0), (19.5, 19.0, 19.2, 84.0)]
    e = Engine(s, st)
    try:
        for k, (a, b, c, beta) in enumerate(edges):
            box = np.array([a, b, c, 90.0, beta, 90.0])
            xyz = s.xyz * (box[:3] / BOX)
            e.set_coords(xyz, box)
            g = e.forward(FLAGS)
            new = Engine(s, st)
            try:
                new.set_coords(xyz, box)
                r = new.forward(FLAGS)
            finally:
                new.close()
            o = oracle.forward(dataclasses.replace(s, xyz=xyz, box=box), ref, tol=1e-11, flags=FLAGS)
            scale = np.abs(o.vir).max()
            for name in ("em", "ep"):
                assert abs(getattr(g, name) - getattr(o, name)) <= 1e-6 * abs(getattr(o, name)), (k, name)
                assert abs(getattr(g, name) - getattr(r, name)) <= 1e-6 * abs(getattr(r, name)), (k, name)
            assert np.abs(g.vir - o.vir).max() <= 1e-5 * scale, k
            assert np.abs(g.vir - r.vir).max() <= 1e-6 * scale, k
            for name in ("dem", "dep"):
                x, y = getattr(g, name), getattr(r, name)
                assert np.linalg.norm(x - y) <= 1e-5 * np.linalg.norm(y), (k, name)
    finally:
        e.close()
