"""PME at the edges of its kernels' sizes, against the FP64 oracle on the same
grid, in both precisions (the parity tests' tolerances): grids where a stencil
line's pairs of points wrap, start at odd places or do not exist (odd sizes),
the smallest grids and a count of sites that fills no block; and the dipole
grid's transform with every kind of radix, in one kernel per plane or one per
axis, beside sizes that only the library's transform takes (8, 10, 14, 21)."""
import numpy as np
import pytest

from oracle import oracle
from polmdqc_b200 import abi, systems
from polmdqc_b200.engine import Engine, Settings

pytestmark = pytest.mark.gpu
FLAGS = abi.DO_ENERGY | abi.DO_GRADIENT | abi.DO_DIPOLES


SMALL = [(8, 9, 8), (10, 8, 9), (12, 15, 14), (21, 16, 27), (9, 12, 15), (16, 30, 25), (50, 45, 48), (16, 36, 75)]
# grids of 7 to 27 points per Angstrom: in FP64 only (FP32 weights and
# differences of neighbouring points lose what their tolerance asks for, with
# any transform)
FINE = [(64, 16, 144), (50, 81, 45), (16, 160, 240), (256, 15, 16)]


@pytest.mark.parametrize("nfft, prec", [(k, p) for k in SMALL for p in (abi.PREC_FP64, abi.PREC_MIXED)] +
                         [(k, abi.PREC_FP64) for k in FINE])
def test_grid_sizes_match_the_oracle(nfft, prec):
    s = systems.water_box(27, 9.4, seed=3)
    kw = dict(nfft=nfft, cutoff=4.6)
    o = oracle.forward(s, Settings(precision=abi.PREC_FP64, **kw), tol=1e-11, flags=FLAGS)
    fp64 = prec == abi.PREC_FP64
    e = Engine(s, Settings(precision=prec, poleps=1e-8 if fp64 else 1e-6, **kw))
    try:
        g = e.forward(FLAGS)
    finally:
        e.close()
    assert abs(g.em - o.em) <= (1e-10 if fp64 else 1e-6) * abs(o.em)
    assert abs(g.ep - o.ep) <= (1e-8 if fp64 else 1e-6) * abs(o.ep)
    if fp64:
        np.testing.assert_allclose(g.dem, o.dem, atol=1e-8, rtol=0)
        np.testing.assert_allclose(g.dep, o.dep, atol=1e-5, rtol=0)
    else:
        assert float(np.sqrt(np.mean((g.dem + g.dep - o.dem - o.dep) ** 2))) < 1e-4
