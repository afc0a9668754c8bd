"""PME spreading and gathers at grid sizes where a stencil line's pairs of
points wrap, start at odd places or do not exist (odd sizes), on the smallest
grids and with a count of sites that fills no block, against the FP64 oracle on
the same grid, in both precisions (the parity tests' tolerances)."""
import numpy as np
import pytest

from oracle import oracle
from polmdqc_b200 import abi, systems
from polmdqc_b200.engine import Engine, Settings

pytestmark = pytest.mark.gpu
FLAGS = abi.DO_ENERGY | abi.DO_GRADIENT | abi.DO_DIPOLES


@pytest.mark.parametrize("prec", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("nfft", [(8, 9, 8), (10, 8, 9), (12, 15, 14), (21, 16, 27)])
def test_small_and_odd_grids_match_the_oracle(nfft, prec):
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
