"""The cell order by counting where the sites are spread unevenly: a droplet, and
a slab in a long periodic cell, with cells of up to 128 sites (counted), some
hundreds and more than a thousand (merged), and counts that are and are not
multiples of a warp's run.  The pair count is exact against the FP64 oracle,
energy and gradient at the FP64 path's tolerances; the first evaluation of the
droplet also overflows its lists, whose rows are estimated from the average
density, and is repeated."""
import dataclasses

import numpy as np
import pytest

from oracle import oracle
from polmdqc_b200 import abi, systems
from polmdqc_b200.engine import Engine, Settings

pytestmark = pytest.mark.gpu
FLAGS = abi.DO_ENERGY | abi.DO_GRADIENT | abi.DO_ANALYSIS


def droplet(waters, far):
    """A water cube of liquid density with its last molecule `far` A away along the diagonal, without a box."""
    s = systems.water_box(waters, (waters * 29.88) ** (1 / 3), seed=waters)
    xyz = s.xyz.copy()
    xyz[-3:] += far
    return dataclasses.replace(s, xyz=xyz, use_bounds=False)


def slab(waters, edge, height):
    """The same cube in a periodic cell that is `height` A long."""
    s = systems.water_box(waters, edge, seed=waters)
    return dataclasses.replace(s, box=np.array([edge, edge, height, 90.0, 90.0, 90.0]))


CASES = {
    "droplet_9": (lambda: droplet(2100, 160.0), 9.0),     # cells of ~80 sites and many empty ones
    "droplet_12": (lambda: droplet(2100, 200.0), 12.0),   # ~190
    "droplet_22": (lambda: droplet(2101, 180.0), 22.0),   # ~1,100
    "slab_12": (lambda: slab(2197, 40.4, 400.0), 12.0),   # ~250, most cells empty
}


@pytest.mark.parametrize("name", CASES)
def test_crowded_cells_match_the_oracle(name):
    make, cutoff = CASES[name]
    s = make()
    assert s.n > 6144  # ordered by counting
    st = Settings(use_ewald=False, poltyp=abi.POL_NONE, cutoff=cutoff, precision=abi.PREC_FP64)
    o = oracle.forward(s, st, flags=FLAGS)
    e = Engine(s, st)
    try:
        for _ in range(2):
            g = e.forward(FLAGS)
            assert g.nem == o.nem and o.nem > 0
            assert abs(g.em - o.em) <= 1e-10 * abs(o.em)
            np.testing.assert_allclose(g.dem, o.dem, atol=1e-8, rtol=0)
    finally:
        e.close()
