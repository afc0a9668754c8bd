"""The cell-grid neighbour lists at the edges of their staging: fewer and more
hits than a warp's queue holds, more home sites and candidates than one chunk,
a last chunk that is not a multiple of the scan, two blocks per cell, sites
with more scaled partners than a warp has lanes, and the cell order by counting
with cells of more and fewer sites than a warp.  The pair count is exact
against the FP64 oracle; energies and gradients at the FP64 path's tolerances
against it (the same pairs, FP64 sums in another order)."""
import dataclasses

import numpy as np
import pytest

from oracle import oracle
from polmdqc_b200 import abi, systems
from polmdqc_b200.engine import Engine, Settings

pytestmark = pytest.mark.gpu
FLAGS = abi.DO_ENERGY | abi.DO_GRADIENT | abi.DO_ANALYSIS


def many_partners(s, count):
    """s with the first atom of every 16th water 1-4 bonded to `count` atoms of other waters."""
    i14 = [list(v) for v in s.lists["i14"]]
    for i in range(0, s.n, 48):
        for k in range(count):
            j = (i + 5 + 7 * k) % s.n
            if j // 3 != i // 3 and j not in i14[i]:
                i14[i].append(j)
                i14[j].append(i)
    return dataclasses.replace(s, lists=dict(s.lists, i14=[sorted(v) for v in i14]))


@pytest.mark.parametrize("waters, box, cutoff, partners", [
    (27, 9.4, 3.1, 0),       # a handful of sites per cell, lists shorter than the queue
    (216, 18.643, 6.2, 0),   # 3 cells per axis
    (512, 24.9, 4.0, 0),     # 6 cells per axis
    (1331, 34.2, 11.3, 0),   # ~150 sites per cell, ~4,000 candidates
    (216, 18.643, 6.0, 40),  # rows with more than 32 scaled partners
    (2197, 40.4, 9.0, 0),    # sites ordered by counting: 64 cells of ~100 sites
    (2200, 80.0, 5.0, 0),    # ... 4,096 cells, most of 1 or 2 sites
])
def test_lists_match_the_oracle(waters, box, cutoff, partners):
    s = systems.water_box(waters, box, seed=waters)
    if partners:
        s = many_partners(s, partners)
    st = Settings(use_ewald=False, poltyp=abi.POL_NONE, cutoff=cutoff, precision=abi.PREC_FP64)
    o = oracle.forward(s, st, flags=FLAGS)
    e = Engine(s, st)
    try:
        g = e.forward(FLAGS)
    finally:
        e.close()
    assert g.nem == o.nem and o.nem > 0
    assert abs(g.em - o.em) <= 1e-10 * abs(o.em)
    np.testing.assert_allclose(g.dem, o.dem, atol=1e-8, rtol=0)
