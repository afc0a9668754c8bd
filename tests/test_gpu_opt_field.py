"""OPT orders apply the dipole field from the pair geometry, in a context's own
precision with the intramolecular (scaled) pairs in FP64: they keep no
coefficient rows.  A row has a slot per partner, so rows would show in the
device memory of a context: 6,591 sites of ~230 slots of 16 bytes are 24 MB or
more, while the orders themselves (5 x 2 sets in FP64) are 2 MB; allocations are
mapped in pieces of 2 MB.  And the induced dipoles against the FP64 path, with
most sites having scaled partners in other molecules too: FP32 terms of 6e-8,
summed over ~150 partners with mixed signs, within 1e-5 of the norm."""
import dataclasses

import numpy as np
import pytest
import torch

from polmdqc_b200 import abi, systems
from polmdqc_b200.engine import Engine, Settings

pytestmark = pytest.mark.gpu


def memory_of(s, poltyp):
    """Device memory that a context holds after its first evaluation."""
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    e = Engine(s, Settings(nfft=(40, 40, 40), poltyp=poltyp, precision=abi.PREC_MIXED))
    try:
        e.forward(abi.DO_ENERGY | abi.DO_GRADIENT)
        return before - torch.cuda.mem_get_info()[0]
    finally:
        e.close()


def test_opt_keeps_no_rows():
    s = systems.water_box(2197, 40.4, seed=3)
    memory_of(s, abi.POL_DIRECT)  # what the first context of a process loads is no context's own
    assert memory_of(s, abi.POL_OPT) - memory_of(s, abi.POL_DIRECT) < 10 * 2 ** 20


@pytest.mark.parametrize("partners", [0, 30])
def test_opt_dipoles_with_many_scaled_pairs(partners):
    s = systems.water_box(216, 18.643, seed=8)
    i14 = [list(v) for v in s.lists["i14"]]
    for i in range(0, s.n, 3):
        for k in range(partners):
            j = (i + 5 + 7 * k) % s.n
            if j // 3 != i // 3 and j not in i14[i]:
                i14[i].append(j)
                i14[j].append(i)
    s = dataclasses.replace(s, lists=dict(s.lists, i14=[sorted(v) for v in i14]))
    out = []
    for prec in (abi.PREC_MIXED, abi.PREC_FP64):
        e = Engine(s, Settings(nfft=(24, 24, 24), cutoff=6.1, poltyp=abi.POL_OPT, precision=prec))
        try:
            out.append(e.forward(abi.DO_ENERGY | abi.DO_GRADIENT | abi.DO_DIPOLES))
        finally:
            e.close()
    for name in ("uind", "uinp", "dep"):
        x, y = getattr(out[0], name), getattr(out[1], name)
        assert np.linalg.norm(x - y) <= 1e-5 * np.linalg.norm(y) > 0, name
