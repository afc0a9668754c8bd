"""Gradient arrays of which only parts are pinned -- the ends, two registrations
side by side, all but the last page -- are the host's to add to: the call takes
them like pageable arrays, without a device copy of the whole.  FP64 with direct
polarization; two evaluations differ by the order of the PME's atomic adds."""
import mmap

import numpy as np
import pytest
import torch

from polmdqc_b200 import abi, systems
from polmdqc_b200.engine import Engine, Settings

pytestmark = pytest.mark.gpu
FLAGS = abi.DO_ENERGY | abi.DO_GRADIENT
PAGE = mmap.PAGESIZE


@pytest.fixture(scope="module")
def box():
    s = systems.water_box(11000, 69.1, seed=2)  # 99,000 values: above the line from which the GPU handles arrays
    e = Engine(s, Settings(nfft=(72, 72, 72), poltyp=abi.POL_DIRECT, precision=abi.PREC_FP64))
    yield s, e
    e.close()


def registered(count, pieces):
    """An array of `count` values on whole pages, of which the (first, last + 1) page ranges are registered."""
    pages = -(-8 * count // PAGE)
    a = np.frombuffer(mmap.mmap(-1, pages * PAGE), np.float64)
    at = [a.ctypes.data + (i if i >= 0 else pages + i) * PAGE for i, _ in pieces]
    for p, (i, j) in zip(at, pieces):
        i, j = (k if k >= 0 else pages + k for k in (i, j if j else pages))
        assert int(torch.cuda.cudart().cudaHostRegister(p, (j - i) * PAGE, 0)) == 0
    return a[:count], at


@pytest.mark.parametrize("pieces", [((0, 3), (-2, 0)),      # the ends
                                    ((0, 60), (60, 0)),     # all of it, in two
                                    ((0, -1),),             # all but the last page
                                    ((0, 0),)])             # all of it, in one: the GPU's
def test_partly_pinned_gradients(box, pieces):
    s, e = box
    e.set_coords(s.xyz)
    rng = np.random.default_rng(3)
    old = rng.standard_normal(3 * s.n)
    dem, dep = old.copy(), old.copy()
    e.forward_into(FLAGS, dem, dep)
    a, at_a = registered(3 * s.n, pieces)
    b, at_b = registered(3 * s.n, pieces)
    try:
        a[:], b[:] = old, old
        e.forward_into(FLAGS, a, b)
        np.testing.assert_allclose(a, dem, atol=1e-9, rtol=0)
        np.testing.assert_allclose(b, dep, atol=1e-9, rtol=0)
    finally:
        for p in at_a + at_b:
            assert int(torch.cuda.cudart().cudaHostUnregister(p)) == 0
