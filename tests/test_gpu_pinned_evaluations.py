"""Large pinned gradient arrays, which the GPU adds to, where an evaluation runs
twice because its neighbour rows overflow (the first attempt must add nothing),
and beside a captured mutual solve in mixed precision; with other numbers in the
arrays before, against pageable arrays.  Repeated evaluations differ by the order
of the PME's atomic adds: in FP64 about 1e-12 of the norm (1e-9 allowed), in mixed
precision FP32 roundings (2e-7 of the norm; 1e-5 allowed)."""
import numpy as np
import pytest
import torch

from polmdqc_b200 import abi, systems
from polmdqc_b200.engine import Engine, Settings

pytestmark = pytest.mark.gpu
FLAGS = abi.DO_ENERGY | abi.DO_GRADIENT
WATERS, BOX, GRID = 11000, 69.1, 72  # 99,000 values: above the line from which the GPU handles arrays


def pinned(a):
    return torch.from_numpy(np.array(a, np.float64).reshape(-1)).pin_memory().numpy()


def check(e, xyz, tol):
    """One call with pinned arrays at new coordinates, then one with pageable ones."""
    rng = np.random.default_rng(4)
    a, b = rng.standard_normal(xyz.size), rng.standard_normal(xyz.size)
    e.set_coords(pinned(xyz))
    first, second = pinned(a), pinned(b)
    e.forward_into(FLAGS, first, second)
    dem, dep = a.copy(), b.copy()
    e.forward_into(FLAGS, dem, dep)
    for x, y, old in ((first, dem, a), (second, dep, b)):
        assert np.linalg.norm(y - old) > np.linalg.norm(old)
        assert np.linalg.norm(x - y) <= tol * np.linalg.norm(y - old)


def test_overflowing_lists_add_once():
    s = systems.water_box(WATERS, BOX, seed=2)
    e = Engine(s, Settings(nfft=(GRID,) * 3, poltyp=abi.POL_DIRECT, precision=abi.PREC_FP64))
    try:
        check(e, s.xyz, 1e-9)
        # molecules moved into the middle half of the cell: twice the density, more partners than the
        # rows estimated from the average density hold (at most 288; the average is 287 now, within the slab more)
        mol = s.xyz.reshape(-1, 3, 3)
        dense = mol.copy()
        dense[:, :, 2] -= 0.5 * mol[:, :1, 2]
        d = dense.reshape(-1, 3)
        check(e, d, 1e-9)
        check(e, s.xyz, 1e-9)
    finally:
        e.close()


def test_pinned_arrays_beside_a_mixed_solve():
    s = systems.water_box(WATERS, BOX, seed=2)
    e = Engine(s, Settings(nfft=(GRID,) * 3, poltyp=abi.POL_MUTUAL, precision=abi.PREC_MIXED))
    try:
        for _ in range(2):
            check(e, s.xyz, 1e-5)
    finally:
        e.close()
