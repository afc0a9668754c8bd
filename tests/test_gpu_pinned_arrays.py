"""Large pinned arrays, which the GPU adds to and checks itself: the sums, what
was in the arrays before, arrays shared by both gradients and the refusal of
non-finite coordinates are those of pageable arrays, which the host handles.
FP64 with direct polarization: two evaluations differ by the order of the PME's
atomic adds (about 1e-12), and the additions are the same IEEE operations."""
import numpy as np
import pytest
import torch

from polmdqc_b200 import abi, systems
from polmdqc_b200.engine import AmgError, Engine, Settings

pytestmark = pytest.mark.gpu
FLAGS = abi.DO_ENERGY | abi.DO_GRADIENT


def pinned(a):
    return torch.from_numpy(np.array(a, np.float64).reshape(-1)).pin_memory().numpy()


@pytest.fixture(scope="module")
def box():
    s = systems.water_box(11000, 69.1, seed=2)  # 99,000 values: above the line
    e = Engine(s, Settings(nfft=(72, 72, 72), poltyp=abi.POL_DIRECT, precision=abi.PREC_FP64))
    yield s, e
    e.close()


def test_pinned_gradients_are_added_like_pageable_ones(box):
    s, e = box
    rng = np.random.default_rng(1)
    a, b = rng.standard_normal(3 * s.n), rng.standard_normal(3 * s.n)
    dem, dep = a.copy(), b.copy()
    e.set_coords(s.xyz)
    e.forward_into(FLAGS, dem, dep)
    assert np.abs(dem - a).max() > 1 and np.abs(dep - b).max() > 1
    for first, second in ((pinned(a), pinned(b)), (pinned(a), b.copy()), (a.copy(), pinned(b))):
        e.set_coords(pinned(s.xyz))
        e.forward_into(FLAGS, first, second)
        np.testing.assert_allclose(first, dem, atol=1e-9, rtol=0)
        np.testing.assert_allclose(second, dep, atol=1e-9, rtol=0)
    one = pinned(a)  # both gradients into one array
    e.forward_into(FLAGS, one, one)
    np.testing.assert_allclose(one, dem + dep - b, atol=1e-9, rtol=0)
    only = pinned(b)
    e.forward_into(FLAGS, None, only)
    np.testing.assert_allclose(only, dep, atol=1e-9, rtol=0)


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("where", [0, -1])
def test_pinned_non_finite_coordinates_are_refused(box, value, where):
    s, e = box
    bad = pinned(s.xyz)
    bad[where] = value
    with pytest.raises(AmgError, match="NAN"):
        e.set_coords(bad)
    with pytest.raises(AmgError, match="BAD_ARG"):
        e.forward(FLAGS)
    e.set_coords(pinned(s.xyz))
    assert np.isfinite(e.forward(FLAGS).em)
