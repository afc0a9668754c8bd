"""amg_set_coords has read the caller's coordinates when it returns, from pinned
memory (which the device copies by itself) as from pageable memory: the array is
overwritten right after the call, with the copies of this device busy for some
milliseconds before it, and the evaluation is that of the coordinates given.
FP64; two evaluations differ by the order of the PME's atomic adds (about
1e-12)."""
import numpy as np
import pytest
import torch

from polmdqc_b200 import abi, systems
from polmdqc_b200.engine import AmgError, Engine, Settings

pytestmark = pytest.mark.gpu
FLAGS = abi.DO_ENERGY | abi.DO_GRADIENT


def pinned(a):
    return torch.from_numpy(np.array(a, np.float64).reshape(-1)).pin_memory().numpy()


@pytest.mark.parametrize("waters, box, nfft", [(216, 18.643, 24), (1820, 37.9, 40), (1821, 37.9, 40), (2744, 43.5, 48),
                                               (11000, 69.1, 72)])  # staged (up to 16,384 values), waited for, the GPU's
def test_coordinates_are_read_before_the_call_returns(waters, box, nfft):
    s = systems.water_box(waters, box, seed=5)
    other = systems.water_box(waters, box, seed=6).xyz.reshape(-1)
    e = Engine(s, Settings(nfft=(nfft,) * 3, poltyp=abi.POL_DIRECT, precision=abi.PREC_FP64))
    big = torch.zeros(64 << 20, dtype=torch.float64).pin_memory()  # 512 MB: about 10 ms
    dst, side = torch.empty_like(big, device="cuda"), torch.cuda.Stream()
    try:
        e.set_coords(s.xyz)
        ref = e.forward(FLAGS)
        xyz = pinned(s.xyz)
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            dst.copy_(big, non_blocking=True)
        e.set_coords(xyz)
        xyz[:] = other
        g = e.forward(FLAGS)
        assert abs(g.em - ref.em) <= 1e-9 * abs(ref.em) and abs(g.ep - ref.ep) <= 1e-9 * abs(ref.ep)
        np.testing.assert_allclose(g.dem, ref.dem, atol=1e-8, rtol=0)
        # a refused array is the caller's again too
        xyz[:] = s.xyz.reshape(-1)
        xyz[-1] = np.nan
        with torch.cuda.stream(side):
            dst.copy_(big, non_blocking=True)
        with pytest.raises(AmgError, match="NAN"):
            e.set_coords(xyz)
        xyz[:] = other
        e.set_coords(s.xyz)
        assert abs(e.forward(FLAGS).em - ref.em) <= 1e-9 * abs(ref.em)
        # two calls in a row: the second one's coordinates
        xyz[:] = other
        with torch.cuda.stream(side):
            dst.copy_(big, non_blocking=True)
        e.set_coords(xyz)
        xyz[:] = s.xyz.reshape(-1)
        e.set_coords(xyz)
        xyz[:] = other
        assert abs(e.forward(FLAGS).em - ref.em) <= 1e-9 * abs(ref.em)
    finally:
        torch.cuda.synchronize()
        e.close()
