"""A context whose box changes from call to call (pressure coupling): the
captured graph is updated in place and the influence function computed again,
so every call equals that of a new context at the same box, in the forward
(virial included) and in the adjoint -- over small changes, changes of the
neighbour cells' count and of the cell shape.  FP64; both contexts sum the same
terms, the atomic adds of the PME in another order (about 1e-12)."""
import numpy as np
import pytest

from polmdqc_b200 import abi, systems
from polmdqc_b200.engine import Engine, Settings

pytestmark = pytest.mark.gpu
FLAGS = abi.DO_ENERGY | abi.DO_GRADIENT | abi.DO_DIPOLES | abi.DO_VIRIAL


def close(a, b, what):
    a, b = np.asarray(a), np.asarray(b)
    assert np.max(np.abs(a - b)) <= 1e-9 * max(1.0, np.max(np.abs(b))), what


@pytest.mark.parametrize("poltyp, nfft", [(abi.POL_MUTUAL, (24, 25, 24)), (abi.POL_OPT, (24, 24, 27)),
                                          (abi.POL_NONE, (24, 24, 24))])
def test_changed_box_equals_a_new_context(poltyp, nfft):
    s = systems.water_box(216, 18.643, seed=8)
    st = Settings(nfft=nfft, cutoff=6.1, poltyp=poltyp, precision=abi.PREC_FP64)
    boxes = [[18.643] * 3 + [90.0] * 3, [18.7, 18.643, 18.8] + [90.0] * 3,
             [18.0, 18.643, 18.643] + [90.0] * 3,        # 2 cells on one axis
             [18.643] * 3 + [90.0] * 3, [19.5, 19.0, 19.2, 90.0, 84.0, 90.0], [18.7] * 3 + [90.0] * 3]
    e = Engine(s, st)
    try:
        for k, box in enumerate(boxes):
            xyz = s.xyz * (np.array(box[:3]) / 18.643) if k else s.xyz
            e.set_coords(xyz, box)
            g, adj = e.forward(FLAGS), None
            if poltyp == abi.POL_MUTUAL:
                adj = e.backward(1.0, np.full(3 * s.n, 0.01), np.full(3 * s.n, 0.02))
            new = Engine(s, st)
            try:
                new.set_coords(xyz, box)
                r = new.forward(FLAGS)
                ref = new.backward(1.0, np.full(3 * s.n, 0.01), np.full(3 * s.n, 0.02)) if adj else None
            finally:
                new.close()
            for name in ("em", "ep", "dem", "dep", "uind", "uinp", "vir"):
                close(getattr(g, name), getattr(r, name), (k, name))
            assert g.pcg_iters == r.pcg_iters
            if adj:
                for name in ref:
                    close(adj[name], ref[name], (k, name))
    finally:
        e.close()
