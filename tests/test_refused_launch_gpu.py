"""A launch that is refused on the host (more rows than a grid takes) is reported by
its own call alone: the next ones work."""
import numpy as np
import pytest

from lbm_mirror_gb300 import Lattice
from lbm_mirror_gb300 import capi as K
from lbm_mirror_gb300.lattice import KelError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [1, 200])
def test_the_next_call_works(steps):
    prog = K.make_program(0.8, K.KEL_COLL_BGK, {2: dict(bc=K.KEL_BC_FLUID, collide=1)})
    tall = Lattice("D3Q19", (4, 70000, 1))
    tall.upload_flags(np.full(280000, 2, np.uint8))
    with pytest.raises(KelError):
        tall.step(prog, steps)
    lat = Lattice("D3Q19", (8, 8, 8))
    lat.upload_flags(np.full(512, 2, np.uint8))
    lat.step(prog, 2)
    assert np.isfinite(lat.populations()).all()
    lat.close()
    tall.set_launch(4, 128)  # a shape whose grid has no such limit
    tall.step(prog, 2)
    assert tall.t == 2
    tall.close()
