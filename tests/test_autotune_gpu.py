"""kel_lattice_autotune times what kel_step then runs: overlapped one-cell sweeps on a
stream, and the multi-step tiles of a D2Q9 lattice.  The time it returns is compared
with that of the steps after it, on the device: equal launches, so within 15 %
(before, sweeps timed without the overlap were 1.2 to 1.5 times the steps after
them, one-step sweeps in place of tiles 1.5 times)."""
import numpy as np
import pytest

from lbm_mirror_gb300 import Lattice
from lbm_mirror_gb300 import capi as K
from lbm_mirror_gb300.workloads import cavity_flags

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

OPS = {1: dict(bc=K.KEL_BC_BOUNCE_BACK), 2: dict(bc=K.KEL_BC_FLUID, collide=1)}


@pytest.mark.parametrize("name,dims", [("D3Q19", (64, 64, 64)), ("D2Q9", (1024, 1024)), ("D2Q9", (400, 240))])
def test_the_returned_time_is_that_of_the_steps(name, dims):
    stream = torch.cuda.Stream()
    lat = Lattice(name, dims, stream=stream.cuda_stream)
    flags = cavity_flags(dims)
    flags[flags == 5] = 1
    lat.upload_flags(flags)
    prog = K.make_program(0.8, K.KEL_COLL_BGK, OPS)
    lat.step(prog, 0)
    tiles = lat.tiles()
    told = min(lat.autotune(prog, steps=96)[2] for _ in range(3))
    assert lat.t == 0 and lat.tiles() == tiles
    assert tiles[0] == (4 if dims == (400, 240) else 1)
    lat.step(prog, 96, write_macros=False)
    took = 1e9
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        lat.step(prog, 96, write_macros=False)
        b.record(stream)
        b.synchronize()
        took = min(took, a.elapsed_time(b) / 96)
    assert 0.85 * took <= told <= 1.15 * took, (told, took)
    lat.close()
