"""The second population array of the multi-step tiles: it is there once the
program has been passed (no allocation in a later call, so another thread's
stream capture is left alone), and a named launch shape gives it back; a lattice
of more rows than the one-step sweep's grid takes is refused as without tiles."""
import threading

import numpy as np
import pytest

from lbm_mirror_gb300 import Lattice
from lbm_mirror_gb300 import capi as K
from lbm_mirror_gb300.lattice import KelError

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

OPS = {1: dict(bc=K.KEL_BC_BOUNCE_BACK), 2: dict(bc=K.KEL_BC_FLUID, collide=1)}


def _lattice(dims, stream=None):
    lat = Lattice("D2Q9", dims, stream=stream)
    lat.upload_flags(np.full(dims[0] * dims[1], 2, np.uint8))
    return lat


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_the_array_comes_with_the_program_and_goes_with_a_named_shape():
    prog = K.make_program(0.8, K.KEL_COLL_BGK, OPS)
    dims = (2304, 2048)  # 170 MB of populations
    size = dims[0] * dims[1] * 36
    lat = _lattice(dims)
    before = _free()
    lat.step(prog, 0)
    assert lat.tiles()[0] == 4
    with_program = _free()
    assert size <= before - with_program < size + (64 << 20)
    lat.step(prog, 24)
    assert _free() == with_program
    lat.set_launch(1, 128)
    assert lat.tiles()[0] == 1
    assert _free() - with_program >= size
    lat.step(prog, 24)
    lat.synchronize()
    lat.close()


def test_a_step_leaves_another_threads_capture_alone():
    prog = K.make_program(0.8, K.KEL_COLL_BGK, OPS)
    stream, other = torch.cuda.Stream(), torch.cuda.Stream()
    first = _lattice((96, 64))  # the kernels are loaded outside the capture
    first.step(prog, 40, write_macros=False)
    first.close()
    lat = _lattice((96, 64), other.cuda_stream)
    lat.step(prog, 0)
    lat.synchronize()
    x = torch.zeros(1024, device="cuda")
    torch.cuda.synchronize()
    failed = []

    def step():
        try:
            lat.step(prog, 40, write_macros=False)
        except KelError as e:
            failed.append(e)

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):  # capture mode "global"
        x += 1.0
        t = threading.Thread(target=step)
        t.start()
        t.join()
        x += 1.0
    graph.replay()
    torch.cuda.synchronize()
    assert not failed, failed
    assert float(x.sum()) == 2048.0
    lat.synchronize()
    assert lat.t == 40
    lat.close()


def test_rows_beyond_the_grid_are_refused():
    lat = _lattice((4, 70000))
    prog = K.make_program(0.8, K.KEL_COLL_BGK, OPS)
    for n in (1, 8, 200):
        with pytest.raises(KelError):
            lat.step(prog, n)
        assert lat.t == 0
    lat.close()
