"""A force field that is uploaded while captured launches exist.  The sweeps do
not read a field that nothing was written to, and graphs hold that choice: the
library's own graph of sweeps, the particles' graph of two coupled steps and a
caller's graph all have to see a field uploaded after their capture.  Each run is
compared, bit for bit, with one whose field of zeros was uploaded at the start
and so was read from the first step on."""
import numpy as np
import pytest

from lbm_mirror_gb300 import Lattice, Particles
from lbm_mirror_gb300 import capi as K
from tests import cases

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

OPS = {1: dict(bc=K.KEL_BC_BOUNCE_BACK), 2: dict(bc=K.KEL_BC_FLUID, collide=1)}
SIZES = [(9, (76, 45)), (9, (400, 300)), (19, (36, 20, 16))]  # tiles, one-step sweep, 3D


def _lattice(q, dims, zeros, periodic=False):
    stream = torch.cuda.Stream()
    lat = Lattice({9: "D2Q9", 19: "D3Q19"}[q], dims, periodic_x=periodic, stream=stream.cuda_stream)
    n = int(np.prod(dims))
    rng = np.random.default_rng(n)
    flags = np.full(n, 2, np.uint8)
    flags.reshape(-1, dims[0])[[0, -1]] = 1
    lat.upload_flags(flags)
    lat.upload_populations(cases.random_populations(q, n, rng).astype(np.float32))
    D = 2 if q == 9 else 3
    if zeros:
        lat.upload_force(np.zeros((n, D), np.float32))
    force = (1e-4 * rng.standard_normal((n, D))).astype(np.float32)
    return lat, stream, force


def _same(a, b):
    assert a.t == b.t
    np.testing.assert_array_equal(a.populations(), b.populations())


@pytest.mark.parametrize("q,dims", SIZES)
@pytest.mark.parametrize("arithmetic", [K.KEL_ARITH_FAST, K.KEL_ARITH_REFERENCE])
def test_upload_after_the_sweeps_were_captured(q, dims, arithmetic):
    prog = K.make_program(0.7, K.KEL_COLL_BGK_GUO, OPS, global_force=(1e-5, 0, 0), arithmetic=arithmetic)
    runs = []
    for zeros in (False, True):
        lat, _, force = _lattice(q, dims, zeros)
        lat.step(prog, 150, write_macros=False)
        before = lat.populations()
        lat.upload_force(force)
        lat.step(prog, 150, write_macros=False)
        runs.append((before, lat.populations()))
        lat.close()
    np.testing.assert_array_equal(runs[0][0], runs[1][0])
    np.testing.assert_array_equal(runs[0][1], runs[1][1])


@pytest.mark.parametrize("q,dims", SIZES)
def test_upload_before_a_callers_graph_is_replayed(q, dims):
    prog = K.make_program(0.7, K.KEL_COLL_BGK_GUO, OPS, global_force=(1e-5, 0, 0))
    lats = []
    for zeros in (False, True):
        lat, stream, force = _lattice(q, dims, zeros)
        lat.step(prog, 2, write_macros=False)
        lat.synchronize()
        if zeros:
            lat.upload_force(force)
            lat.step(prog, 10, write_macros=False)
        else:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                lat.step(prog, 10, write_macros=False)
            lat.upload_force(force)
            with torch.cuda.stream(stream):
                graph.replay()
            stream.synchronize()
        lats.append(lat)
    _same(*lats)
    for lat in lats:
        lat.close()


def test_upload_after_the_coupled_steps_were_captured():
    dims = (256, 96)
    prog = K.make_program(0.7, K.KEL_COLL_PSM_GUO, OPS, global_force=(0.0, -1e-5, 0.0))
    prm = K.make_particle_params(K.KEL_POROSITY_SUBCELL, k_n=100.0, zeta_n=0.1, body_acceleration=(0.0, -1e-5),
                                 wall_axes=0b10)
    st = np.zeros((3, 28))
    st[:, 0], st[:, 1] = (40.0, 51.5, 200.0), (30.0, 34.0, 60.0)
    st[:, 3:5] = st[:, 0:2] - 0.01
    st[:, 26], st[:, 27] = 6.0, 1.5
    st[:, 24] = np.pi * 36 * 1.5
    st[:, 25] = 0.5 * st[:, 24] * 36
    runs = []
    for zeros in (False, True):
        lat, _, force = _lattice(9, dims, zeros, periodic=True)
        ps = Particles(lat, st)
        ps.step(prm, prog, 21)
        lat.upload_force(force)
        ps.step(prm, prog, 21)
        runs.append((ps.download(), lat.populations()))
        ps.close()
        lat.close()
    for a, b in zip(*runs):
        np.testing.assert_array_equal(a, b)
