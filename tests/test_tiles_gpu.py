"""Multi-step tiles of D2Q9 lattices against the one-step sweep: the same bits
for every collision, arithmetic and storage, with every boundary kind, on
extents around the tile edges, from even and odd time steps, bounded and
periodic, and for tiles of either shape.  (The one-step sweep itself is pinned
against the oracle and the golden vectors; a lattice whose launch shape was
asked for runs it for every step.)"""
import numpy as np
import pytest

from lbm_mirror_gb300 import capi as K
from tests import cases
from tests.gpu_util import make_lattice, with_arith

pytestmark = pytest.mark.gpu

COLLS = [K.KEL_COLL_BGK, K.KEL_COLL_BGK_GUO, K.KEL_COLL_PSM, K.KEL_COLL_PSM_GUO]


def both(case, arithmetic, storage, chunks):
    """Populations and macros after the chunks: multi-step default, one-step shape."""
    out = []
    for launch in (None, (1, 128)):
        lat = make_lattice(case, storage, launch)
        prog = with_arith(case["program"], arithmetic)
        for k, n in enumerate(chunks):
            lat.step(prog, n, write_macros=k % 2 == 1)
        out.append((lat.populations(), *lat.macros(), lat.t))
        lat.close()
    return out


def assert_same(a, b):
    assert a[3] == b[3]
    for x, y, what in zip(a[:3], b[:3], ("populations", "density", "velocity")):
        np.testing.assert_array_equal(x, y, err_msg=what)


@pytest.mark.parametrize("mode", ["fast", "reference", "fp16s"])
@pytest.mark.parametrize("collision", COLLS)
@pytest.mark.parametrize("periodic", [False, True])
def test_every_boundary_and_collision(mode, collision, periodic):
    case = cases.mixed_2d(collision, dims=(76, 45), periodic=periodic)
    arith = K.KEL_ARITH_REFERENCE if mode == "reference" else K.KEL_ARITH_FAST
    assert_same(*both(case, arith, "fp16s" if mode == "fp16s" else "fp32", (17, 3, 24)))


@pytest.mark.parametrize("dims", [(5, 3), (23, 4), (24, 5), (25, 9), (48, 1), (49, 2), (3, 200), (301, 13), (97, 24)])
def test_extents_around_the_tile_edges(dims):
    rng = np.random.default_rng(dims[0] * 1000 + dims[1])
    case = cases.mixed_2d(K.KEL_COLL_BGK, dims=(76, 45))
    n = dims[0] * dims[1]
    case.update(dims=dims, flags=rng.choice([0, 1, 2, 2, 2, 2, 5, 6, 7, 9], n).astype(np.uint8),
                init=cases.random_populations(9, n, rng))
    assert_same(*both(case, K.KEL_ARITH_FAST, "fp32", (1, 16, 9)))


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("collision", [K.KEL_COLL_BGK, K.KEL_COLL_BGK_GUO])
@pytest.mark.parametrize("mode", ["fast", "reference", "fp16s"])
def test_wide_tiles(mode, collision, periodic):
    dims = (2052, 733)  # above the size from which the wide tiles run; a last tile column of 36 cells, 29 rows
    rng = np.random.default_rng(7)
    case = cases.mixed_2d(collision, dims=(76, 45), periodic=periodic)
    n = dims[0] * dims[1]
    flags = np.full((dims[1], dims[0]), 2, np.uint8)
    flags[0] = flags[-1] = 1
    flags[rng.integers(0, dims[1], 900), rng.integers(0, dims[0], 900)] = 1
    if not periodic:
        flags[1:-1, 0], flags[1:-1, -1] = 4, 3
    case.update(dims=dims, flags=flags.reshape(-1), init=cases.random_populations(9, n, rng), force=None)
    arith = K.KEL_ARITH_REFERENCE if mode == "reference" else K.KEL_ARITH_FAST
    assert_same(*both(case, arith, "fp16s" if mode == "fp16s" else "fp32", (9, 12)))
