"""The wide tiles of D2Q9 lattices beyond the L2 (FP32) against the one-step sweep:
the same bits for every collision that takes them, bounded and periodic, with every
boundary kind anywhere on the tiles, last tiles that are ragged in both
directions, from even and odd time steps.  The extents follow from the device's
L2, and the lattice's tiles are asked for, so that a lattice that takes others
(or none) fails the test.  Reference arithmetic takes none."""
import numpy as np
import pytest

from lbm_mirror_gb300 import capi as K
from tests import cases
from tests.gpu_util import make_lattice, with_arith

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# share of the L2 from which a collision takes wide tiles, and some more
COLLS = {K.KEL_COLL_BGK: 0.95, K.KEL_COLL_PSM: 1.2, K.KEL_COLL_BGK_GUO: 1.8}


def _case(collision, periodic):
    l2 = torch.cuda.get_device_properties(0).L2_cache_size
    nx = 2052 if periodic else 2053  # 36 or 37 columns of 56 and a part
    ny = int(COLLS[collision] * l2) // (36 * nx) | 1
    rng = np.random.default_rng(11)
    case = cases.mixed_2d(collision, dims=(76, 45), periodic=periodic)
    n = nx * ny
    flags = np.full((ny, nx), 2, np.uint8)
    flags.reshape(-1)[rng.integers(0, n, n // 150)] = rng.choice([0, 1, 1, 5, 6, 7], n // 150)
    flags[0], flags[-1] = 1, 5
    flags[0, 40:90] = 6
    if not periodic:
        flags[1:-1, 0], flags[1:-1, -1] = 4, 3
    case.update(dims=(nx, ny), flags=flags.reshape(-1), init=cases.random_populations(9, n, rng))
    if case["porosity"] is not None:
        por = rng.uniform(0.0, 1.0, n)
        por[rng.uniform(size=n) < 0.4] = 1.0
        case["porosity"] = por
    if case["force"] is not None:
        case["force"] = 1e-4 * rng.standard_normal(n * 2)
    return case


def _run(case, prog, launch):
    lat = make_lattice(case, launch=launch)
    for k, n in enumerate((9, 12)):
        lat.step(prog, n, write_macros=k == 1)
    out = (lat.populations(), *lat.macros(), lat.t)
    tiles = lat.tiles()
    lat.close()
    return out, tiles


@pytest.mark.parametrize("collision", list(COLLS))
@pytest.mark.parametrize("periodic", [False, True])
def test_wide_tiles_equal_the_one_step_sweep(collision, periodic):
    case = _case(collision, periodic)
    prog = with_arith(case["program"], K.KEL_ARITH_FAST)
    a, tiles = _run(case, prog, None)
    assert tiles[0] == 4 and tiles[1] == 56, tiles
    b, none = _run(case, prog, (1, 128))
    assert none[0] == 1, none
    assert a[3] == b[3] == 21
    for x, y, what in zip(a[:3], b[:3], ("populations", "density", "velocity")):
        np.testing.assert_array_equal(x.view(np.uint32), y.view(np.uint32), err_msg=what)

