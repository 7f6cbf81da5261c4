"""Which D2Q9 lattices take the multi-step tiles, and of which shape: both sides of
every line of the rule (cells covered, populations in shares of the device's L2,
columns against rows, boundary kinds, collision, storage, arithmetic, named shape)."""
import numpy as np
import pytest

from lbm_mirror_gb300 import Lattice
from lbm_mirror_gb300 import capi as K

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

BGK, GUO, PSM, PSM_GUO = K.KEL_COLL_BGK, K.KEL_COLL_BGK_GUO, K.KEL_COLL_PSM, K.KEL_COLL_PSM_GUO
OPS = {1: dict(bc=K.KEL_BC_BOUNCE_BACK), 2: dict(bc=K.KEL_BC_FLUID, collide=1),
       4: dict(bc=K.KEL_BC_ZOUHE_PRESSURE_X, collide=1, east=0)}


def _tiles(dims, collision=BGK, opened=False, storage="fp32", arithmetic=K.KEL_ARITH_FAST, launch=None):
    lat = Lattice("D2Q9", dims, storage=storage)
    if launch:
        lat.set_launch(*launch)
    f = np.full((dims[1], dims[0]), 2, np.uint8)
    f[[0, -1]] = 1
    if opened:
        f[1:-1, -1] = 4
    lat.upload_flags(f.reshape(-1))
    lat.step(K.make_program(0.8, collision, OPS, arithmetic=arithmetic), 0)
    t = lat.tiles()
    lat.close()
    return t


SMALL, NONE = (4, 24), (1, 0)


@pytest.mark.parametrize("want,dims,kw", [
    (SMALL, (256, 64), {}), (SMALL, (256, 64), dict(opened=True, collision=PSM_GUO)),
    (SMALL, (256, 64), dict(opened=True, storage="fp16s")),
    (SMALL, (512, 128), dict(opened=True)), (SMALL, (512, 128), dict(opened=True, collision=PSM)),
    (NONE, (512, 128), dict(opened=True, collision=GUO)), (SMALL, (512, 128), dict(collision=PSM_GUO)),
    (SMALL, (512, 128), dict(opened=True, collision=GUO, storage="fp16s")),
    (NONE, (512, 128), dict(opened=True, collision=PSM_GUO, storage="fp16s")),
    (NONE, (64, 1024), dict(opened=True)), (SMALL, (64, 1024), {}),
    (NONE, (333, 290), dict(opened=True)), (SMALL, (333, 290), {}), (NONE, (340, 300), {}),
    (NONE, (256, 64), dict(arithmetic=K.KEL_ARITH_REFERENCE)), (NONE, (256, 64), dict(launch=(1, 128)))])
def test_small(want, dims, kw):
    assert _tiles(dims, **kw)[:2] == want


WIDE = (4, 56)


@pytest.mark.parametrize("want,nx,share,kw", [
    (NONE, 2053, 0.85, {}), (WIDE, 2053, 0.95, {}), (WIDE, 2053, 0.95, dict(opened=True)),
    (WIDE, 2053, 0.95, dict(collision=PSM)), (NONE, 2053, 0.95, dict(collision=PSM, opened=True)),
    (WIDE, 2053, 1.2, dict(collision=PSM, opened=True)), (NONE, 2053, 1.5, dict(collision=GUO)),
    (WIDE, 2053, 1.9, dict(collision=GUO, opened=True)), (NONE, 2053, 1.9, dict(collision=PSM_GUO)),
    (NONE, 2053, 1.9, dict(storage="fp16s")), (NONE, 2053, 1.9, dict(arithmetic=K.KEL_ARITH_REFERENCE)),
    (WIDE, 512, 1.0, dict(opened=True)), (NONE, 200, 1.0, dict(opened=True)), (WIDE, 120, 1.0, {}),
    (NONE, 64, 1.0, {}), (NONE, 512, 1.9, dict(collision=GUO))])
def test_wide(want, nx, share, kw):
    size = 9 * (2 if kw.get("storage") == "fp16s" else 4) * ((nx + 7) // 8 * 8)
    ny = int(share * torch.cuda.get_device_properties(0).L2_cache_size / size)
    assert _tiles((nx, ny), **kw)[:2] == want
