"""Channels of a batch on extents around warp and tile edges, where the sweep's
division-free row index, its per-warp interior path and its partial last tile
can go wrong: the same bits as the channel run alone as a lattice (which is
pinned against the oracle and the golden vectors), in both arithmetics that a
lattice has."""
import numpy as np
import pytest

from lbm_mirror_gb300 import Batch, Lattice
from lbm_mirror_gb300 import capi as K
from tests import cases

pytestmark = pytest.mark.gpu

EXTENTS = [(3, 3), (4, 3), (23, 5), (32, 8), (33, 7), (128, 3), (130, 9), (255, 4), (257, 5), (31, 130), (512, 33)]


@pytest.mark.parametrize("tile", [128, 256, 512])
@pytest.mark.parametrize("arithmetic", [K.KEL_ARITH_FAST, K.KEL_ARITH_REFERENCE])
def test_channels_equal_single_lattices(tile, arithmetic):
    rng = np.random.default_rng(5)
    chans = []
    for nx, ny in EXTENTS:
        f = cases.channel_flags((nx, ny)).reshape(ny, nx)
        f[rng.integers(0, ny, 3), rng.integers(0, nx, 3)] = 1
        chans.append(dict(nx=nx, ny=ny, tau=float(rng.uniform(0.6, 1.0)), u_max=0.04, flags=f))
    batch = Batch(chans, cases.channel_program(0.8, arithmetic), tile=tile)
    for n in (1, 6, 11):
        batch.step(n)
    for k, c in enumerate(chans):
        lat = Lattice("D2Q9", (c["nx"], c["ny"]))
        lat.set_launch(1, 128)
        lat.upload_flags(c["flags"])
        lat.upload_inlet_profile(cases.parabolic_profile(c["ny"], c["u_max"]))
        lat.step(cases.channel_program(c["tau"], arithmetic), 18)
        np.testing.assert_array_equal(batch.populations(k), lat.populations(), err_msg=f"channel {k} {EXTENTS[k]}")
        rho, u = batch.macros(k)
        want = lat.macros()
        np.testing.assert_array_equal(rho, want[0])
        np.testing.assert_array_equal(u, want[1])
        lat.close()
    batch.close()
