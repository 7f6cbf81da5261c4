"""The reference-arithmetic equilibrium (FP32 pair sums with an FP64 branch) has
the reference's bits: every population of an equilibrium start equals the
double-bracket formula (equilibrium.hpp:7-48) evaluated by numpy, for velocities
on both sides of the bound up to which the FP32 sums are used, tiny and
subnormal ones, densities of any size and sign, infinities and NaN."""
import numpy as np
import pytest

from lbm_mirror_gb300 import Lattice
from oracle import oracle as O
from tests import cases

NAME = {9: "D2Q9", 19: "D3Q19", 27: "D3Q27"}


def reference_equilibrium(q, rho, u):
    """(n, q) float32: the reference's rounding sequence."""
    c, w = directions(q)
    D = u.shape[0]
    vv = u[0] * u[0]
    for k in range(1, D):
        vv = vv + u[k] * u[k]
    out = np.empty((rho.size, q), np.float32)
    for i in range(q):
        vc = np.zeros_like(rho)
        for k in range(D):
            if c[i][k] > 0:
                vc = vc + u[k]
            if c[i][k] < 0:
                vc = vc - u[k]
        vcc = vc * np.float32(3)
        br = 1.0 + vcc.astype(np.float64) - 1.5 * vv.astype(np.float64) + (vcc * vcc).astype(np.float64) * 0.5
        out[:, i] = ((np.float32(w[i]) * rho).astype(np.float64) * br).astype(np.float32)
    return out


def directions(q):
    """Directions in the order of the AoS populations, and weights."""
    if q == 9:
        c = [(0, 0), (-1, 0), (1, 0), (0, -1), (0, 1), (-1, -1), (1, 1), (-1, 1), (1, -1)]
    elif q == 19:
        c = [(0, 0, 0), (-1, 0, 0), (1, 0, 0), (0, -1, 0), (0, 1, 0), (0, 0, -1), (0, 0, 1), (-1, -1, 0), (1, -1, 0),
             (-1, 1, 0), (1, 1, 0), (-1, 0, -1), (1, 0, -1), (-1, 0, 1), (1, 0, 1), (0, -1, -1), (0, 1, -1),
             (0, -1, 1), (0, 1, 1)]
    else:
        o = (0, -1, 1)
        c = [(o[i % 3], o[i // 3 % 3], o[i // 9]) for i in range(27)]
    return c, cases._weights(q)


def fields(D, n, rng):
    rho = (1.0 + 0.1 * rng.standard_normal(n)).astype(np.float32)
    u = (0.05 * rng.standard_normal((D, n))).astype(np.float32)
    k = n // 8
    u[:, k:2 * k] = rng.uniform(-0.2, 0.2, (D, k)).astype(np.float32)  # around the bound on u^2
    u[:, 2 * k:3 * k] *= (10.0 ** rng.uniform(-44, 0, k)).astype(np.float32)  # down to subnormals
    u[:, 3 * k:4 * k] = 0.0
    rho[4 * k:5 * k] = (2.0 ** rng.uniform(-149, 127, k)).astype(np.float32)
    rho[5 * k:5 * k + k // 2] *= -1.0
    u[:, 5 * k + k // 2:6 * k] *= np.float32(100.0)
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 3e38, 1e-45], np.float32)
    m = special.size
    rho[6 * k:6 * k + m] = special
    u[0, 6 * k + m:6 * k + 2 * m] = special
    return rho, u


def test_the_formula_is_the_oracles():
    for q in (9, 19, 27):
        D = 2 if q == 9 else 3
        rho, u = fields(D, 4096, np.random.default_rng(q))
        want = reference_equilibrium(q, rho[:512], u[:, :512])
        for c in range(0, 512, 37):
            np.testing.assert_array_equal(want[c], O.equilibrium_f32(q, rho[c], u[:, c].copy()))


@pytest.mark.gpu
@pytest.mark.parametrize("q", [9, 19, 27])
def test_equilibrium_bits_equal_the_double_bracket(q):
    torch = pytest.importorskip("torch")
    D = 2 if q == 9 else 3
    dims = (512, 1024) if q == 9 else (64, 64, 64)
    n = int(np.prod(dims))
    rho, u = fields(D, n, np.random.default_rng(1000 + q))
    lat = Lattice(NAME[q], dims)
    dr, du = torch.from_numpy(rho).cuda(), torch.from_numpy(u.copy()).cuda()
    torch.cuda.synchronize()
    lat.init_equilibrium(d_rho=dr.data_ptr(), d_u=du.data_ptr())
    got = lat.populations(np.float32)
    lat.close()
    with np.errstate(all="ignore"):
        want = reference_equilibrium(q, rho, u)
    same = (got == want) | (np.isnan(got) & np.isnan(want))
    assert same.all(), f"{(~same).sum()} of {same.size} populations differ"
