"""The contact and integration of a coupled step (kel_particles_step, PSM)
against the oracle: bodies a rounding apart to deeply overlapping, also across
the periodic seam and at walls, far from the origin, one and several sub-steps,
2D and 3D, ramp and sub-cell porosity.

Bounds, derived before the first run.  A force is the gather's sum (FP64; order
of summation: within 1e-12 of S = sum |cell force|; with the ramp porosity also
1e-6 S, the FP32 porosity's last bits) plus contacts, which both sides compute
in the same operations from the same states.  A contact that one side leaves out
shows: at the smallest depths drawn here, 1e-6, its force is above 1e-5."""
import numpy as np
import pytest

from lbm_mirror_gb300 import Lattice, Particles
from lbm_mirror_gb300 import capi as K
from oracle import oracle as O
from tests import cases

pytestmark = pytest.mark.gpu

OPS = {1: dict(bc=K.KEL_BC_BOUNCE_BACK), 2: dict(bc=K.KEL_BC_FLUID, collide=1)}
QNAME = {9: "D2Q9", 19: "D3Q19", 27: "D3Q27"}
# gap between two surfaces (negative: overlap)
GAPS = [-1.5, -0.3, -1e-3, -1e-5, -1e-6, -1e-9, -1e-13, 0.0, 1e-13, 1e-9, 1e-6, 1e-5, 1e-3, 0.4]


def _bodies(D, dims, periodic, rng):
    """Rows of pairs at the given gaps in seeded directions, one pair across the seam, bodies at the walls."""
    r = 4.0 if D == 2 else 3.0
    pos = []

    def pair(p, direction, gap):
        d = np.asarray(direction, float)
        d /= np.sqrt((d ** 2).sum())
        pos.append(np.array(p, float))
        pos.append(pos[-1] + d * (2 * r + gap))

    gaps = list(rng.permutation(GAPS))
    pitch = 4 * r + 4.0
    spots = [np.array(s) for s in np.ndindex(*(int((n - 2 * r - 8) // pitch) for n in dims))]
    spots = [spots[i] for i in rng.permutation(len(spots))][:len(gaps)]
    for s, gap in zip(spots, gaps):
        pair(r + 5.0 + s * pitch + rng.uniform(0, 1, D), rng.uniform(0.2, 1.0, D), gap)
    if periodic:  # across x = 0
        pair([dims[0] - 2.0] + [float(n) / 2 for n in dims[1:]], [1.0] + [0.1] * (D - 1), -1e-4)
        pos[-1][0] -= dims[0]
    return r, np.array(pos)


def _states(D, dims, periodic, walls, rng):
    r, pos = _bodies(D, dims, periodic, rng)
    edge = []  # bodies at the walls: distances around the radius
    for ax in range(D):
        if not walls >> ax & 1:
            continue
        for side in (0, 1):
            for k, gap in enumerate((-0.2, -1e-6, 1e-9)):
                p = np.array([dims[i] * (0.2 + 0.25 * k) for i in range(D)], float)
                p[ax] = r + gap if side == 0 else dims[ax] - r - gap
                edge.append(p)
    pos = np.concatenate([pos, np.array(edge)]) if edge else pos
    n = len(pos)
    st = np.zeros((n, 28))
    st[:, 0:D] = pos
    st[:, 3:3 + D] = pos - rng.uniform(-0.02, 0.02, (n, D))
    st[:, 6] = rng.uniform(-1, 1, n)
    st[:, 9] = st[:, 6] - rng.uniform(-0.01, 0.01, n)
    st[:, 15] = rng.uniform(-1e-4, 1e-4, n)  # 3D rotations keep it
    if D == 3:
        st[:, 7:9] = rng.uniform(-1, 1, (n, 2))
        st[:, 10:12] = st[:, 7:9] - rng.uniform(-0.01, 0.01, (n, 2))
        st[:, 16:18] = rng.uniform(-1e-4, 1e-4, (n, 2))
    st[:, 26], st[:, 27] = r, 1.5
    st[:, 24] = 1.5 * (np.pi * r * r if D == 2 else 4 / 3 * np.pi * r ** 3)
    st[:, 25] = 0.5 * st[:, 24] * r * r
    return st


@pytest.mark.parametrize("q,dims,periodic,walls", [(9, (160, 96), True, 0b10), (9, (157, 99), False, 0b11),
                                                   (9, (2048, 72), True, 0b10), (19, (72, 56, 48), False, 0b111),
                                                   (27, (64, 52, 56), True, 0b110)])
@pytest.mark.parametrize("sub_steps", [1, 3])
@pytest.mark.parametrize("mode", [K.KEL_POROSITY_SUBCELL, K.KEL_POROSITY_RAMP])
def test_coupled_steps_vs_oracle(q, dims, periodic, walls, sub_steps, mode):
    D = 2 if q == 9 else 3
    rng = np.random.default_rng(q + dims[0] + sub_steps)
    st0 = _states(D, dims, periodic, walls, rng)
    n = int(np.prod(dims))
    init = cases.random_populations(q, n, rng)
    flags = np.full(n, 2, np.uint8)
    prog = K.make_program(0.7, K.KEL_COLL_PSM, OPS, arithmetic=K.KEL_ARITH_REFERENCE)
    prm = K.make_particle_params(mode, sub_steps=sub_steps, k_n=100.0, zeta_n=0.1, gamma_t=0.05, mu=0.2,
                                 body_acceleration=(0.0, -1e-5, 2e-6), wall_axes=walls)
    o = O.OracleLattice(q, dims, periodic_x=periodic)
    o.set_flags(flags)
    o.set_populations(init.astype(np.float32).astype(np.float64))
    st = K.states_from_array(st0)
    lat = Lattice(QNAME[q], dims, periodic_x=periodic)
    lat.upload_flags(flags)
    lat.upload_populations(init.astype(np.float32))
    ps = Particles(lat, st0)
    loose = 1e-6 if mode == K.KEL_POROSITY_RAMP else 1e-12
    lever = 2 * st0[:, 26].max()
    bound_x = 0.0
    for step in range(3):
        ps.step(prm, prog, 1)
        O.particles_reset(st)
        o.particles_couple(st, prm)
        por = o.porosity()
        cell = np.abs(o.particles_gather(st, prm, want_cell_force=True)).sum()
        O.particles_contact(st, D, prm, dims, periodic_x=periodic)
        O.particles_integrate(st, D, prm, dims, periodic_x=periodic)
        o.run(prog, 1)
        got, ref = ps.download(), K.states_to_array(st)
        got_por = lat.download_field(K.KEL_FIELD_POROSITY, 1).astype(np.float64)
        if mode == K.KEL_POROSITY_SUBCELL:
            np.testing.assert_array_equal(got_por, por)
        else:
            assert np.abs(got_por - por).max() <= 1e-7 + 2 * bound_x
        # the force's error of this step; contacts pass on the positions' error so far (stiffness and damping)
        bound_f = loose * cell + 1e3 * bound_x
        assert np.abs(got[:, 18:21] - ref[:, 18:21]).max() <= bound_f, step
        assert np.abs(got[:, 21:24] - ref[:, 21:24]).max() <= lever * bound_f, step
        # position Verlet: a force error moves position by F / m, the error so far doubles and adds the one before
        bound_x = 3 * bound_x + bound_f * max(1 / st0[:, 24].min(), 1 / st0[:, 25].min() * lever) + 1e-12
        for a, b, what in ((0, 3, "position"), (3, 6, "position before"), (6, 9, "rotation"), (9, 12, "rotation before")):
            assert np.abs(got[:, a:b] - ref[:, a:b]).max() <= bound_x, (step, what)
        for a, b in ((12, 15), (15, 18)):
            assert np.abs(got[:, a:b] - ref[:, a:b]).max() <= bound_f * max(1 / st0[:, 24].min(), lever / st0[:, 25].min()) + 1e-15
        np.testing.assert_array_equal(got[:, 24:], ref[:, 24:])
    ps.close()
    lat.close()
