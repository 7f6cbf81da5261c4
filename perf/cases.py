"""The work that programs have this library do, as cases that can be timed and compared.

Each case is one pass through the public entry points (lbm_mirror_gb300.lattice and the C ABI of
include/kel_lbm_cuda.h): a lattice advanced some steps and its density and velocity read back, a batch of
channels advanced or run towards its steady state, a particle-laden channel, a training step and an
inference of the warm-start U-Net.

    listed()            the cases by name
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what a program holds before the call
    run(state)          one pass and its outputs
    work(case)          bytes and operations of a pass
    exact(case, seed)   the outputs in 64 bits, by torch alone
"""
import ctypes as C
import math

import numpy as np
import torch

from lbm_mirror_gb300 import Batch, Lattice, Particles, UNet
from lbm_mirror_gb300 import capi as K

# ---- the lattices' direction tables (order of the AoS populations) ------------------------------


def _tables(q):
    """Directions (q, 3) and weights (q,) of the descriptor, in the order of its AoS populations."""
    if q == 9:
        c = [(0, 0), (-1, 0), (1, 0), (0, -1), (0, 1), (-1, -1), (1, 1), (-1, 1), (1, -1)]
        c = [(x, y, 0) for x, y in c]
        w = [4 / 9] + [1 / 9] * 4 + [1 / 36] * 4
    elif q == 19:
        c = [(0, 0, 0), (-1, 0, 0), (1, 0, 0), (0, -1, 0), (0, 1, 0), (0, 0, -1), (0, 0, 1)]
        c += [(-1, -1, 0), (1, -1, 0), (-1, 1, 0), (1, 1, 0), (-1, 0, -1), (1, 0, -1), (-1, 0, 1), (1, 0, 1)]
        c += [(0, -1, -1), (0, 1, -1), (0, -1, 1), (0, 1, 1)]
        w = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
    else:
        o = (0, -1, 1)
        c = [(o[i % 3], o[i // 3 % 3], o[i // 9]) for i in range(27)]
        w = [(8 / 27, 2 / 27, 1 / 54, 1 / 216)[sum(k != 0 for k in v)] for v in c]
    return c, w


def _opposite(c):
    return [c.index(tuple(-k for k in v)) for v in c]


# ---- the cases ----------------------------------------------------------------------------------


def listed():
    return [
        # the Poiseuille channel of the drivers (256x64): the smallest lattice in use, bound by latency
        _lattice("poiseuille_d2q9_256x64", 9, 256, 64, 1, "channel", steps=400, pops=True),
        # a 2D channel with obstacles and odd extents, advanced in the blocks between two file outputs
        _lattice("channel_d2q9_1021x347", 9, 1021, 347, 1, "channel", steps=40, calls=5, obstacles=6, pops=True),
        # a 3D lattice that fits the L2 cache: an ordinary trial run
        _lattice("cavity_d3q19_64", 19, 64, 64, 64, "cavity", steps=100, pops=True),
        # the headline: lid-driven cavity, FP32
        _lattice("cavity_d3q19_256", 19, 256, 256, 256, "cavity", steps=40),
        # the same cavity in half-precision storage
        _lattice("cavity_d3q19_256_fp16s", 19, 256, 256, 256, "cavity", steps=40, storage="fp16s"),
        # D3Q27 with a body force on ragged extents, macros and populations read back
        _lattice("force_d3q27_173x131x97", 27, 173, 131, 97, "force", steps=24, pops=True),
        # a run that has to match the reference bit for bit (its rounding sequence)
        _lattice("cavity_d3q19_128_reference", 19, 128, 128, 128, "cavity", steps=12, arithmetic="reference"),
        # many uneven channels advanced together (a parameter sweep)
        dict(name="batch_192", kind="batch", channels=192, nx_lo=64, nx_hi=512, ny_lo=32, ny_hi=128, steps=800,
             arithmetic="fast"),
        # channels of one size run towards the steady state: the training data of the warm start
        dict(name="batch_until_64", kind="until", channels=64, nx_lo=256, nx_hi=256, ny_lo=64, ny_hi=64, check=500,
             steps=2000, arithmetic="shifted"),
        # the particle-laden channel: PSM + gravity, 64 discs, sub-cell solid fraction
        dict(name="particles_2048x512", kind="particles", nx=2048, ny=512, bodies=64, radius=8.0, steps=50),
        # one training step of the warm-start network at its training batch
        dict(name="unet_train_256x64_b32", kind="train", nx=256, ny=64, batch=32, w0=32, w1=64, w2=128, w3=128),
        # inference of the wider network on a handful of geometries
        dict(name="unet_infer_256x64_b8", kind="infer", nx=256, ny=64, batch=8, w0=48, w1=96, w2=128, w3=128),
    ]


def _lattice(name, q, nx, ny, nz, flow, steps, calls=1, storage="fp32", arithmetic="fast", obstacles=0, pops=False):
    """A lattice advanced `calls` times by `steps` steps; the macros (and populations) are read at the end."""
    c = dict(kind="lattice", q=q, nx=nx, ny=ny, nz=nz, flow=flow, steps=steps, calls=calls, storage=storage,
             arithmetic=arithmetic, obstacles=obstacles, pops=pops)
    return dict(c, name=name) if name else c


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lattice2", "lattice2", "lattice3", "lattice3", "lattice3", "batch", "until", "particles", "net"])
    if kind == "lattice2":
        flow = rng.choice(["channel", "channel", "cavity", "force"])
        nx, ny = _log_int(rng, 48, 2048), _log_int(rng, 20, 1024)
        if flow == "force":
            nx = (nx + 3) // 4 * 4  # periodic rows
        arithmetic = rng.choice(["fast", "fast", "reference"])
        storage = rng.choice(["fp32", "fp32", "fp16s"]) if arithmetic == "fast" and flow != "force" else "fp32"
        return _lattice(None, 9, nx, ny, 1, flow, steps=_log_int(rng, 4, 400), calls=rng.choice([1, 1, 3]),
                        storage=storage, arithmetic=arithmetic, obstacles=rng.randint(0, 8) if flow == "channel" else 0,
                        pops=rng.random() < 0.5)
    if kind == "lattice3":
        q, flow = rng.choice([19, 19, 27]), rng.choice(["cavity", "cavity", "force"])
        n = [_log_int(rng, 24, 250) for _ in range(3)]
        if flow == "force" and rng.random() < 0.5:
            n[0] = (n[0] + 3) // 4 * 4  # the periodic form (else walled in x)
        cells = n[0] * n[1] * n[2]
        arithmetic = rng.choice(["fast", "fast", "fast", "reference"]) if cells < 3_000_000 else "fast"
        storage = rng.choice(["fp32", "fp16s"]) if arithmetic == "fast" and flow == "cavity" else "fp32"
        most = max(4, min(60, int(6e8 / cells / (4 if arithmetic == "reference" else 1))))
        return _lattice(None, q, n[0], n[1], n[2], flow, steps=_log_int(rng, 3, most), storage=storage,
                        arithmetic=arithmetic, pops=cells < 4_000_000 and rng.random() < 0.5)
    if kind == "batch":
        lo, hi = rng.randint(48, 128), rng.randint(160, 512)
        return dict(kind="batch", channels=_log_int(rng, 4, 190), nx_lo=lo, nx_hi=hi, ny_lo=rng.randint(24, 40),
                    ny_hi=rng.randint(48, 128), steps=_log_int(rng, 50, 800),
                    arithmetic=rng.choice(["fast", "shifted", "reference"]) if rng.random() < 0.7 else "fast")
    if kind == "until":
        nx, ny = rng.randint(64, 320), rng.randint(32, 96)
        return dict(kind="until", channels=_log_int(rng, 2, 60), nx_lo=nx, nx_hi=nx, ny_lo=ny, ny_hi=ny,
                    check=2 * rng.randint(50, 250), steps=1000, arithmetic="shifted")
    if kind == "particles":
        nx, ny = 4 * rng.randint(64, 512), rng.randint(128, 512)
        r = round(rng.uniform(4.0, 9.0), 2)
        return dict(kind="particles", nx=nx, ny=ny, bodies=max(1, min(96, int(nx * ny / (r * r) / rng.uniform(200, 400)))),
                    radius=r, steps=2 * rng.randint(4, 25))
    w0 = 16 * rng.randint(1, 3)
    return dict(kind=rng.choice(["train", "infer"]), nx=rng.choice([64, 128, 256]), ny=8 * rng.randint(2, 8),
                batch=rng.randint(1, 32), w0=w0, w1=2 * w0, w2=128 if w0 > 16 else 64, w3=128)


# ---- inputs, the same for prepare() and exact() ----------------------------------------------------


def _dims(case):
    return (case["nx"], case["ny"]) if case["q"] == 9 else (case["nx"], case["ny"], case["nz"])


def _periodic(case):
    return case["kind"] == "particles" or (case["flow"] == "force" and case["nx"] % 4 == 0)


def _obstacles(f, n, rng):
    """n discs and rectangles in the flag rows f (ny, nx), clear of the ends and of the walls."""
    ny, nx = f.shape
    if nx < 40 or ny < 24:
        return
    y, x = np.ogrid[:ny, :nx]
    for _ in range(n):
        r = rng.uniform(1.5, min(12.0, ny / 8.0))
        cx, cy = rng.uniform(12 + r, nx - 12 - r), rng.uniform(5 + r, ny - 6 - r)
        if rng.uniform() < 0.5:
            f[(x - cx) ** 2 + (y - cy) ** 2 <= r * r] = 1
        else:
            f[int(cy - r):int(cy + r) + 1, int(cx - r / 2):int(cx + r / 2) + 1] = 1


def _flags(case, seed):
    """Flags (nz, ny, nx): 1 wall, 2 fluid, 3 inlet, 4 outlet, 5 lid."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    f = np.full((nz, ny, nx), 2, np.uint8)
    f[:, 0] = f[:, -1] = 1
    if nz > 1:
        f[0] = f[-1] = 1
    inner_z = slice(1, -1) if nz > 1 else slice(None)
    if case["flow"] == "cavity":
        f[:, :, 0] = f[:, :, -1] = 1
        f[inner_z, -1, 1:-1] = 5
    elif case["flow"] == "channel":
        f[inner_z, 1:-1, 0] = 3
        f[inner_z, 1:-1, -1] = 4
        _obstacles(f[0], case["obstacles"], np.random.default_rng(seed))
    elif not _periodic(case):
        f[:, :, 0] = f[:, :, -1] = 1
    return f


def _profile(ny, u_max):
    eta = (np.arange(ny) - 0.5) / (ny - 2)
    u = 4.0 * u_max * eta * (1.0 - eta)
    u[0] = u[-1] = 0.0
    return u


FORCE = (3e-6, -2e-6, 1e-6)
LID = (0.1, 0.0, 0.0)


def _constants(case, seed):
    """Relaxation time and inlet velocity of a lattice case."""
    rng = np.random.default_rng(seed + 17)
    tau = {"channel": 0.7, "cavity": 0.56, "force": 0.65, "particles": 0.8}[case.get("flow", "particles")]
    return float(tau + 0.02 * rng.uniform()), float(rng.uniform(0.03, 0.05))


def _start_fields(nx, ny, nz, D, seed):
    """Smooth seeded density (n,) and velocity (D, n) in FP32 on the GPU."""
    g = np.random.default_rng(seed + 29)
    x = torch.arange(nx, device="cuda", dtype=torch.float32) * (2 * math.pi / nx)
    y = torch.arange(ny, device="cuda", dtype=torch.float32) * (2 * math.pi / ny)
    z = torch.arange(nz, device="cuda", dtype=torch.float32) * (2 * math.pi / nz)
    planes = []
    for k in range(D + 1):
        a = g.integers(1, 4, 3)
        p = g.uniform(0, 2 * math.pi, 3)
        s = (torch.sin(float(a[0]) * x + float(p[0]))[None, None, :] * torch.sin(float(a[1]) * y + float(p[1]))[None, :, None]
             * (torch.sin(float(a[2]) * z + float(p[2]))[:, None, None] if nz > 1 else 1.0))
        planes.append((1.0 + 0.004 * s if k == 0 else 0.02 * s).reshape(-1))
    return planes[0].contiguous(), torch.stack(planes[1:]).contiguous()


def _ops():
    return {1: dict(bc=K.KEL_BC_BOUNCE_BACK), 2: dict(bc=K.KEL_BC_FLUID, collide=1),
            3: dict(bc=K.KEL_BC_ZOUHE_VELOCITY_X, collide=1, east=1, use_profile=1),
            4: dict(bc=K.KEL_BC_ZOUHE_PRESSURE_X, collide=1, east=0, rho=1.0), 5: dict(bc=K.KEL_BC_MOVING_WALL, u=LID)}


def _channels(case, seed):
    """Channel descriptions: the sizes go with the case, obstacles, relaxation time and inlet with the seed."""
    sizes, rng = np.random.default_rng(case["channels"]), np.random.default_rng(seed + 41)
    out = []
    for _ in range(case["channels"]):
        nx = int(sizes.integers(case["nx_lo"], case["nx_hi"] + 1))
        ny = int(sizes.integers(case["ny_lo"], case["ny_hi"] + 1))
        f = np.full((ny, nx), 2, np.uint8)
        f[0] = f[-1] = 1
        f[1:-1, 0], f[1:-1, -1] = 3, 4
        _obstacles(f, int(rng.integers(0, 5)), rng)
        out.append(dict(nx=nx, ny=ny, tau=float(rng.uniform(0.6, 1.0)), u_max=float(rng.uniform(0.01, 0.06)), flags=f))
    return out


def _bodies(case, seed):
    """Disc states (n, 28) on a jittered grid, at least three cells apart, moving slowly."""
    rng = np.random.default_rng(seed + 53)
    nx, ny, n, r = case["nx"], case["ny"], case["bodies"], case["radius"]
    pitch = 2 * r + 5.0
    spots = [(i, j) for i in range(int(nx // pitch)) for j in range(int((ny - 2 * r - 10) // pitch) + 1)]
    st = np.zeros((n, 28))
    for k, s in enumerate(rng.permutation(len(spots))[:n]):
        i, j = spots[s]
        p = (np.array([i * pitch + pitch / 2, j * pitch + r + 4.0]) + rng.uniform(-1.0, 1.0, 2))
        v = rng.uniform(-0.004, 0.004, 2)
        m = math.pi * r * r * 1.5
        st[k, 0:2], st[k, 3:5] = p, p - v
        st[k, 9] = -rng.uniform(-2e-4, 2e-4)  # previous angle: a slow spin
        st[k, 24:28] = m, 0.5 * m * r * r, r, 1.5
    return st[:len(spots)]


GRAVITY = 1e-6
TOL = 1e-11  # below what the channels reach: a pass is the same stretch of a longer run each time


def _layers(case):
    w = [case["w%d" % k] for k in range(4)]
    convs, c = [], 16
    for l in range(3):
        convs += [(w[l], 3, c), (w[l], 3, w[l])]
        c = w[l]
    convs += [(w[3], 3, c), (w[3], 3, w[3])]
    up = w[3]
    for l in (2, 1, 0):
        convs += [(w[l], 3, up + w[l]), (w[l], 3, w[l])]
        up = w[l]
    return convs + [(3, 1, w[0])]


def _weights(case, seed):
    """Flat FP32 parameters: per layer [c_out][ky][kx][c_in], then the biases."""
    g = torch.Generator().manual_seed(seed + 61)
    parts = []
    for co, k, ci in _layers(case):
        bound = math.sqrt(6.0 / (k * k * ci))
        parts += [(torch.rand(co * k * k * ci, generator=g) * 2 - 1) * bound, (torch.rand(co, generator=g) - 0.5) * 0.02]
    return torch.cat(parts)


def _net_inputs(case, seed):
    """Masks (b, ny, nx), u_max, tau and targets (b, ny, nx, 3) on the GPU."""
    rng = np.random.default_rng(seed + 71)
    b, ny, nx = case["batch"], case["ny"], case["nx"]
    mask = np.zeros((b, ny, nx), np.uint8)
    mask[:, 0] = mask[:, -1] = 1
    for k in range(b):
        _obstacles(mask[k], int(rng.integers(1, 6)), rng)
    mask = torch.from_numpy(mask).cuda()
    u = torch.from_numpy(rng.uniform(0.01, 0.08, b).astype(np.float32)).cuda()
    tau = torch.from_numpy(rng.uniform(0.55, 1.0, b).astype(np.float32)).cuda()
    g = torch.Generator(device="cuda").manual_seed(seed + 73)
    target = torch.randn((b, ny, nx, 3), device="cuda", generator=g) * 0.3
    return mask, u, tau, target * (1 - mask[..., None].float())


# ---- prepare and run -------------------------------------------------------------------------------


def _host(*shape):
    return torch.empty(shape, dtype=torch.float32, pin_memory=True)


def _p(t):
    return C.c_void_p(t.data_ptr())


def _ok(rc, lib):
    if rc != K.KEL_OK:
        raise RuntimeError(lib.kel_last_error_string().decode())


_ARITH = {"fast": K.KEL_ARITH_FAST, "reference": K.KEL_ARITH_REFERENCE, "shifted": K.KEL_ARITH_SHIFTED}


def prepare(case, seed):
    s = {"case": case, "lib": K.load_library()}
    kind = case["kind"]
    if kind == "lattice":
        tau, u_max = _constants(case, seed)
        s["stream"] = torch.cuda.Stream()
        lat = Lattice({9: "D2Q9", 19: "D3Q19", 27: "D3Q27"}[case["q"]], _dims(case), storage=case["storage"],
                      periodic_x=_periodic(case), stream=s["stream"].cuda_stream)
        lat.upload_flags(_flags(case, seed))
        if case["flow"] == "channel":
            lat.upload_inlet_profile(_profile(case["ny"], u_max))
        D = 2 if case["q"] == 9 else 3
        rho, u = _start_fields(case["nx"], case["ny"], case["nz"], D, seed)
        torch.cuda.synchronize()
        lat.init_equilibrium(d_rho=rho.data_ptr(), d_u=u.data_ptr())
        s["lat"] = lat
        s["program"] = K.make_program(tau, K.KEL_COLL_BGK_GUO if case["flow"] == "force" else K.KEL_COLL_BGK, _ops(),
                                      global_force=FORCE[:D] if case["flow"] == "force" else (0.0, 0.0, 0.0),
                                      arithmetic=_ARITH[case["arithmetic"]])
        s["rho"], s["u"] = _host(lat.n), _host(lat.n, D)
        s["f"] = _host(lat.n, case["q"]) if case["pops"] else None
    elif kind in ("batch", "until"):
        ch = _channels(case, seed)
        ops = {k: v for k, v in _ops().items() if k < 5}
        s["batch"] = Batch(ch, K.make_program(0.8, K.KEL_COLL_BGK, ops, arithmetic=_ARITH[case["arithmetic"]]))
    elif kind == "particles":
        tau, _ = _constants(case, seed)
        s["stream"] = torch.cuda.Stream()
        lat = Lattice("D2Q9", (case["nx"], case["ny"]), periodic_x=True, stream=s["stream"].cuda_stream)
        f = np.full((case["ny"], case["nx"]), 2, np.uint8)
        f[0] = f[-1] = 1
        lat.upload_flags(f)
        s["lat"], s["bodies"] = lat, Particles(lat, _bodies(case, seed))
        s["program"] = K.make_program(tau, K.KEL_COLL_PSM_GUO, {1: dict(bc=K.KEL_BC_BOUNCE_BACK), 2: dict(bc=K.KEL_BC_FLUID, collide=1)},
                                      global_force=(0.0, -GRAVITY, 0.0))
        s["params"] = K.make_particle_params(K.KEL_POROSITY_SUBCELL, sub_steps=1, k_n=100.0, zeta_n=0.1,
                                             body_acceleration=(0.0, -GRAVITY), wall_axes=0b10)
        s["rho"], s["u"] = _host(lat.n), _host(lat.n, 2)
    else:
        net = UNet(height=case["ny"], width=case["nx"], widths=tuple(case["w%d" % k] for k in range(4)),
                   max_batch=case["batch"], seed=1)
        net.set_params(_weights(case, seed).numpy())
        s["net"] = net
        s["mask"], s["umax"], s["tau"], s["target"] = _net_inputs(case, seed)
        s["out"] = torch.empty((case["batch"], case["ny"], case["nx"], 3), device="cuda")
        s["grads"], s["weights"] = _host(net.n_params), _host(net.n_params)
        torch.cuda.synchronize()
    return s


def run(s):
    case, lib, kind = s["case"], s["lib"], s["case"]["kind"]
    if kind == "lattice":
        lat = s["lat"]
        for k in range(case["calls"]):
            lat.step(s["program"], case["steps"], write_macros=k + 1 == case["calls"])
        # page-locked host buffers, as a program that writes its fields keeps them
        _ok(lib.kel_download_macros(lat.handle, _p(s["rho"]), _p(s["u"])), lib)
        out = {"rho": s["rho"], "u": s["u"]}
        if s["f"] is not None:
            _ok(lib.kel_download_populations(lat.handle, _p(s["f"]), K.KEL_DTYPE_F32, K.KEL_LAYOUT_AOS), lib)
            out["f"] = s["f"]
        return out
    if kind in ("batch", "until"):
        b = s["batch"]
        out = {}
        if kind == "batch":
            b.step(case["steps"])
        else:
            out["steps"], out["residual"] = b.run_until(tol=TOL, check_every=case["check"], max_steps=case["steps"])
            out["steps"] = out["steps"].astype(np.int64)
        fields = [b.macros(c) for c in range(b.n)]
        out["rho"] = np.concatenate([r for r, _ in fields])
        out["u"] = np.concatenate([u for _, u in fields])
        return out
    if kind == "particles":
        lat = s["lat"]
        s["bodies"].step(s["params"], s["program"], case["steps"])
        _ok(lib.kel_download_macros(lat.handle, _p(s["rho"]), _p(s["u"])), lib)
        return {"rho": s["rho"], "u": s["u"], "bodies": s["bodies"].download()}
    net, n = s["net"], case["batch"]
    net.make_input(s["mask"].data_ptr(), s["umax"].data_ptr(), s["tau"].data_ptr(), n)
    if kind == "infer":
        net.forward(n, s["out"].data_ptr())
        net.synchronize()
        return s["out"]
    net.train_step(s["target"].data_ptr(), n, lr=1e-3)
    _ok(lib.kel_unet_get_grads(net._h, _p(s["grads"])), lib)
    _ok(lib.kel_unet_get_params(net._h, _p(s["weights"])), lib)
    return {"loss": net.last_loss(), "grads": s["grads"], "weights": s["weights"]}


# ---- work ------------------------------------------------------------------------------------------

_FLOPS = {9: 130, 19: 300, 27: 430}  # moments, equilibrium and relaxation of one cell


def work(case):
    """A lattice's time step reads and writes every population once and reads the flag; a call's last step
    writes the macros, which are then read back.  The U-Net's products count twice, three times in training."""
    kind = case["kind"]
    if kind == "lattice":
        n, q, size = case["nx"] * case["ny"] * case["nz"], case["q"], 2 if case["storage"] == "fp16s" else 4
        D = 2 if q == 9 else 3
        steps = case["steps"] * case["calls"]
        field = 4 * D if case["flow"] == "force" else 0
        return {"bytes": n * (steps * (2 * q * size + 1 + field) + 8 * (1 + D) + (q * (size + 4) if case["pops"] else 0)),
                "flops": n * steps * _FLOPS[q]}
    if kind in ("batch", "until"):
        n = sum(c["nx"] * c["ny"] for c in _channels(case, 0))
        return {"bytes": n * (case["steps"] * 73 + 24), "flops": n * case["steps"] * _FLOPS[9]}
    if kind == "particles":
        n = case["nx"] * case["ny"]
        return {"bytes": n * (case["steps"] * (73 + 4) + 24), "flops": n * case["steps"] * (_FLOPS[9] + 80)}
    b, ny, nx = case["batch"], case["ny"], case["nx"]
    layers = _layers(case)
    level = [0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0, 0]
    flops = sum(2 * k * k * ci * co * b * (ny >> l) * (nx >> l) for (co, k, ci), l in zip(layers, level))
    params = sum(co * k * k * ci + co for co, k, ci in layers)
    pixels = b * ny * nx
    if kind == "infer":
        return {"bytes": pixels * (1 + 12) + 4 * params, "flops": flops}
    return {"bytes": pixels * (1 + 12) + 4 * params * 7, "flops": 3 * flops}


# ---- exact: the same in 64 bits, by torch alone ------------------------------------------------------


class _Flow:
    """Collide, boundary and stream steps in FP64 on populations (q, ...) for any cell layout."""

    def __init__(self, q, flags, tau, stream, profile=None, force=None, lid=None):
        self.c, w = _tables(q)
        self.D = 2 if q == 9 else 3
        self.q, self.opp, self.stream = q, _opposite(self.c), stream
        self.w = w
        self.omega = 1.0 / tau
        self.force = force
        self.profile, self.lid = profile, lid
        self.bounce = (flags == 1) | (flags == 5)
        self.top, self.inlet, self.outlet = flags == 5, flags == 3, flags == 4
        self.fluid = (flags >= 2) & (flags <= 4)

    def equilibrium(self, rho, u):
        vv = sum(v * v for v in u)
        out = []
        for i in range(self.q):
            cu = self._cu(i, u)
            out.append(self.w[i] * rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * vv))
        return torch.stack(out)

    def _cu(self, i, u):
        t = torch.zeros_like(u[0])
        for k in range(self.D):
            if self.c[i][k]:
                t = t + self.c[i][k] * u[k]
        return t

    def macros(self, f):
        rho = f.sum(0)
        return rho, [sum(self.c[i][k] * f[i] for i in range(self.q) if self.c[i][k]) / rho for k in range(self.D)]

    def step(self, f, solid=None):
        """One time step; returns the new populations and the moments of the collided ones."""
        if self.profile is not None:  # Zou-He ends, D2Q9
            ux = self.profile
            rho = (f[0] + f[4] + f[3] + 2 * (f[1] + f[5] + f[7])) / (1 + ux)
            g = f.clone()
            g[2] = f[1] + 2 / 3 * rho * ux
            g[6] = f[5] + rho * ux / 6 + 0.5 * (f[3] - f[4])
            g[8] = f[7] + rho * ux / 6 + 0.5 * (f[4] - f[3])
            f1 = torch.where(self.inlet, g, f)
            r = f[0] + f[3] + f[4] + 2 * (f[2] + f[6] + f[8]) - 1.0
            g = f.clone()
            g[1] = f[2] - 2 / 3 * r
            g[5] = f[6] - r / 6 + 0.5 * (f[4] - f[3])
            g[7] = f[8] - r / 6 + 0.5 * (f[3] - f[4])
            f = torch.where(self.outlet, g, f1)
            del g, f1
        rho, u = self.macros(f)
        safe = torch.where(rho == 0, torch.ones_like(rho), rho)
        u = [torch.where(rho == 0, torch.zeros_like(v), v) for v in u]
        vv = sum(v * v for v in u)
        new = torch.empty_like(f)
        for i in range(self.q):
            cu = self._cu(i, u)
            eq = self.w[i] * safe * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * vv)
            d = self.omega * (eq - f[i])
            v = f[i] + d if solid is None else f[i] + d * solid + (f[self.opp[i]] - f[i]) * (1 - solid)
            if self.force is not None:
                p = sum(((self.c[i][k] - u[k]) * 3 + self.c[i][k] * cu * 9) * self.force[k] for k in range(self.D))
                v = v + self.w[i] * p * (1 - 0.5 * self.omega)
            back = f[self.opp[i]]
            if self.lid is not None:
                edge = sum(self.c[i][k] * self.lid[k] for k in range(self.D))
                back = back + torch.where(self.top, 6 * self.w[i] * edge, 0.0)
            new[i] = self.stream(torch.where(self.fluid, v, torch.where(self.bounce, back, torch.zeros_like(v))), self.c[i])
        return new, rho, u


def _grid_stream(periodic):
    def stream(a, c):  # a (nz, ny, nx): f(x) = a(x - c), zero from outside
        out = torch.zeros_like(a)
        dst, src = [], []
        for axis, k in ((0, c[2]), (1, c[1]), (2, c[0])):
            if axis == 2 and periodic and k:
                a, k = torch.roll(a, k, 2), 0
            n = a.shape[axis]
            dst.append(slice(max(k, 0), n + min(k, 0)))
            src.append(slice(max(-k, 0), n - max(k, 0)))
        out[tuple(dst)] = a[tuple(src)]
        return out
    return stream


def exact(case, seed):
    kind = case["kind"]
    if kind == "lattice":
        return _exact_lattice(case, seed)
    if kind in ("batch", "until"):
        return _exact_batch(case, seed)
    if kind == "particles":
        return _exact_particles(case, seed)
    return _exact_net(case, seed)


def _exact_lattice(case, seed):
    nx, ny, nz, q = case["nx"], case["ny"], case["nz"], case["q"]
    D = 2 if q == 9 else 3
    tau, u_max = _constants(case, seed)
    flags = torch.from_numpy(_flags(case, seed)).cuda()
    profile = torch.from_numpy(_profile(ny, u_max)).cuda()[None, :, None] if case["flow"] == "channel" else None
    flow = _Flow(q, flags, tau, _grid_stream(_periodic(case)), profile, FORCE[:D] if case["flow"] == "force" else None,
                 LID if case["flow"] == "cavity" else None)
    rho, u = _start_fields(nx, ny, nz, D, seed)
    f = flow.equilibrium(rho.double().reshape(nz, ny, nx), [v.double().reshape(nz, ny, nx) for v in u])
    for _ in range(case["steps"] * case["calls"]):
        f, r, v = flow.step(f)
    # the macros of cells that do not collide keep their first values
    r = torch.where(flow.fluid, r, torch.ones_like(r)).reshape(-1)
    v = torch.stack([torch.where(flow.fluid, x, torch.zeros_like(x)).reshape(-1) for x in v], 1)
    out = {"rho": r, "u": v}
    if case["pops"]:
        out["f"] = f.reshape(q, -1).t().contiguous()
    return out


def _exact_batch(case, seed):
    ch = _channels(case, seed)
    flags = torch.from_numpy(np.concatenate([c["flags"].reshape(-1) for c in ch])).cuda()
    n = flags.numel()
    tau = torch.cat([torch.full((c["nx"] * c["ny"],), c["tau"], dtype=torch.float64, device="cuda") for c in ch])
    profile = torch.from_numpy(np.concatenate([np.repeat(_profile(c["ny"], c["u_max"]), c["nx"]) for c in ch])).cuda()
    owner = torch.cat([torch.full((c["nx"] * c["ny"],), k, dtype=torch.int64, device="cuda") for k, c in enumerate(ch)])
    source = {}
    for d in _tables(9)[0]:  # where each cell's population of a direction comes from; n: nowhere
        parts, base = [], 0
        for c in ch:
            at = np.full((c["ny"], c["nx"]), n, np.int64)
            y, x = np.mgrid[:c["ny"], :c["nx"]]
            sy, sx = y - d[1], x - d[0]
            ok = (sy >= 0) & (sy < c["ny"]) & (sx >= 0) & (sx < c["nx"])
            at[ok] = (base + sy * c["nx"] + sx)[ok]
            parts.append(at.reshape(-1))
            base += c["nx"] * c["ny"]
        source[d] = torch.from_numpy(np.concatenate(parts)).cuda()
    zero = torch.zeros(1, dtype=torch.float64, device="cuda")
    flow = _Flow(9, flags, tau, lambda a, c: torch.cat([a, zero])[source[c]], profile)
    f = torch.tensor(flow.w, dtype=torch.float64, device="cuda")[:, None].repeat(1, n)
    live = torch.ones(len(ch), dtype=torch.bool, device="cuda")
    steps = torch.zeros(len(ch), dtype=torch.int64, device="cuda")
    old = torch.zeros((2, n), dtype=torch.float64, device="cuda")
    rho, u, residual = torch.ones_like(tau), torch.zeros_like(old), torch.zeros(len(ch), dtype=torch.float64, device="cuda")
    done = 0
    while done < case["steps"] and bool(live.any()):
        block = case.get("check", case["steps"])
        g = f
        for _ in range(block):
            g, r, v = flow.step(g)
        cells = live[owner]
        f = torch.where(cells, g, f)
        at = cells & flow.fluid
        rho = torch.where(at, r, rho)
        u = torch.where(at, torch.stack(v), u)
        done += block
        if case["kind"] == "until":
            num = torch.zeros_like(residual).index_add_(0, owner, ((u - old) ** 2).sum(0))
            den = torch.zeros_like(residual).index_add_(0, owner, (u ** 2).sum(0))
            residual = torch.where(live, torch.sqrt(num / den), residual)
            steps = steps + block * live
            old = torch.where(cells, u, old)
            live = live & (residual >= TOL)
    out = {"rho": rho, "u": u.t().contiguous()}
    if case["kind"] == "until":
        out["residual"], out["steps"] = residual, None
    return out


def _exact_particles(case, seed):
    """The coupled steps; the discs start three cells apart and move a fraction of a cell, so none touch."""
    nx, ny, R = case["nx"], case["ny"], case["radius"]
    tau, _ = _constants(case, seed)
    flags = torch.full((1, ny, nx), 2, dtype=torch.uint8, device="cuda")
    flags[:, 0] = flags[:, -1] = 1
    flow = _Flow(9, flags, tau, _grid_stream(True), force=(0.0, -GRAVITY))
    f = torch.tensor(flow.w, dtype=torch.float64, device="cuda")[:, None, None, None].repeat(1, 1, ny, nx)
    st = torch.from_numpy(_bodies(case, seed)).cuda()
    span = 2 * int(R + 2) + 3
    k = torch.arange(span, device="cuda") - span // 2
    sub = torch.tensor([-0.375, -0.125, 0.125, 0.375], device="cuda", dtype=torch.float64)
    for _ in range(case["steps"]):
        X, V = st[:, 0:2], st[:, 0:2] - st[:, 3:5]
        near = torch.round(X).long()
        cx, cy = near[:, 0, None] + k, near[:, 1, None] + k  # each disc's window of cells
        rx, ry = cx - X[:, 0, None], cy - X[:, 1, None]
        d2 = (rx[:, :, None] + sub)[:, None, :, None, :] ** 2 + (ry[:, :, None] + sub)[:, :, None, :, None] ** 2
        inside = (cy >= 0) & (cy < ny)
        part = 1 - (d2 <= R * R).double().mean((3, 4))  # (body, y, x)
        part = torch.where(inside[:, :, None], part, torch.ones_like(part))
        gx, gy = (cx % nx)[:, None, :].expand_as(part), cy.clamp(0, ny - 1)[:, :, None].expand_as(part)
        por = torch.ones((ny, nx), dtype=torch.float64, device="cuda")
        cell = part < 1
        por.index_put_((gy[cell], gx[cell]), part[cell])  # no cell belongs to two discs
        mom = torch.zeros(part.shape + (2,), dtype=torch.float64, device="cuda")
        for i in range(1, 9):
            e = flow.c[i]
            ue = (e[0] * V[:, 0] + e[1] * V[:, 1])[:, None, None]
            there = f[flow.opp[i], 0][(gy + e[1]).clamp(0, ny - 1), (gx + e[0]) % nx]
            a = f[i, 0][gy, gx] * (1 - ue) + there * (1 + ue)
            mom += a[..., None] * torch.tensor([e[0], e[1]], dtype=torch.float64, device="cuda")
        F = mom * (1 - part)[..., None] * cell[..., None]
        force = -F.sum((1, 2))
        torque = -(rx[:, None, :] * F[..., 1] - ry[:, :, None] * F[..., 0]).sum((1, 2))
        f, rho, u = flow.step(f, solid=por[None])
        new = st.clone()
        acc = force / st[:, 24:25]
        acc[:, 1] -= GRAVITY
        new[:, 0:2], new[:, 3:5] = 2 * X - st[:, 3:5] + acc, X
        new[:, 6], new[:, 9] = 2 * st[:, 6] - st[:, 9] + torque / st[:, 25], st[:, 6]
        new[:, 12:14], new[:, 15], new[:, 18:20], new[:, 21] = acc, torque / st[:, 25], force, torque
        wrap = (new[:, 0] < 0).double() * nx - (new[:, 0] >= nx).double() * nx
        new[:, 0] += wrap
        new[:, 3] += wrap
        st = new
    rho = torch.where(flow.fluid, rho, torch.ones_like(rho)).reshape(-1)
    u = torch.stack([torch.where(flow.fluid, v, torch.zeros_like(v)).reshape(-1) for v in u], 1)
    return {"rho": rho, "u": u, "bodies": st}


def _planes(mask, umax, tau):
    """The network's 16 input planes (b, 16, ny, nx): mask, flow parameters, coordinates, and of the fluid
    cells the column's open fraction and resistance, the height of the cell's vertical gap, the position
    across it, and the lubrication estimates of velocity and pressure."""
    b, H, W = mask.shape
    solid = mask.bool()
    y = torch.arange(H, device=mask.device, dtype=torch.float64)[None, :, None].expand(b, H, W)
    x = torch.arange(W, device=mask.device, dtype=torch.float64)[None, None, :].expand(b, H, W)
    below = torch.cummax(torch.where(solid, y, torch.full_like(y, -1.0)), 1).values
    above = torch.flip(torch.cummin(torch.flip(torch.where(solid, y, torch.full_like(y, float(H))), (1,)), 1).values, (1,))
    h = above - below - 1
    fluid = (~solid).double()
    hin = float(H - 2 if H > 2 else H)
    opened = (fluid.sum(1) / hin).clamp(max=1.0)
    h3 = (torch.where(solid, torch.zeros_like(h), h) ** 2).sum(1)  # a gap of h cells gives h * h^2
    suffix = lambda v: torch.flip(torch.cumsum(torch.flip(v, (1,)), 1), (1,))  # noqa: E731
    S = suffix(1 / h3.clamp(min=1.0))
    pos = (y - below - 0.5) / h.clamp(min=1.0)
    shape = 4 * pos * (1 - pos)
    col = lambda v: v[:, None, :].expand(b, H, W)  # noqa: E731
    full = lambda v: v.double()[:, None, None].expand(b, H, W)  # noqa: E731
    inner = [col(opened), col(suffix(1 / opened.clamp(min=0.125) ** 3) / W), h / hin, shape,
             0.5 * (hin * h * h / col(h3).clamp(min=1.0) * shape).clamp(max=8.0), col(S / S[:, :1])]
    planes = [mask.double(), full(umax) / 0.08, (full(tau) - 0.55) / 0.45, y / (H - 1), x / (W - 1)]
    planes += [p * fluid for p in inner]
    return torch.stack(planes + [torch.zeros_like(y)] * 5, 1)


def _exact_net(case, seed):
    F = torch.nn.functional
    mask, umax, tau, target = _net_inputs(case, seed)
    flat = _weights(case, seed).double().cuda().requires_grad_(case["kind"] == "train")
    layers, o = [], 0
    for co, k, ci in _layers(case):
        n = co * k * k * ci
        layers.append((flat[o:o + n].reshape(co, k, k, ci).permute(0, 3, 1, 2), flat[o + n:o + n + co]))
        o += n + co

    def conv(h, i):
        """A 3x3 convolution and ReLU as nine products, which FP64 does at the matrix rate."""
        w, bias = layers[i]
        p = F.pad(h, (1, 1, 1, 1))
        H, W = h.shape[2:]
        y = bias[None, :, None, None]
        for ky in range(3):
            for kx in range(3):
                y = y + torch.einsum("nchw,oc->nohw", p[:, :, ky:ky + H, kx:kx + W], w[:, :, ky, kx])
        return torch.relu(y)

    def net(x):
        h, skips, i = x, [], 0
        for _ in range(3):
            h = conv(conv(h, i), i + 1)
            skips.append(h)
            h, i = F.avg_pool2d(h, 2), i + 2
        h, i = conv(conv(h, i), i + 1), i + 2
        for l in (2, 1, 0):
            h = torch.cat([h.repeat_interleave(2, 2).repeat_interleave(2, 3), skips[l]], 1)
            h, i = conv(conv(h, i), i + 1), i + 2
        w, bias = layers[i]
        return (torch.einsum("nchw,oc->nohw", h, w[:, :, 0, 0]) + bias[None, :, None, None]).permute(0, 2, 3, 1)

    planes = _planes(mask, umax, tau)
    if case["kind"] == "infer":
        with torch.no_grad():
            return net(planes).contiguous()
    total, count = 0.0, target.numel()
    for k in range(0, case["batch"], 4):  # samples in fours, for the memory that the gradients keep
        part = ((net(planes[k:k + 4]) - target[k:k + 4].double()) ** 2).sum() / count
        part.backward()
        total += float(part)
    g = flat.grad
    # the first step of Adam: the moments' corrections cancel
    return {"loss": total, "grads": g, "weights": flat.detach() - 1e-3 * g / (g.abs() + 1e-8)}
