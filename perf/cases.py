"""Performance cases of the GB300 lattice-Boltzmann framework.

Each case is one pass of work as a user's program asks for it, through the
public Python entry points (Solver, Batch, CgSolver, UNet):

* a single lattice advanced between two looks at it (a chunk of time steps,
  the residual where a steady run would check it, the fields read back);
* a batch of independent domains advanced the same way;
* a colour-gradient two-phase lattice, 2D and 3D;
* the warm-start U-Net: parameter gradients, a training step, a prediction.

Sizes are those of the project's configurations (128^2 BGK cavity, sphere
ducts of 70 % porosity, 1024 x 256 TRT channels, 1024^2 droplets, a sweep of
MRT cavities with sides 64..768, the 4-level 32-channel U-Net on 256 x 1024
images and its quarter-size pilot), scaled so that a case runs within
milliseconds, and odd sizes beside them.
"""
import math

import numpy as np
import torch

from thesis_gb300 import lattice
from thesis_gb300 import native as N
from thesis_gb300.batch import Batch
from thesis_gb300.lattice import Lattice
from thesis_gb300.multiphase import CgArguments, CgSolver
from thesis_gb300.solver import Arguments, Solver
from thesis_gb300.warmstart import UNet

COLLISION = {"bgk": N.BGKW, "trt": N.TRT, "mrt": N.MRT}
STORAGE = {"f32": N.STORE_F32, "f16s": N.STORE_F16S}
MODE = {"reference": N.MODE_REFERENCE, "physics": N.MODE_PHYSICS}
U_CHANNEL = 0.05  # centre-line inlet velocity of the channels


# --------------------------------------------------------------------------
# The cases
# --------------------------------------------------------------------------
def listed():
    return [
        # The plain method at its configured size: 128^2 BGK cavity in the
        # reference's semantics, 1000 of its 20,000 steps.  Every step is a
        # few microseconds: launches and latency.
        dict(name="cavity_128_bgk_ref", kind="flow", shape="cavity2d", n=128, m=128, h=1, collision="bgk",
             mode="reference", storage="f32", steps=1000, residual=False),
        # The smallest call: a ragged little cavity looked at every 50 steps.
        dict(name="cavity_61x47_mrt", kind="flow", shape="cavity2d", n=61, m=47, h=1, collision="mrt",
             mode="physics", storage="f32", steps=50, residual=True),
        # One channel of the warm-start workload: inlet, outlet, obstacles,
        # residual every 500 steps.
        dict(name="channel_1024x256_trt", kind="flow", shape="channel2d", n=1024, m=256, h=1, collision="trt",
             mode="physics", storage="f32", steps=500, residual=True),
        # A small three-dimensional cavity of odd extents, MRT.
        dict(name="cavity3d_75x61x47_mrt", kind="flow", shape="cavity3d", n=75, m=61, h=47, collision="mrt",
             mode="physics", storage="f32", steps=200, residual=False),
        # The headline workload's kernel: the sphere-packed D3Q19 MRT duct in
        # FP16-shifted storage (populations larger than L2).
        dict(name="duct_128x128x256_f16s", kind="flow", shape="duct", n=128, m=128, h=256, collision="mrt",
             mode="physics", storage="f16s", steps=200, residual=False),
        # The same duct, larger, in FP32 storage (the default storage).
        dict(name="duct_192x192x256_f32", kind="flow", shape="duct", n=192, m=192, h=256, collision="mrt",
             mode="physics", storage="f32", steps=120, residual=False),
        # The sweep: MRT cavities of uneven sides, one launch per step, FP16S.
        dict(name="batch_16_cavities_f16s", kind="batch", shape="cavity2d", domains=16, n=0, m=0, lo=64, hi=768,
             collision="mrt", storage="f16s", steps=1000, check=0),
        # Steady channel solves as the warm start makes them: TRT, FP32,
        # residuals every 100 steps, domains of one size.
        dict(name="batch_8_channels_f32", kind="batch", shape="channel2d", domains=8, n=1024, m=256, lo=0, hi=0,
             collision="trt", storage="f32", steps=1000, check=100),
        # Two-phase droplet at its configured size.
        dict(name="cg2d_1024_f32", kind="cg", n=1024, m=1024, h=1, storage="f32", high_order=False, enhanced=False,
             steps=400),
        # Two-phase drop in three dimensions, uneven extents.
        dict(name="cg3d_160x131x97_f32", kind="cg", n=160, m=131, h=97, storage="f32", high_order=False,
             enhanced=False, steps=100),
        # The stated network's parameter gradients (forward and backward) on a
        # training batch of 16 full-size channels.
        dict(name="unet_gradients_16x256x1024", kind="unet", op="gradients", height=256, width=1024, batch=16,
             levels=4, base=32),
        # The pilot network's prediction of a set of quarter-size channels.
        dict(name="unet_predict_32x64x256", kind="unet", op="predict", height=64, width=256, batch=32, levels=3,
             base=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _steps(nodes, rate, lo, hi):
    """Steps that take about 25 ms at `rate` nodes a second."""
    return int(min(hi, max(lo, 0.025 * rate / nodes)))


def draw(rng):
    kind = rng.choice(["flow2d", "flow2d", "flow3d", "flow3d", "batch", "cg2d", "cg3d", "unet"])
    if kind == "flow2d":
        shape = rng.choice(["cavity2d", "channel2d"])
        mode = rng.choice(["reference", "physics"]) if shape == "cavity2d" else "physics"
        n = _log_int(rng, 48, 1024)
        m = max(40, int(n * rng.uniform(0.25, 1.0)))
        return dict(kind="flow", shape=shape, n=n, m=m, h=1,
                    collision="bgk" if mode == "reference" else rng.choice(["bgk", "trt", "mrt"]), mode=mode,
                    storage="f32", steps=_steps(n * m, 20e9, 50, 1000), residual=rng.random() < 0.5)
    if kind == "flow3d":
        shape = rng.choice(["cavity3d", "duct"])
        lo = 24 if shape == "cavity3d" else 48
        n, m, h = (_log_int(rng, lo, 224) for _ in range(3))
        return dict(kind="flow", shape=shape, n=n, m=m, h=h, collision="mrt", mode="physics",
                    storage=rng.choice(["f32", "f16s"]) if shape == "duct" else "f32",
                    steps=_steps(n * m * h, 20e9, 40, 200), residual=False)
    if kind == "batch":
        if rng.random() < 0.5:
            hi = 32 * rng.randint(4, 20)
            return dict(kind="batch", shape="cavity2d", domains=rng.randint(2, 16), n=0, m=0, lo=32, hi=hi,
                        collision=rng.choice(["bgk", "mrt"]), storage=rng.choice(["f32", "f16s"]),
                        steps=rng.choice([200, 400, 800]), check=0)
        m = 8 * rng.randint(8, 32)
        return dict(kind="batch", shape="channel2d", domains=rng.randint(2, 8), n=4 * m, m=m, lo=0, hi=0,
                    collision="trt", storage="f32", steps=rng.choice([200, 400, 800]), check=100)
    if kind == "cg2d":
        n, m = _log_int(rng, 96, 1100), _log_int(rng, 96, 1000)
        return dict(kind="cg", n=n, m=m, h=1, storage=rng.choice(["f32", "f32", "f16s"]),
                    high_order=rng.random() < 0.3, enhanced=rng.random() < 0.3, steps=_steps(n * m, 15e9, 50, 400))
    if kind == "cg3d":
        n, m, h = (_log_int(rng, 32, 130) for _ in range(3))
        return dict(kind="cg", n=n, m=m, h=h, storage="f32", high_order=False, enhanced=rng.random() < 0.3,
                    steps=_steps(n * m * h, 8e9, 20, 100))
    base = rng.choice([16, 32])
    levels = rng.choice([3, 4])
    hgt = 16 * rng.randint(2, 14)
    return dict(kind="unet", op=rng.choice(["gradients", "train", "predict"]), height=hgt,
                width=16 * rng.randint(2, 60), batch=rng.randint(1, 12), levels=levels, base=base)


# --------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------
def _rng(seed, salt):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, salt])


def _channel_lattice(n, m, seed):
    return lattice.channel2d(n, m, seed=int(seed), size_scale=min(1.0, m / 256.0))


def _profile(m):
    y = np.arange(m) + 0.5
    return 4.0 * U_CHANNEL * y * (m - y) / (m * m)


def _flow_inputs(case, seed):
    """Lattice, Arguments and the initial or inlet velocity of a single run."""
    g = _rng(seed, 1)
    n, m, h = case["n"], case["m"], case["h"]
    shape = case["shape"]
    common = dict(collision_model=COLLISION[case["collision"]], mode=MODE[case["mode"]],
                  storage=STORAGE[case["storage"]], init_equilibrium=1)
    if shape == "cavity2d":
        u = float(g.uniform(0.08, 0.12))
        re = float(g.uniform(80.0, 200.0))
        return lattice.cavity2d(n, m), Arguments(u=u, viscosity=u * n / re, outlet_profile=N.OUTLET_ZOUHE, **common)
    if shape == "channel2d":
        re = float(g.uniform(20.0, 200.0))
        return (_channel_lattice(n, m, g.integers(1 << 30)),
                Arguments(u=U_CHANNEL, viscosity=U_CHANNEL * m / re, outlet_profile=N.OUTLET_PRESSURE, rho_out=1.0,
                          **common))
    if shape == "cavity3d":
        u = float(g.uniform(0.05, 0.1))
        re = float(g.uniform(50.0, 150.0))
        return lattice.cavity3d(n, m, h), Arguments(u=u, viscosity=u * n / re, outlet_profile=N.OUTLET_ZOUHE, **common)
    # pressure-driven duct: tau = 0.8, rho_in about 1.005
    lat = lattice.sphere_duct(n, m, h, porosity=0.70, rmin=6.0, rmax=14.0, seed=int(g.integers(1 << 30)))
    return lat, Arguments(u=0.0, viscosity=0.1, inlet_profile=N.INLET_PRESSURE, outlet_profile=N.OUTLET_PRESSURE,
                          rho_in=float(g.uniform(1.004, 1.006)), rho_out=1.0, **common)


def _batch_inputs(case, seed):
    g = _rng(seed, 2)
    common = dict(collision_model=COLLISION[case["collision"]], mode=N.MODE_PHYSICS, storage=STORAGE[case["storage"]],
                  init_equilibrium=1)
    lats, args = [], []
    sides = _rng(case["domains"] * 1009 + case["hi"], 3)  # the sweep's sides belong to the case
    for _ in range(case["domains"]):
        if case["shape"] == "cavity2d":
            n = int(32 * sides.integers(case["lo"] // 32, case["hi"] // 32 + 1))
            re = float(g.uniform(100.0, 3200.0 if case["collision"] == "mrt" else 320.0))
            lats.append(lattice.cavity2d(n))
            args.append(Arguments(u=0.1, viscosity=0.1 * n / re, outlet_profile=N.OUTLET_ZOUHE, **common))
        else:
            re = float(g.uniform(20.0, 200.0))
            lats.append(_channel_lattice(case["n"], case["m"], g.integers(1 << 30)))
            args.append(Arguments(u=U_CHANNEL, viscosity=U_CHANNEL * case["m"] / re, outlet_profile=N.OUTLET_PRESSURE,
                                  rho_out=1.0, **common))
    return lats, args


def _cg_inputs(case, seed):
    """Model parameters and the drop's nodes (red inside a circle or sphere)."""
    g = _rng(seed, 4)
    n, m, h = case["n"], case["m"], case["h"]
    small = min(n, m) if h == 1 else min(n, m, h)
    radius = float(g.uniform(0.2, 0.35)) * small
    a = CgArguments(A=float(g.uniform(0.003, 0.006)), beta=0.7, high_order=case["high_order"],
                    enhanced_distrib=case["enhanced"], storage=STORAGE[case["storage"]],
                    r_viscosity=float(g.uniform(0.12, 0.2)), b_viscosity=float(g.uniform(0.12, 0.2)))
    cx, cy, cz = (float(g.uniform(0.4, 0.6)) * s for s in (n, m, h))
    i = np.arange(n * m * h)
    x, y, z = i % n, (i // n) % m, i // (n * m)
    d2 = (x - cx) ** 2 + (y - cy) ** 2 + ((z - cz) ** 2 if h > 1 else 0.0)
    return a, d2 <= radius * radius


def _cg_start(case, inside):
    """Both colours at rest (density 1) as post-stream populations."""
    q = 9 if case["h"] == 1 else 19
    if q == 9:
        al = 4.0 / 9.0
        phi = np.array([al] + [(1 - al) / 5] * 4 + [(1 - al) / 20] * 4)
    else:
        phi = np.array([0.0] + [1 / 12] * 6 + [1 / 24] * 12)
    phi = phi.astype(np.float32)
    r = np.where(inside[None, :], phi[:, None], np.float32(0))
    return r, phi[:, None] - r


def _unet_spec(levels, base):
    """(cin, cout, relu) of the network's convolutions in parameter order."""
    c = lambda l: min(base << l, 64)  # noqa: E731
    s = []
    for l in range(levels):
        s += [(16 if l == 0 else c(l - 1), c(l), True), (c(l), c(l), True)]
    s += [(c(levels - 1), c(levels), True), (c(levels), c(levels), True)]
    for l in range(levels - 1, -1, -1):
        up = c(levels) if l == levels - 1 else c(l)
        s += [(up + c(l), c(l), True), (c(l), c(l - 1) if l > 0 else c(0), True)]
    return s + [(c(0), 16, False)]


def _unet_inputs(case, seed):
    """Parameters, images, targets and weights: channels with obstacles, the
    target a channel flow that slows in the wake of the solid nodes."""
    g = _rng(seed, 5)
    H, W, B = case["height"], case["width"], case["batch"]
    spec = _unet_spec(case["levels"], case["base"])
    parts = []
    for k, (ci, co, _) in enumerate(spec):
        real_i = 4 if k == 0 else ci
        real_o = 3 if k == len(spec) - 1 else co
        w = np.zeros((9, co, ci), np.float32)
        w[:, :real_o, :real_i] = g.standard_normal((9, real_o, real_i)) * math.sqrt(2.0 / (9 * real_i))
        b = np.zeros(co, np.float32)
        b[:real_o] = 0.02 * g.standard_normal(real_o)
        parts += [w.reshape(-1), b]
    params = np.concatenate(parts).astype(np.float32)
    x = np.zeros((B, H, W, 4), np.float32)
    t = np.zeros((B, H, W, 3), np.float32)
    prof = (4.0 * (np.arange(H) + 0.5) * (H - np.arange(H) - 0.5) / (H * H))[:, None]
    xs, ys = np.arange(W)[None, :], np.arange(H)[:, None]
    for i in range(B):
        fluid = np.ones((H, W), bool)
        wake = np.zeros((H, W))
        for _ in range(int(g.integers(1, 7))):
            r = g.uniform(0.04, 0.12) * H
            cx, cy = g.uniform(0.1, 0.85) * W, g.uniform(0.15, 0.85) * H
            fluid &= (xs - cx) ** 2 + (ys - cy) ** 2 > r * r
            wake += np.where(xs > cx, np.exp(-((ys - cy) / (1.5 * r)) ** 2 - (xs - cx) / (8 * r)), 0.0)
        x[i, ..., 0] = fluid
        x[i, ..., 1] = g.uniform(0.1, 1.0)
        x[i, ..., 2] = prof
        x[i, ..., 3] = np.linspace(0.0, 1.0, W)[None, :]
        u = prof * (1.0 - np.minimum(wake, 1.0)) * fluid
        t[i, ..., 0] = u
        t[i, ..., 1] = 0.1 * u * np.sin(6.28 * ys / H)
        t[i, ..., 2] = (1.0 - xs / W) * fluid
    return params, x, t, np.ascontiguousarray(x[..., 0])


def _pinned(n, k=4):
    return [torch.empty(n, dtype=torch.float32, pin_memory=True).numpy() for _ in range(k)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "flow":
        lat, args = _flow_inputs(case, seed)
        s = Solver(lat, args)
        nn = lat.num_nodes
        if case["shape"] == "channel2d":
            s.set_inlet_velocity(u=np.broadcast_to(_profile(lat.m)[:, None], (lat.m, lat.n)))
        zero = np.zeros(nn, np.float32)
        s.init(np.ones(nn, np.float32), zero, zero, zero)
        return dict(case=case, solver=s, out=_pinned(nn))
    if kind == "batch":
        lats, args = _batch_inputs(case, seed)
        b = Batch(lats, args)
        b.init()
        for d, lat in enumerate(lats):
            if case["shape"] == "channel2d":
                b.set_inlet_velocity(d, u=np.broadcast_to(_profile(lat.m)[:, None], (lat.m, lat.n)))
            nn = lat.num_nodes
            zero = np.zeros(nn, np.float32)
            b.init_fields(d, np.ones(nn, np.float32), zero, zero, zero)
        return dict(case=case, batch=b)
    if kind == "cg":
        a, inside = _cg_inputs(case, seed)
        s = CgSolver(case["n"], case["m"], a, h=None if case["h"] == 1 else case["h"])
        s.init(*_cg_start(case, inside))
        return dict(case=case, cg=s)
    params, x, t, w = _unet_inputs(case, seed)
    net = UNet(case["height"], case["width"], max_batch=case["batch"], levels=case["levels"],
               base_channels=case["base"])
    net.set_params(params)
    if case["op"] != "predict":
        net.set_dataset(x, t, w)
    return dict(case=case, net=net, x=x, idx=np.arange(case["batch"], dtype=np.int32))


# --------------------------------------------------------------------------
# One pass
# --------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "flow":
        s = state["solver"]
        s.step(case["steps"], write_macro=True)
        res = float(s.residual()[0]) if case["residual"] else None
        rho, u, v, w = s.macro(out=state["out"])
        out = dict(rho=rho, u=u, v=v)
        if case["h"] > 1:
            out["w"] = w
        if res is not None:
            out["residual"] = res
        return out
    if kind == "batch":
        b = state["batch"]
        # a steady solve looks at the residuals between chunks; they are
        # differences of FP32 fields, so the fields themselves are returned
        chunk = case["check"] or case["steps"]
        for _ in range(case["steps"] // chunk):
            b.step(chunk, write_macro=True)
            if case["check"]:
                b.residuals()
        return dict(fields=[b.macro(d)[:3] for d in range(case["domains"])])
    if kind == "cg":
        s = state["cg"]
        s.step(case["steps"], write_macro=True)
        return list(s.macro())
    net = state["net"]
    if case["op"] == "gradients":
        g, loss = net.gradients(state["idx"])
        return dict(grad=g, loss=float(loss))
    if case["op"] == "train":
        loss = net.train_step(state["idx"], 1e-3)
        return dict(params=net.params(), loss=float(loss))
    return net.predict(state["x"])


# --------------------------------------------------------------------------
# The work a pass cannot do without
# --------------------------------------------------------------------------
def _unet_flops(case):
    H, W, L = case["height"], case["width"], case["levels"]
    levels = []
    for l in range(L):
        levels += [l, l]
    levels += [L, L]
    for l in range(L - 1, -1, -1):
        levels += [l, l]
    levels.append(0)
    return sum(2 * 9 * ci * co * (H >> l) * (W >> l) for (ci, co, _), l in zip(_unet_spec(L, case["base"]), levels))


def work(case):
    kind = case["kind"]
    nodes = case.get("n", 0) * case.get("m", 0) * case.get("h", 1)
    eb = 2 if case.get("storage") == "f16s" else 4
    if kind == "flow":
        q = 9 if case["h"] == 1 else 19
        fluid = nodes * (0.70 if case["shape"] == "duct" else 1.0)
        # populations read once and written once a step, a flag word a node
        return dict(bytes=case["steps"] * fluid * (2 * q * eb + 4) + 16.0 * nodes,
                    flops=case["steps"] * fluid * (250.0 if q == 19 else 100.0))
    if kind == "batch":
        if case["shape"] == "cavity2d":
            sides = _rng(case["domains"] * 1009 + case["hi"], 3)
            nodes = sum(int(32 * sides.integers(case["lo"] // 32, case["hi"] // 32 + 1)) ** 2
                        for _ in range(case["domains"]))
        else:
            nodes *= case["domains"]
        return dict(bytes=case["steps"] * nodes * (18.0 * eb + 4) + 16.0 * nodes, flops=case["steps"] * nodes * 100.0)
    if kind == "cg":
        q = 9 if case["h"] == 1 else 19
        # both colours read once and written once a step
        return dict(bytes=case["steps"] * nodes * 4.0 * q * eb + 16.0 * nodes,
                    flops=case["steps"] * nodes * (300.0 if q == 9 else 700.0))
    B = case["batch"]
    px = B * case["height"] * case["width"]
    f = B * _unet_flops(case)
    if case["op"] == "predict":
        return dict(bytes=px * 28.0, flops=float(f))
    # 3 GEMMs a layer; every activation stored once and read once in BF16
    c = [(ci + co) * 4.0 ** -l for (ci, co, _), l in zip(_unet_spec(case["levels"], case["base"]), _unet_levels(case))]
    return dict(bytes=px * (32.0 + 16.0) + 4.0 * px * sum(c), flops=3.0 * f)


def _unet_levels(case):
    L = case["levels"]
    out = []
    for l in range(L):
        out += [l, l]
    out += [L, L]
    for l in range(L - 1, -1, -1):
        out += [l, l]
    return out + [0]


# --------------------------------------------------------------------------
# The same results in 64 bits, in plain torch
# --------------------------------------------------------------------------
_C2 = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (-1, 0, 0), (0, -1, 0), (1, 1, 0), (-1, 1, 0), (-1, -1, 0), (1, -1, 0)]
_C3 = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, 1, 0),
       (1, -1, 0), (-1, -1, 0), (1, 0, 1), (-1, 0, 1), (1, 0, -1), (-1, 0, -1), (0, 1, 1), (0, -1, 1), (0, 1, -1),
       (0, -1, -1)]


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _weights(C):
    if len(C) == 9:
        return [4 / 9 if d == 0 else (1 / 9 if d < 5 else 1 / 36) for d in range(9)]
    return [1 / 3 if d == 0 else (1 / 18 if d < 7 else 1 / 36) for d in range(19)]


def _mrt(C, omega):
    """Moment matrix rows and relaxation rates of the model."""
    if len(C) == 9:
        rows = []
        for x, y, _ in C:
            s = x * x + y * y
            rows.append([1, -4 + 3 * s, 4 - 10.5 * s + 4.5 * s * s, x, (-5 + 3 * s) * x, y, (-5 + 3 * s) * y,
                         x * x - y * y, x * y])
        rates = [1, 1.4, 1.4, 1, 1.2, 1, 1.2, omega, omega]
    else:
        rows = []
        for x, y, z in C:
            s = x * x + y * y + z * z
            rows.append([1, 19 * s - 30, (21 * s * s - 53 * s + 24) / 2, x, (5 * s - 9) * x, y, (5 * s - 9) * y, z,
                         (5 * s - 9) * z, 3 * x * x - s, (3 * s - 5) * (3 * x * x - s), y * y - z * z,
                         (3 * s - 5) * (y * y - z * z), x * y, y * z, x * z, (y * y - z * z) * x, (z * z - x * x) * y,
                         (x * x - y * y) * z])
        rates = [0, 1.19, 1.4, 0, 1.2, 0, 1.2, 0, 1.2, omega, 1.4, omega, 1.4, omega, omega, omega, 1.98, 1.98, 1.98]
    M = torch.tensor(rows, dtype=torch.float64).T.contiguous()
    return M, torch.tensor(rates, dtype=torch.float64)


class _Exact:
    """One lattice in FP64: post-collision populations f[q, h, m, n]."""

    def __init__(self, case, lat, args, inlet=None):
        self.dev = _device()
        self.case, self.args = case, args
        n, m, h = lat.n, lat.m, lat.h
        self.C = _C2 if lat.dims == 2 else _C3
        Q = len(self.C)
        self.w = _weights(self.C)
        self.opp = [self.C.index((-x, -y, -z)) for x, y, z in self.C]
        self.fluid = torch.from_numpy(lat.node_type.reshape(h, m, n) == 1).to(self.dev)
        self.omega = 1.0 / (3.0 * args.viscosity + 0.5)
        self.omega_m = 8.0 * (2.0 - self.omega) / (8.0 - self.omega)
        self.coll = case["collision"]
        if self.coll == "mrt":
            M, s = _mrt(self.C, self.omega)
            self.M = M.to(self.dev)
            self.K = (M.T @ torch.diag(s / (M * M).sum(1))).to(self.dev)
        # links into a solid node or out of the lattice
        self.blocked = []
        for c in self.C:
            x, y, z = c
            src = torch.roll(self.fluid, (z, y, x), (0, 1, 2)).clone()
            for axis, k in ((2, x), (1, y), (0, z)):
                if k:
                    src.select(axis, 0 if k > 0 else src.shape[axis] - 1).fill_(False)
            self.blocked.append(~src)
        f = torch.zeros((Q, h, m, n), dtype=torch.float64, device=self.dev)
        one = torch.ones((h, m, n), dtype=torch.float64, device=self.dev)
        u = [torch.zeros_like(one) for _ in range(3)]
        for d in range(Q):
            f[d] = self.w[d]
        self.macro = [one.clone()] + [a.clone() for a in u]
        self.f = self.collide(f, one, u)
        self.inlet = inlet

    def feq(self, d, rho, u, usq):
        x, y, z = self.C[d]
        cu = x * u[0] + y * u[1] + z * u[2]
        return self.w[d] * rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * usq)

    def collide(self, f, rho, u):
        Q = len(self.C)
        if self.coll == "mrt":
            if Q == 9:
                usq = u[0] ** 2 + u[1] ** 2
                j = [rho * u[0], rho * u[1]]
                eq = [rho, rho * (-2 + 3 * usq), rho * (1 - 3 * usq), j[0], -j[0], j[1], -j[1],
                      rho * (u[0] ** 2 - u[1] ** 2), rho * u[0] * u[1]]
            else:
                jx, jy, jz = (rho * a for a in u)
                jsq = jx * jx + jy * jy + jz * jz
                o = torch.zeros_like(rho)
                eq = [rho, -11 * rho + 19 * jsq, -475.0 / 63.0 * jsq, jx, -2 / 3 * jx, jy, -2 / 3 * jy, jz, -2 / 3 * jz,
                      2 * jx * jx - jy * jy - jz * jz, o, jy * jy - jz * jz, o, jx * jy, jy * jz, jx * jz, o, o, o]
            mom = (self.M @ f.reshape(Q, -1)).reshape(f.shape)
            for k in range(Q):
                mom[k] -= eq[k]
            return f - (self.K @ mom.reshape(Q, -1)).reshape(f.shape)
        usq = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
        e = [self.feq(d, rho, u, usq) for d in range(Q)]
        out = torch.empty_like(f)
        for d in range(Q):
            o = self.opp[d]
            if self.coll == "bgk":
                out[d] = f[d] - self.omega * (f[d] - e[d])
            else:
                out[d] = (f[d] - self.omega * 0.5 * (f[d] + f[o] - e[d] - e[o])
                          - self.omega_m * 0.5 * (f[d] - f[o] - e[d] + e[o]))
        return out

    def face(self, f, idx, e, pressure, rho, u):
        """Zou-He with transverse corrections on the nodes f[:, idx]; e the inward normal."""
        C = self.C
        g = [f[d][idx] for d in range(len(C))]
        dot = lambda a, b: a[0] * b[0] + a[1] * b[1] + a[2] * b[2]  # noqa: E731
        s0 = sum(g[d] for d in range(len(C)) if dot(C[d], e) == 0)
        sm = sum(g[d] for d in range(len(C)) if dot(C[d], e) == -1)
        if pressure:
            ue = 1.0 - (s0 + 2 * sm) / rho
            u = [ue * k for k in e]
        else:
            ue = sum(a * k for a, k in zip(u, e))
            rho = (s0 + 2 * sm) / (1.0 - ue)
        for d in range(1, len(C)):
            if dot(C[d], e) != 1:
                continue
            t = tuple(a - b for a, b in zip(C[d], e))
            o = self.opp[d]
            if t == (0, 0, 0):
                f[d][idx] = g[o] + 6 * self.w[d] * rho * ue
            else:
                st = sum(dot(C[c], t) * g[c] for c in range(len(C)) if dot(C[c], e) == 0 and dot(C[c], t) != 0)
                f[d][idx] = g[o] + rho * ue / 6 + rho * dot(u, t) / 2 - st / 2

    def boundary(self, f):
        a, shape = self.args, self.case["shape"]
        top = slice(1, -1)
        if shape == "cavity2d" and self.case.get("mode") == "reference":
            lid = (0, -1, top)
            t = (f[0][lid] + f[1][lid] + f[3][lid] + 2 * (f[2][lid] + f[6][lid] + f[5][lid])) * a.u / 6
            f[4][lid] = f[2][lid]
            f[8][lid] = f[6][lid] + t
            f[7][lid] = f[5][lid] - t
            _, _, m, n = f.shape
            left, right, low = (0, slice(None), 0), (0, slice(None), n - 1), (0, 0, slice(None))
            for d in range(1, 9):
                x, y, _ = self.C[d]
                wall = torch.zeros((1, m, n), dtype=torch.bool, device=self.dev)
                if x < 0:
                    wall[left] = True
                if x > 0:
                    wall[right] = True
                if y < 0:
                    wall[low] = True
                o = self.opp[d]
                f[o] = torch.where(wall, f[d], f[o])
            # the lid's corners: diagonal links leaving through both faces are walls (set above)
        elif shape in ("cavity2d", "cavity3d"):
            lid = (0, -1, top) if shape == "cavity2d" else (-1, top, top)
            axis = 1 if shape == "cavity2d" else 2
            for d, c in enumerate(self.C):
                if c[axis] == -1 and c[0]:
                    f[d][lid] += 6 * self.w[d] * 1.0 * c[0] * a.u
        elif shape == "channel2d":
            west, east = (0, top, 0), (0, top, -1)
            self.face(f, west, (1, 0, 0), False, None, [self.inlet[top], torch.zeros_like(self.inlet[top]), 0.0])
            self.face(f, east, (-1, 0, 0), True, a.rho_out, None)
        else:
            for k, e, r in ((0, (0, 0, 1), a.rho_in), (-1, (0, 0, -1), a.rho_out)):
                self.face(f, (k, self.fluid[k]), e, True, r, None)

    def step(self, steps):
        Q = len(self.C)
        ref = self.case.get("mode") == "reference"
        for _ in range(steps):
            g = torch.empty_like(self.f)
            for d, (x, y, z) in enumerate(self.C):
                own = self.f[d if ref else self.opp[d]]
                g[d] = torch.where(self.blocked[d], own, torch.roll(self.f[d], (z, y, x), (0, 1, 2)))
            self.boundary(g)
            rho = torch.where(self.fluid, g.sum(0), torch.ones_like(g[0]))
            u = [sum(c[k] * g[d] for d, c in enumerate(self.C) if c[k]) / rho if any(c[k] for c in self.C)
                 else torch.zeros_like(rho) for k in range(3)]
            u = [torch.where(self.fluid, a, torch.zeros_like(a)) for a in u]
            self.f = self.collide(g, rho, u)
            self.macro = [rho] + u

    def fields(self):
        return [a.reshape(-1) for a in self.macro]


def _exact_inlet(lat):
    return torch.from_numpy(_profile(lat.m).astype(np.float32).astype(np.float64)).to(_device())


def _exact_flow(case, seed):
    lat, args = _flow_inputs(case, seed)
    e = _Exact(case, lat, args, _exact_inlet(lat) if case["shape"] == "channel2d" else None)
    e.step(case["steps"])
    rho, u, v, w = e.fields()
    out = dict(rho=rho, u=u, v=v)
    if case["h"] > 1:
        out["w"] = w
    if case["residual"]:
        out["residual"] = 1.0  # against the zero fields before the first check
    return out


def _exact_batch(case, seed):
    lats, args = _batch_inputs(case, seed)
    c = dict(case, mode="physics")
    out = []
    for lat, a in zip(lats, args):
        e = _Exact(c, lat, a, _exact_inlet(lat) if case["shape"] == "channel2d" else None)
        e.step(case["steps"])
        out.append(e.fields()[:3])
    return dict(fields=out)


def _cg_gradient(p, offsets):
    g = [torch.zeros_like(p) for _ in range(3)]
    for (x, y, z), w in offsets:
        q = torch.roll(p, (-z, -y, -x), (0, 1, 2)) * w
        for k, c in enumerate((x, y, z)):
            if c:
                g[k] = g[k] + c * q
    return g


def _cg_offsets(case, C):
    if not case["high_order"]:
        if len(C) == 9:
            return [(C[k], 4 / 12 if k <= 4 else 1 / 12) for k in range(1, 9)]
        return [(C[k], 1 / 6 if k <= 6 else 1 / 12) for k in range(1, 19)]
    wt = {1: 960, 2: 448, 4: 84, 5: 32, 8: 1}
    return [((x, y, 0), wt[x * x + y * y] / 5040) for x in range(-2, 3) for y in range(-2, 3) if x or y]


def _exact_cg(case, seed):
    a, inside = _cg_inputs(case, seed)
    n, m, h = case["n"], case["m"], case["h"]
    dev = _device()
    r, b = (torch.from_numpy(np.asarray(v, np.float64)).reshape(-1, h, m, n).to(dev) for v in _cg_start(case, inside))
    two = h == 1
    C = _C2 if two else _C3
    Q = len(C)
    w = _weights(C)
    axis = 4 if two else 6
    cls = lambda d, v0, v1, v2: v0 if d == 0 else (v1 if d <= axis else v2)  # noqa: E731
    offs = _cg_offsets(case, C)

    def collide(r, b):
        f = r + b
        rr, bb = r.sum(0), b.sum(0)
        rho = rr + bb
        u = [sum(c[k] * f[d] for d, c in enumerate(C) if c[k]) / rho if any(c[k] for c in C) else torch.zeros_like(rho)
             for k in range(3)]
        g = _cg_gradient((rr - bb) / rho, offs)
        gn = torch.sqrt(g[0] ** 2 + g[1] ** 2 + g[2] ** 2)
        face = gn > a.g_limit
        safe = torch.where(face, gn, torch.ones_like(gn))
        nu = 1.0 / (rr / (rho * a.r_viscosity) + bb / (rho * a.b_viscosity))
        om = 1.0 / (3.0 * nu + 0.5)
        alpha = a.r_alpha * rr / rho + a.b_alpha * bb / rho
        usq = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
        gr = _cg_gradient(rho, offs) if case["enhanced"] else None
        ro, bo = torch.empty_like(r), torch.empty_like(b)
        for d, c in enumerate(C):
            if two:
                rest = cls(d, 0.0, 0.2, 0.05) + cls(d, 1.0, -0.2, -0.05) * alpha
                bk, chi, psi = cls(d, -4 / 27, 2 / 27, 5 / 108), cls(d, -8 / 3, -1 / 6, 1 / 12), cls(d, 0, 0.5, 0.125)
            else:
                rest = cls(d, 0.0, 1 / 12, 1 / 24) + cls(d, 1.0, -1 / 12, -1 / 24) * alpha
                bk, chi, psi = cls(d, -2 / 9, 1 / 54, 1 / 27), cls(d, -2.5, -1 / 6, 1 / 24), cls(d, 0, 0.25, 0.125)
            cg = sum(k * v for k, v in zip(c, g))
            cu = sum(k * v for k, v in zip(c, u))
            cos = torch.where(face, cg / safe, torch.zeros_like(gn)) * cls(d, 0.0, 1.0, math.sqrt(0.5)) if d else 0.0 * gn
            pert = torch.where(face, a.A * gn * (w[d] * cg * cg / (safe * safe) - bk), torch.zeros_like(gn))
            feq = rho * (rest + w[d] * (3 * cu + 4.5 * cu * cu - 1.5 * usq))
            if gr is not None:
                tc = sum(c[i] * c[j] * (u[i] * gr[j] + u[j] * gr[i]) for i in range(3) for j in range(3) if c[i] * c[j])
                ugr = sum(p * q for p, q in zip(u, gr))
                feq = feq + nu * (chi * ugr + psi * tc)
            fp = om * feq + (1 - om) * f[d] + pert
            k = a.beta * rr * bb / rho * cos * rest
            ro[d], bo[d] = rr / rho * fp + k, bb / rho * fp - k
        return ro, bo, [rr, bb] + u[:2 if two else 3]

    r, b, mac = collide(r, b)
    for _ in range(case["steps"]):
        for d, (x, y, z) in enumerate(C):
            r[d] = torch.roll(r[d], (z, y, x), (0, 1, 2))
            b[d] = torch.roll(b[d], (z, y, x), (0, 1, 2))
        r, b, mac = collide(r, b)
    return [v.reshape(-1) for v in mac]


def _conv64(x, w, b):
    """3x3 convolution in FP64: x [B, H, W, ci], w [9, co, ci]."""
    B, H, W, _ = x.shape
    xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    out = b.expand(B, H, W, -1)
    for t in range(9):
        out = out + xp[:, t // 3:t // 3 + H, t % 3:t % 3 + W, :] @ w[t].T
    return out


def _exact_unet(case, seed):
    dev = _device()
    params, x, t, w = _unet_inputs(case, seed)
    L = case["levels"]
    spec = _unet_spec(L, case["base"])
    train = case["op"] != "predict"
    flat = torch.from_numpy(params.astype(np.float64)).to(dev).requires_grad_(train)
    P, off = [], 0
    for ci, co, relu in spec:
        k = 9 * ci * co
        P.append((flat[off:off + k].reshape(9, co, ci), flat[off + k:off + k + co], relu))
        off += k + co

    def net(xi):
        c = lambda k, v: torch.relu(_conv64(v, P[k][0], P[k][1])) if P[k][2] else _conv64(v, P[k][0], P[k][1])  # noqa
        v = torch.nn.functional.pad(xi, (0, 12))
        skips = []
        for l in range(L):
            v = c(2 * l + 1, c(2 * l, v))
            skips.append(v)
            B, H, W, Cc = v.shape
            v = v.reshape(B, H // 2, 2, W // 2, 2, Cc).mean((2, 4))
        v = c(2 * L + 1, c(2 * L, v))
        for l in range(L - 1, -1, -1):
            k = 2 * L + 2 + 2 * (L - 1 - l)
            v = torch.cat([v.repeat_interleave(2, 1).repeat_interleave(2, 2), skips[l]], -1)
            v = c(k + 1, c(k, v))
        return c(len(spec) - 1, v)[..., :3]

    tgt = torch.from_numpy(t.astype(np.float64)).to(dev)
    wt = torch.from_numpy(w.astype(np.float64)).to(dev)
    norm = 3.0 * float(wt.sum())
    outs, loss = [], 0.0
    for i in range(case["batch"]):  # one image at a time: a full-size batch in FP64 is large
        xi = torch.from_numpy(x[i:i + 1].astype(np.float64)).to(dev)
        if train:
            d = net(xi) - tgt[i:i + 1]
            part = (wt[i:i + 1, ..., None] * d * d).sum() / norm
            part.backward()
            loss += float(part.detach())
        else:
            with torch.no_grad():
                outs.append(net(xi))
    if case["op"] == "predict":
        return torch.cat(outs)
    if case["op"] == "gradients":
        return dict(grad=flat.grad, loss=torch.tensor(loss, dtype=torch.float64))
    return dict(params=None, loss=torch.tensor(loss, dtype=torch.float64))


def _exact_cost(case):
    """Seconds of the FP64 run, roughly."""
    if case["kind"] == "unet":
        f = case["batch"] * _unet_flops(case)
        return f * (1 if case["op"] == "predict" else 3) / 4e11
    nodes = case["n"] * case["m"] * case.get("h", 1) * case.get("domains", 1)
    if case["kind"] == "batch" and case["shape"] == "cavity2d":
        nodes = case["domains"] * (0.5 * (case["lo"] + case["hi"])) ** 2
    q = 19 if case.get("h", 1) > 1 else 9
    launches = 12 * q * case.get("domains", 1) * (3 if case["kind"] == "cg" else 1)
    return case["steps"] * max(launches * 6e-6, nodes * q * (60 if case["kind"] == "cg" else 25) * 8 / 4e12)


def exact(case, seed):
    if _exact_cost(case) > 20:
        return None
    return {"flow": _exact_flow, "batch": _exact_batch, "cg": _exact_cg, "unet": _exact_unet}[case["kind"]](case, seed)
