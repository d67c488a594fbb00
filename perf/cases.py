"""The calls whose speed matters to a user of this framework, with the inputs that such a user has in hand.

Every case goes through the package's public entry points (vortegrid_gb300 and its C ABI).  Sizes come from the benchmark,
the tests and the batched effects, and from the ranges around them; odd and ragged sizes stand beside the round ones.

  frame      one frame of a scene on the host's particle records in pinned memory: the direct step and the vortons' Euler
             step, then the tracers' (vg_step_advect)
  device     the same frame on particles that live on the GPU (vg_step_evolve_device, vg_advect_device)
  points     direct-sum velocities at arbitrary points (probes, a second particle group)
  treecode   the treecode step on a grid that follows the particles' box, and its tracers
  plugin     the default step (Poisson technique, grid from the box, multigrid to 1e-6) as a host program's particle
             operation calls it, on pageable records
  poisson    the default step on GPU-resident vortons and a fixed grid, and the advection of its tracers
  solve      the multigrid solver alone, on a right-hand side and boundary values of the caller's
  batch      one frame of many small independent effects
  guess      the warm-start network's forward pass
  train      the network's forward and backward pass on one training pair, and its gradients
  scene      the particle and surface operations around the step: density grid, signed distance, marching cubes, heat
             diffusion, baroclinic generation, wind, and collisions with three bodies
"""
import ctypes
import math

import numpy as np
import torch

import vortegrid_gb300 as vg
from vortegrid_gb300 import batch as vgbatch
from vortegrid_gb300 import warmstart

RADIUS = 0.05            # the scenes' vorton radius
DT = 1.0 / 30.0
SLOW_DT = 1e-6           # for frames that move their particles in place: thousands of them stay inside the grid
FLOPS_PER_PAIR = 26      # one vorton's velocity at one point

# (ci, co, level) of the network's fifteen convolutions, in the order of its parameters
LAYERS = [(16, 16, 0), (16, 16, 0), (16, 32, 1), (32, 32, 1), (32, 64, 2), (64, 64, 2), (64, 128, 3), (128, 128, 3),
          (192, 64, 2), (64, 64, 2), (96, 32, 1), (32, 32, 1), (48, 16, 0), (16, 16, 0), (16, 16, 0)]
OUT_SCALE = 22.4         # the trained network's output scale

_stream = None


def stream():
    """The one stream that every state's work runs on, as in a program with one simulation thread."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # the smallest: a spark of 257 vortons on a ragged grid, all on the GPU; launches and latency are the frame
        {"name": "device_spark", "kind": "device", "vortons": 257, "nx": 17, "ny": 15, "nz": 19, "tracers": 1021},
        # the benchmark's headline frame, end to end through host records
        {"name": "frame_ring", "kind": "frame", "vortons": 4096, "nx": 33, "ny": 33, "nz": 33, "tracers": 65536},
        # velocities of a large field at an odd number of scattered points
        {"name": "points_32k", "kind": "points", "vortons": 32768, "points": 200003},
        # the benchmark's treecode workload: eight rings, a million tracers
        {"name": "treecode_rings", "kind": "treecode", "vortons": 65536, "rings": 8, "tracers": 1048576},
        # the default particle operation of a small effect, odd count, called from a host program
        {"name": "plugin_small", "kind": "plugin", "vortons": 3001, "shape": "ring"},
        # the benchmark's multigrid workload with its four million tracers
        {"name": "poisson_puff", "kind": "poisson", "vortons": 262144, "nx": 129, "ny": 129, "nz": 129,
         "tracers": 4194304},
        # a large scene on a grid whose axes differ and are no powers of two
        {"name": "poisson_large", "kind": "poisson", "vortons": 1000003, "nx": 225, "ny": 161, "nz": 193,
         "tracers": 2000003},
        # the solver by itself, at the network's grid size
        {"name": "solve_129", "kind": "solve", "nx": 129, "ny": 129, "nz": 129},
        # a frame of 32 of the benchmark's batched effects
        {"name": "batch_32", "kind": "batch", "effects": 32, "streams": 8},
        # the network at the size it is trained for, forward
        {"name": "guess_128", "kind": "guess", "edge": 128},
        # and forward and backward on one BF16 pair, as a training run does
        {"name": "train_128", "kind": "train", "edge": 128, "bf16": True},
        # the operations around the step at the multigrid workload's sizes
        {"name": "scene_129", "kind": "scene", "vortons": 262144, "nx": 129, "ny": 129, "nz": 129,
         "tracers": 4194304},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["device", "frame", "points", "treecode", "plugin", "poisson", "solve", "batch", "guess", "train",
                       "scene"])
    if kind == "device":
        return {"kind": kind, "vortons": _log(rng, 100, 8192), "nx": rng.randint(9, 49), "ny": rng.randint(9, 49),
                "nz": rng.randint(9, 49), "tracers": _log(rng, 500, 200000)}
    if kind == "frame":
        return {"kind": kind, "vortons": _log(rng, 200, 8192), "nx": rng.randint(13, 41), "ny": rng.randint(13, 41),
                "nz": rng.randint(13, 41), "tracers": _log(rng, 1000, 100000)}
    if kind == "points":
        return {"kind": kind, "vortons": _log(rng, 300, 40000), "points": _log(rng, 1000, 200000)}
    if kind == "treecode":
        return {"kind": kind, "vortons": _log(rng, 2000, 262144), "rings": rng.randint(1, 12),
                "tracers": _log(rng, 10000, 2000000)}
    if kind == "plugin":
        return {"kind": kind, "vortons": _log(rng, 1000, 60000), "shape": rng.choice(["ring", "puff"])}
    if kind == "poisson":
        # the multigrid's grids: cell counts that halve, each axis its own
        return {"kind": kind, "vortons": _log(rng, 4000, 600000), "nx": 8 * rng.randint(4, 20) + 1,
                "ny": 8 * rng.randint(4, 20) + 1, "nz": 8 * rng.randint(4, 20) + 1, "tracers": _log(rng, 10000, 4000000)}
    if kind == "solve":
        return {"kind": kind, "nx": 8 * rng.randint(2, 24) + 1, "ny": 8 * rng.randint(2, 24) + 1,
                "nz": 8 * rng.randint(2, 24) + 1}
    if kind == "batch":
        return {"kind": kind, "effects": rng.randint(2, 32), "streams": rng.choice([1, 2, 4, 8])}
    if kind == "guess":
        return {"kind": kind, "edge": rng.choice([32, 64, 128]), "seed": rng.randint(0, 1 << 20)}
    if kind == "train":
        return {"kind": kind, "edge": rng.choice([32, 64, 128]), "bf16": rng.random() < 0.5,
                "seed": rng.randint(0, 1 << 20)}
    return {"kind": kind, "vortons": _log(rng, 4000, 400000), "nx": rng.randint(33, 140), "ny": rng.randint(33, 140),
            "nz": rng.randint(33, 140), "tracers": _log(rng, 50000, 4000000)}


# ---------------------------------------------------------------- inputs

def _gen(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * (int(seed) + 1) + 7919 * int(case.get("seed", 0)))
    return g


def _rand(g, n, lo, hi):
    return lo + (hi - lo) * torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64)


def _f4(xyz, w=None):
    o = torch.zeros((xyz.shape[0], 4), dtype=torch.float32, device="cuda")
    o[:, :3] = xyz.float()
    if w is not None:
        o[:, 3] = w
    return o


def _rings(g, n, count, box, tube=0.25, sigma=0.1, peak=10.0, major=(0.3, 1.0)):
    """n vortons in `count` vortex rings inside [-box, box]^3: positions and angular velocities (vorticity / 2)."""
    k = torch.arange(n, device="cuda") % count
    R = major[0] + (major[1] - major[0]) * torch.rand(count, generator=g, device="cuda", dtype=torch.float64)
    c = _rand(g, count, -1.0, 1.0) * (box - R - tube).clamp(min=0.0)[:, None]
    axis = torch.nn.functional.normalize(torch.randn((count, 3), generator=g, device="cuda", dtype=torch.float64), dim=1)
    e1 = torch.nn.functional.normalize(torch.linalg.cross(
        axis, torch.roll(axis, 1, dims=1) + torch.tensor([0.31, -0.17, 0.23], device="cuda", dtype=torch.float64)), dim=1)
    e2 = torch.linalg.cross(axis, e1)
    u = torch.rand((3, n), generator=g, device="cuda", dtype=torch.float64)
    phi, theta, r = 2 * math.pi * u[0], 2 * math.pi * u[1], tube * torch.sqrt(u[2])
    rho = (R[k] + r * torch.cos(theta))[:, None]
    cs, sn = torch.cos(phi)[:, None], torch.sin(phi)[:, None]
    pos = c[k] + rho * (cs * e1[k] + sn * e2[k]) + (r * torch.sin(theta))[:, None] * axis[k]
    mag = (peak * torch.exp(-r * r / (2 * sigma * sigma)))[:, None]
    return pos, 0.5 * mag * (cs * e2[k] - sn * e1[k])


def _puff(g, n, half, sigma=0.25):
    """A turbulent puff: Gaussian positions about the middle of a box of half extents `half`, i.i.d. vorticity."""
    h = torch.tensor(half, device="cuda", dtype=torch.float64)
    x = torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64) * sigma
    w = torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64) * 2.0
    return x.clamp(-0.95, 0.95) * h, 0.5 * w


def _box_grid(case, spacing):
    """A fixed grid of the case's points about the origin: (GridGeom, half extents)."""
    ext = [spacing * (case[a] - 1) for a in ("nx", "ny", "nz")]
    return vg.GridGeom.make([-0.5 * e for e in ext], ext, [case["nx"], case["ny"], case["nz"]]), [0.5 * e for e in ext]


def _inner(g, n, half, share):
    return _rand(g, n, -share, share) * torch.tensor(half, device="cuda", dtype=torch.float64)


def _direct_inputs(case, seed):
    """Grid, vortons and tracers of a direct-sum frame: a ring in a box, tracers in the box's inner part."""
    g = _gen(case, seed)
    half = [1.5, 1.5, 1.5]
    grid = vg.GridGeom.make([-1.5] * 3, [3.0] * 3, [case["nx"], case["ny"], case["nz"]])
    pos, w = _rings(g, case["vortons"], 1, 1.3, major=(0.9, 1.0))
    return grid, _f4(pos, 2 * RADIUS), _f4(w), _f4(_inner(g, case["tracers"], half, 0.93))


def _solve_inputs(case, seed):
    """A right-hand side like a puff's (white under an envelope) and smooth boundary values."""
    g = _gen(case, seed)
    grid, half = _box_grid(case, 1.0 / 32.0)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    ax = [torch.linspace(-1.0, 1.0, n, device="cuda", dtype=torch.float64) for n in (nx, ny, nz)]
    x, y, z = ax[0][None, None, :, None], ax[1][None, :, None, None], ax[2][:, None, None, None]
    env = torch.exp(-8.0 * (x * x + y * y + z * z))
    rhs = (env * torch.randn((nz, ny, nx, 3), generator=g, device="cuda", dtype=torch.float64) * 4.0).float()
    a = torch.randn((4, 3), generator=g, device="cuda", dtype=torch.float64) * 0.02
    soln = (a[0] * x + a[1] * y + a[2] * z + a[3] * torch.sin(2 * x + y) * torch.cos(z)).float()
    soln[1:-1, 1:-1, 1:-1] = 0.0
    return grid, rhs.contiguous(), soln.contiguous()


def _net_params(case, seed):
    """Parameters as a weight file holds them: BF16 weights (He-normal), FP32 biases."""
    g = _gen(case, seed + 101)
    parts = []
    for i, (ci, co, _) in enumerate(LAYERS):
        fan = 6 if i == 0 else ci
        w = torch.randn((27, co, ci), generator=g, device="cuda") * math.sqrt(2.0 / (1.01 * 27 * fan))
        if i == 0:
            w[:, :, 6:] = 0.0
        if i == len(LAYERS) - 1:
            w[:, 3:] = 0.0
        b = 0.05 * torch.randn(co, generator=g, device="cuda")
        if i == len(LAYERS) - 1:
            b[3:] = 0.0
        parts += [w.bfloat16().float().reshape(-1), b]
    return torch.cat(parts)


def _net_inputs(case, seed):
    """Right-hand side, vector potential with boundary values, on the network's grid."""
    e = case["edge"]
    grid, rhs, soln = _solve_inputs({"nx": e + 1, "ny": e + 1, "nz": e + 1, "seed": case.get("seed", 0)}, seed)
    return warmstart.field_grid(e + 1), rhs, soln


def _pair(case, seed):
    """A training pair: right-hand side and a smooth solution of its magnitude."""
    grid, rhs, soln = _net_inputs(case, seed)
    e = case["edge"]
    ax = torch.linspace(-1.0, 1.0, e + 1, device="cuda", dtype=torch.float64)
    x, y, z = ax[None, None, :, None], ax[None, :, None, None], ax[:, None, None, None]
    amp = torch.tensor([0.05, -0.04, 0.03], device="cuda", dtype=torch.float64)
    sol = (amp * torch.exp(-3.0 * (x * x + y * y + z * z)) + soln.double()).float()
    if case["bf16"]:
        return grid, rhs.bfloat16().contiguous(), sol.bfloat16().contiguous()
    return grid, rhs, sol.contiguous()


def _bodies():
    def body(shape, position, dims, hole=0.0, velocity=(0, 0, 0), spin=(0, 0, 0), rot=np.eye(3), temperature=300.0,
             conductivity=0.0):
        b = np.zeros(32, np.float32)
        b[0], b[1] = shape, hole
        b[2:5], b[5:8], b[8:11], b[11:20] = position, velocity, spin, np.asarray(rot, np.float32).ravel()
        b[20:20 + len(dims)] = dims
        b[23], b[24] = temperature, conductivity
        return b
    c, s = np.cos(0.3), np.sin(0.3)
    rot = np.array([[c, -s, 0], [s, c, 0], [0, 0, 1]])
    return np.ascontiguousarray(np.stack([
        body(0, (0.2, 0, 0), (0.4,), velocity=(0.5, 0, 0), spin=(0, 0, 1), temperature=350, conductivity=0.5),
        body(1, (0, 0, 0), (3.6, 3.6, 3.2), hole=1.0, rot=rot, conductivity=0.1),
        body(1, (0, 0.5, 0.3), (0.3, 0.4, 0.5), velocity=(0, 0.2, 0), spin=(0.3, 0, 0), rot=rot, temperature=320,
             conductivity=0.2)]))


def _scene_inputs(case, seed):
    g = _gen(case, seed)
    grid = vg.GridGeom.make([-2.0] * 3, [4.0] * 3, [case["nx"], case["ny"], case["nz"]])
    pos, w = _puff(g, case["vortons"], [2.0] * 3)
    ps, w = _f4(pos, 2 * RADIUS), _f4(w)
    dens = (1.0 + 0.2 * torch.exp(-(pos ** 2).sum(1) / 0.2)).float()
    tr = _f4(_rand(g, case["tracers"], -1.9, 1.9), 0.01)
    trv = _f4(torch.randn((case["tracers"], 3), generator=g, device="cuda", dtype=torch.float64))
    return grid, ps, w, dens, tr, trv


def _effects(case, seed):
    """The benchmark's effects (their counts and grids), each with its vortons shaken and turned by the seed."""
    rng = np.random.default_rng(int(seed))
    effects = []
    for i in range(case["effects"]):
        e = vgbatch.make_effect(1000 + i)
        half = 0.5 * float(e.grid.extent[0])
        e.pos = np.clip(e.pos + rng.normal(0.0, 0.02 * half, e.pos.shape), -0.8 * half, 0.8 * half).astype(np.float32)
        e.vort = (e.vort * rng.uniform(0.7, 1.3)).astype(np.float32)
        effects.append(e)
    return effects


def _config(**kw):
    cfg = vg.default_config(**kw)
    cfg.stream = stream().cuda_stream
    return cfg


def _pinned(records):
    t = torch.empty(records.nbytes, dtype=torch.uint8, pin_memory=True)
    a = t.numpy().view(vg.PARTICLE_DTYPE)
    a[...] = records
    return a, t


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "run": globals()["_run_" + kind]}
    if kind in ("device", "frame"):
        grid, ps, w, tr = _direct_inputs(case, seed)
        s["sim"] = vg.VortonSim(cfg=_config(velocity_technique=vg.VELOCITY_DIRECT, fixed_grid=grid, enable_stretch=0,
                                            enable_diffusion=0))
        if kind == "device":
            s.update(ps=ps, w=w, vel=torch.zeros_like(ps), tr=tr, trv=torch.zeros_like(tr))
            s["grid"] = grid
        else:
            rec = vg.make_particles(ps[:, :3].cpu().numpy(), w[:, :3].cpu().numpy(), ps[:, 3].cpu().numpy())
            s["rec"], s["keep0"] = _pinned(rec)
            s["trec"], s["keep1"] = _pinned(vg.make_particles(tr[:, :3].cpu().numpy()))
    elif kind == "points":
        g = _gen(case, seed)
        pos, w = _rings(g, case["vortons"], 4, 2.0)
        s.update(ctx=vg.Context(_config()), ps=_f4(pos, 2 * RADIUS), w=_f4(w), q=_f4(_rand(g, case["points"], -2.0, 2.0)))
        s["out"] = torch.zeros_like(s["q"])
    elif kind == "treecode":
        g = _gen(case, seed)
        pos, w = _rings(g, case["vortons"], case["rings"], 2.0)
        s.update(sim=vg.VortonSim(cfg=_config(velocity_technique=vg.VELOCITY_TREE, enable_stretch=0, enable_diffusion=0)),
                 ps=_f4(pos, 2 * RADIUS), w=_f4(w), tr0=_f4(_rand(g, case["tracers"], -1.8, 1.8)),
                 box=np.array([-1.8] * 3 + [1.8] * 3, np.float32))
        s.update(vel=torch.zeros_like(s["ps"]), tr=s["tr0"].clone(), trv=torch.zeros_like(s["tr0"]))
    elif kind == "plugin":
        g = _gen(case, seed)
        pos, w = _rings(g, case["vortons"], 1, 1.4) if case["shape"] == "ring" else _puff(g, case["vortons"], [1.5] * 3)
        s["op"] = vg.PclOpVortonSim(cfg=_config())
        s["rec0"] = vg.make_particles(pos.float().cpu().numpy(), w.float().cpu().numpy(),
                                      np.full(case["vortons"], 2 * RADIUS, np.float32))
        s["rec"] = s["rec0"].copy()
    elif kind == "poisson":
        g = _gen(case, seed)
        grid, half = _box_grid(case, 1.0 / 32.0)
        pos, w = _puff(g, case["vortons"], half)
        s.update(sim=vg.VortonSim(cfg=_config(fixed_grid=grid)), ps=_f4(pos, 2 * RADIUS), w0=_f4(w),
                 tr0=_f4(_inner(g, case["tracers"], half, 0.95)))
        s.update(w=s["w0"].clone(), vel=torch.zeros_like(s["ps"]), tr=s["tr0"].clone(), trv=torch.zeros_like(s["tr0"]))
    elif kind == "solve":
        s["grid"], s["rhs"], s["soln0"] = _solve_inputs(case, seed)
        s["ctx"], s["soln"] = vg.Context(_config()), s["soln0"].clone()
        s["out"] = (ctypes.c_int(), ctypes.c_double(), ctypes.c_double())
    elif kind == "batch":
        s["batch"] = vgbatch.Batch(_effects(case, seed), streams=case["streams"])
        s["batch"].calibrate(1.0 / 60.0)
        s["batch"].step(1.0 / 60.0)
        s["batch"].synchronize()
    elif kind in ("guess", "train"):
        s["net"] = warmstart.Network(case["edge"], 0, stream())
        s["net"].set_params(_net_params(case, seed).cpu().numpy(), OUT_SCALE)
        if kind == "guess":
            s["grid"], s["rhs"], s["vp"] = _net_inputs(case, seed)
        else:
            s["grid"], s["rhs"], s["vp"] = _pair(case, seed)
    elif kind == "scene":
        s["grid"], s["ps0"], s["w0"], s["dens0"], s["tr0"], s["trv0"] = _scene_inputs(case, seed)
        s.update(ctx=vg.Context(_config()), bodies=_bodies(), grav=np.array([0, -9.8, 0], np.float32),
                 wind=np.array([1, 0, 0], np.float32))
        for k in ("ps", "w", "dens", "tr", "trv"):
            s[k] = s[k + "0"].clone()
        pts = s["grid"].capacity
        s["vel"] = torch.zeros_like(s["ps"])
        s["grid_dens"] = torch.zeros(pts, device="cuda")
        s["sdf"] = torch.zeros(pts, device="cuda")
        s["verts"] = torch.zeros((2 * pts, 9), device="cuda")
        n = len(s["bodies"])
        s.update(tris=ctypes.c_size_t(), applied=ctypes.c_int(), hits=np.zeros(n, np.uint64),
                 out9=np.zeros((n, 9), np.float32), out6=np.zeros((n, 6), np.float32))
    return s


# ---------------------------------------------------------------- the passes

def run(s):
    with torch.cuda.stream(stream()):
        return s["run"](s)


def _run_device(s):
    sim = s["sim"]
    sim.UpdateAndEvolveDevice(s["ps"], s["w"], s["vel"], SLOW_DT)
    sim.AdvectDevice(s["tr"], s["trv"], SLOW_DT)
    return [s["ps"], s["vel"], s["tr"], s["trv"]]


def _run_frame(s):
    s["sim"].UpdateAndAdvect(s["rec"], s["trec"], SLOW_DT)
    return [s["rec"]["position"], s["rec"]["velocity"], s["trec"]["position"], s["trec"]["velocity"]]


def _run_points(s):
    ctx, ps, q = s["ctx"], s["ps"], s["q"]
    ctx.check(vg.lib().vg_direct_device(ctx.h, 0, vg._ptr(ps), vg._ptr(s["w"]), ps.shape[0], vg._ptr(q), q.shape[0], 1.0,
                                        1.0, vg._ptr(s["out"])), "vg_direct_device")
    return s["out"]


def _run_treecode(s):
    s["tr"].copy_(s["tr0"])
    s["sim"].UpdateDevice(s["ps"], s["w"], s["vel"], DT, extra_minmax=s["box"])
    s["sim"].AdvectDevice(s["tr"], s["trv"], DT)
    return [s["vel"], s["tr"], s["trv"]]


def _run_plugin(s):
    s["rec"].view(np.uint8)[...] = s["rec0"].view(np.uint8)
    s["op"].Operate(s["rec"], DT)
    return [s["rec"]["velocity"], s["rec"]["angular_velocity"]]


def _run_poisson(s):
    s["w"].copy_(s["w0"])
    s["tr"].copy_(s["tr0"])
    s["sim"].UpdateDevice(s["ps"], s["w"], s["vel"], DT)
    s["sim"].AdvectDevice(s["tr"], s["trv"], DT)
    return [s["vel"], s["w"], s["tr"], s["trv"]]


def _run_solve(s):
    ctx, (cyc, r0, r1) = s["ctx"], s["out"]
    s["soln"].copy_(s["soln0"])
    ctx.check(vg.lib().vg_multigrid_device(ctx.h, ctypes.byref(s["grid"]), vg._ptr(s["soln"]), vg._ptr(s["rhs"]), 1e-6, 50,
                                           ctypes.byref(cyc), ctypes.byref(r0), ctypes.byref(r1)), "vg_multigrid_device")
    return s["soln"]


def _run_batch(s):
    s["batch"].step(1.0 / 60.0)
    return [t for p, _, v in s["batch"].arrays for t in (p, v)]


def _run_guess(s):
    s["net"].guess(s["grid"], s["rhs"], s["vp"])
    return s["vp"]


def _run_train(s):
    loss = s["net"].backward(s["grid"], s["rhs"], s["vp"], want_loss=True)
    return [loss, s["net"].grads()]


def _run_scene(s):
    ctx, L, P, g = s["ctx"], vg.lib(), vg._ptr, ctypes.byref(s["grid"])
    n, m, b = s["ps"].shape[0], s["tr"].shape[0], s["bodies"]
    for k in ("ps", "w", "dens", "tr", "trv"):
        s[k].copy_(s[k + "0"])
    s["vel"].zero_()
    ctx.check(L.vg_density_grid_device(ctx.h, g, P(s["ps"]), P(s["dens"]), n, 1.0, P(s["grid_dens"])), "density grid")
    ctx.check(L.vg_signed_distance_device(ctx.h, g, P(s["grid_dens"]), 1.0, 0, P(s["sdf"])), "signed distance")
    ctx.check(L.vg_marching_cubes_device(ctx.h, g, P(s["sdf"]), 0.0, P(s["verts"]), None, s["verts"].shape[0],
                                         ctypes.byref(s["tris"])), "marching cubes")
    ctx.check(L.vg_heat_pse_device(ctx.h, g, P(s["ps"]), P(s["dens"]), n, 1e-3, 1.0, DT), "heat diffusion")
    ctx.check(L.vg_baroclinic_device(ctx.h, g, P(s["ps"]), P(s["dens"]), P(s["w"]), n, P(s["grav"]), 1.0, DT,
                                     ctypes.byref(s["applied"])), "baroclinic generation")
    ctx.check(L.vg_collide_vortons_device(ctx.h, P(b), len(b), P(s["ps"]), P(s["vel"]), P(s["w"]), P(s["dens"]), n, 1.0,
                                          1.0, P(s["out9"]), P(s["hits"])), "vorton collisions")
    ctx.check(L.vg_wind_device(ctx.h, P(s["trv"]), m, P(s["wind"]), 0.125, 0.875), "wind")
    ctx.check(L.vg_collide_tracers_device(ctx.h, P(b), len(b), P(s["tr"]), P(s["trv"]), None, m, P(s["out6"])),
              "tracer collisions")
    return [s["grid_dens"], s["sdf"], s["verts"], s["tris"].value, s["ps"], s["vel"], s["w"], s["dens"], s["tr"],
            s["trv"], s["out9"], s["out6"], s["hits"].astype(np.int64)]


# ---------------------------------------------------------------- the work of one pass

def _points_of(case):
    return case["nx"] * case["ny"] * case["nz"]


def _conv_flops(edge):
    return sum(2.0 * 27 * ci * co * (edge >> lv) ** 3 for ci, co, lv in LAYERS)


def _poisson_flops(pts):
    """A fast transform solve of three components: what a Poisson solve of so many points takes at least."""
    return 15.0 * pts * math.log2(pts)


def work(case):
    kind = case["kind"]
    if kind in ("device", "frame"):
        n, m, pts = case["vortons"], case["tracers"], _points_of(case)
        rec = 96 if kind == "frame" else 16
        return {"bytes": n * (32 + 32 if kind == "device" else 2 * rec) + m * (48 if kind == "device" else 2 * rec),
                "flops": FLOPS_PER_PAIR * n * (n + pts) + 45 * m}
    if kind == "points":
        return {"bytes": 32 * (case["vortons"] + case["points"]), "flops": FLOPS_PER_PAIR * case["vortons"] * case["points"]}
    if kind == "treecode":
        n, m = case["vortons"], case["tracers"]
        # about one grid cell per vorton; eight pair laws a layer at every gridpoint
        return {"bytes": 48 * n + 12 * n + 48 * m, "flops": FLOPS_PER_PAIR * 8 * math.log2(n) / 3 * n + 45 * m}
    if kind == "plugin":
        n = case["vortons"]
        return {"bytes": 2 * 96 * n, "flops": _poisson_flops(n) + 300 * n}
    if kind == "poisson":
        n, m, pts = case["vortons"], case["tracers"], _points_of(case)
        return {"bytes": 64 * n + 12 * pts + 48 * m, "flops": _poisson_flops(pts) + 300 * n + 45 * m}
    if kind == "solve":
        pts = _points_of(case)
        return {"bytes": 24 * pts, "flops": _poisson_flops(pts)}
    if kind == "batch":
        # the effects' medians: 8,192 vortons, 81^3 points
        k = case["effects"]
        return {"bytes": k * (64.0 * 8192 + 24 * 81 ** 3), "flops": k * (_poisson_flops(81 ** 3) + 300 * 8192)}
    if kind in ("guess", "train"):
        e, times = case["edge"], 1 if kind == "guess" else 3
        size = 2 if case.get("bf16") else 4
        return {"bytes": (e + 1) ** 3 * (3 * size + (12 if kind == "guess" else 3 * size)) + 6e6 * times,
                "flops": times * _conv_flops(e)}
    n, m, pts = case["vortons"], case["tracers"], _points_of(case)
    return {"bytes": 104 * n + 64 * m + 8 * pts, "flops": 300 * n + 100 * m + 50 * pts}


# ---------------------------------------------------------------- the same in 64 bits

def _velocity64(q, ps, w):
    """The mollified Biot-Savart sum at points q (float64 [m, 3])."""
    p, r = ps[:, :3].double(), 0.5 * ps[:, 3].double()
    a = w[:, :3].double() * ((2.0 / 3.0) * r ** 3)[:, None]
    right = torch.cat([a, torch.linalg.cross(a, p)], dim=1)
    out = torch.empty((q.shape[0], 3), dtype=torch.float64, device="cuda")
    step = max(1, (1 << 27) // max(1, p.shape[0]))
    for i in range(0, q.shape[0], step):
        x = q[i:i + step]
        d2 = (x[:, 0:1] - p[None, :, 0]) ** 2
        d2 += (x[:, 1:2] - p[None, :, 1]) ** 2
        d2 += (x[:, 2:3] - p[None, :, 2]) ** 2
        law = torch.where(d2 < r * r, 1.0 / r ** 3, d2.clamp(min=1e-300) ** -1.5)
        f = law @ right
        out[i:i + step] = torch.linalg.cross(f[:, :3], x) - f[:, 3:]
    return out


def _grid_positions(grid):
    nudge = np.float32(1.0) - np.float32(2.0) * np.finfo(np.float32).eps
    ax = [np.float32(grid.min_corner[a]) + np.arange(grid.num_points[a], dtype=np.float32) *
          (np.float32(grid.cell_spacing[a]) * nudge) for a in range(3)]
    z, y, x = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    return torch.from_numpy(np.stack([x.ravel(), y.ravel(), z.ravel()], 1).astype(np.float64)).cuda()


def _trilinear64(grid, field, p):
    """field [points, k] (float64) at positions p [m, 3]."""
    np3 = grid.points
    f = field.reshape(np3[2], np3[1], np3[0], -1)
    idx, t = [], []
    for a in range(3):
        u = (p[:, a] - float(grid.min_corner[a])) / float(grid.cell_spacing[a])
        i = u.floor().long().clamp(0, np3[a] - 2)
        idx.append(i)
        t.append((u - i)[:, None])
    out = 0.0
    for dz in (0, 1):
        for dy in (0, 1):
            for dx in (0, 1):
                wgt = (t[0] if dx else 1 - t[0]) * (t[1] if dy else 1 - t[1]) * (t[2] if dz else 1 - t[2])
                out = out + wgt * f[idx[2] + dz, idx[1] + dy, idx[0] + dx]
    return out


def _exact_direct(case, seed):
    grid, ps, w, tr = _direct_inputs(case, seed)
    p = ps[:, :3].double()
    v = _velocity64(p, ps, w)
    tp = tr[:, :3].double()
    tv = _trilinear64(grid, _velocity64(_grid_positions(grid), ps, w), tp)
    new, tnew = p + v * SLOW_DT, tp + tv * SLOW_DT
    if case["kind"] == "frame":
        return [new, v, tnew, tv]
    pad = lambda x, c: torch.cat([x, torch.full_like(x[:, :1], c)], dim=1)  # noqa: E731
    return [torch.cat([new, ps[:, 3:].double()], dim=1), pad(v, 0.0), pad(tnew, 0.0), pad(tv, 0.0)]


def _sine(n):
    k = torch.arange(1, n + 1, device="cuda", dtype=torch.float64)
    return torch.sin(math.pi * k[:, None] * k[None, :] / (n + 1)) * math.sqrt(2.0 / (n + 1))


def _exact_solve(case, seed):
    """The seven-point operator's solution, by sine transforms along each axis."""
    grid, rhs, soln = _solve_inputs(case, seed)
    h = [1.0 / float(grid.cell_spacing[a]) ** 2 for a in range(3)]
    x = soln.double()
    b = rhs.double()[1:-1, 1:-1, 1:-1].clone()
    b[:, :, 0] -= h[0] * x[1:-1, 1:-1, 0]
    b[:, :, -1] -= h[0] * x[1:-1, 1:-1, -1]
    b[:, 0] -= h[1] * x[1:-1, 0, 1:-1]
    b[:, -1] -= h[1] * x[1:-1, -1, 1:-1]
    b[0] -= h[2] * x[0, 1:-1, 1:-1]
    b[-1] -= h[2] * x[-1, 1:-1, 1:-1]
    n = [case["nx"] - 2, case["ny"] - 2, case["nz"] - 2]
    S = [_sine(k) for k in n]
    lam = [-4.0 * h[a] * torch.sin(math.pi * torch.arange(1, n[a] + 1, device="cuda", dtype=torch.float64) /
                                   (2 * (n[a] + 1))) ** 2 for a in range(3)]

    def spin(v):
        return torch.einsum("kz,zyxc->kyxc", S[2], torch.einsum("jy,zyxc->zjxc", S[1],
                                                               torch.einsum("ix,zyxc->zyic", S[0], v)))
    t = spin(b) / (lam[0][None, None, :, None] + lam[1][None, :, None, None] + lam[2][:, None, None, None])
    x[1:-1, 1:-1, 1:-1] = spin(t)
    return x


def _conv64(x, w, b):
    """3x3x3 convolution of x [z, y, x, ci] with w [27, co, ci], zero outside."""
    n = x.shape[0]
    xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    out = b.expand(n, n, n, w.shape[1]).clone()
    for t in range(27):
        dz, dy, dx = t // 9, t // 3 % 3, t % 3
        out = out + xp[dz:dz + n, dy:dy + n, dx:dx + n] @ w[t].T
    return out


def _net64(case, params, rhs, vp, cell):
    """The network's output [n, n, n, 16], and the scale of its output."""
    n = case["edge"]
    h2 = sum(c * c for c in cell) / 3.0 * OUT_SCALE
    s = rhs.double().pow(2).mean().sqrt()
    x = torch.zeros((n, n, n, 16), dtype=torch.float64, device="cuda")
    x[..., :3] = rhs[:n, :n, :n].double() / s
    k = torch.arange(n, device="cuda")
    low = (k[:, None, None] == 0) | (k[None, :, None] == 0) | (k[None, None, :] == 0)
    high = ~low & ((k[:, None, None] == n - 1) | (k[None, :, None] == n - 1) | (k[None, None, :] == n - 1))
    up = torch.where(k == n - 1, n, k)
    v = vp.double()
    x[..., 3:6] = torch.where(low[..., None], v[:n, :n, :n], torch.where(
        high[..., None], v[up][:, up][:, :, up], torch.zeros((), dtype=torch.float64, device="cuda"))) / (s * h2)
    W, at = [], 0
    for ci, co, _ in LAYERS:
        W.append((params[at:at + 27 * ci * co].reshape(27, co, ci), params[at + 27 * ci * co:at + 27 * ci * co + co]))
        at += 27 * ci * co + co

    def conv(i, y):
        y = _conv64(y, *W[i])
        return y if i == len(LAYERS) - 1 else torch.nn.functional.leaky_relu(y, 0.1)

    def pool(y):
        m = y.shape[0] // 2
        return y.reshape(m, 2, m, 2, m, 2, -1).mean(dim=(1, 3, 5))

    def double(y):
        return y.repeat_interleave(2, 0).repeat_interleave(2, 1).repeat_interleave(2, 2)
    e0 = conv(1, conv(0, x))
    e1 = conv(3, conv(2, pool(e0)))
    e2 = conv(5, conv(4, pool(e1)))
    e3 = conv(7, conv(6, pool(e2)))
    d2 = conv(9, conv(8, torch.cat([double(e3), e2], dim=3)))
    d1 = conv(11, conv(10, torch.cat([double(d2), e1], dim=3)))
    d0 = conv(13, conv(12, torch.cat([double(d1), e0], dim=3)))
    return conv(14, d0), s * h2


def _exact_guess(case, seed):
    grid, rhs, vp = _net_inputs(case, seed)
    with torch.no_grad():
        out, scale = _net64(case, _net_params(case, seed).double(), rhs, vp, [float(c) for c in grid.cell_spacing])
    n = case["edge"]
    x = vp.double()
    x[1:n, 1:n, 1:n] = out[1:, 1:, 1:, :3] * scale
    return x


def _exact_train(case, seed):
    grid, rhs, vp = _pair(case, seed)
    params = _net_params(case, seed).double().requires_grad_(True)
    out, scale = _net64(case, params, rhs, vp, [float(c) for c in grid.cell_spacing])
    n = case["edge"]
    t = vp.double()[1:n, 1:n, 1:n] / scale
    loss = (out[1:, 1:, 1:, :3] - t).pow(2).sum() / t.pow(2).sum()
    loss.backward()
    return [float(loss.detach()), params.grad]


def _exact_density(case, seed):
    """The density grid: the vortons' mass spread to the corners of their cells, the ambient where there is none."""
    grid, ps, _, dens, _, _ = _scene_inputs(case, seed)
    np3 = grid.points
    vol = math.pi / 6.0 * float(ps[0, 3]) ** 3
    cell = math.prod(float(c) for c in grid.cell_spacing)
    idx, t = [], []
    for a in range(3):
        u = (ps[:, a].double() - float(grid.min_corner[a])) / float(grid.cell_spacing[a])
        i = u.floor().long().clamp(0, np3[a] - 2)
        idx.append(i)
        t.append(u - i)
    mass = torch.zeros(grid.capacity, dtype=torch.float64, device="cuda")
    part = torch.zeros_like(mass)
    for dz in (0, 1):
        for dy in (0, 1):
            for dx in (0, 1):
                wgt = (t[0] if dx else 1 - t[0]) * (t[1] if dy else 1 - t[1]) * (t[2] if dz else 1 - t[2])
                at = idx[0] + dx + np3[0] * (idx[1] + dy + np3[1] * (idx[2] + dz))
                part.index_add_(0, at, wgt * (vol / cell))
                mass.index_add_(0, at, wgt * (vol / cell) * dens.double())
    return [mass + (1.0 - part).clamp(min=0.0)] + [None] * 12


def exact(case, seed):
    kind = case["kind"]
    if kind in ("device", "frame"):
        return _exact_direct(case, seed)
    if kind == "points":
        g = _gen(case, seed)
        pos, w = _rings(g, case["vortons"], 4, 2.0)
        v = _velocity64(_rand(g, case["points"], -2.0, 2.0).float().double(), _f4(pos, 2 * RADIUS), _f4(w))
        return torch.cat([v, torch.zeros_like(v[:, :1])], dim=1)
    if kind == "solve":
        return _exact_solve(case, seed)
    if kind == "guess":
        return _exact_guess(case, seed)
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "scene":
        return _exact_density(case, seed)
    # the treecode's far field and the steps that rest on it have no plain definition; the batch carries its own state on
    return None
