"""What a user of this package has it do, as cases to time.

A case is a simulation between two outputs: `steps` explicit MPM steps of a scene that
is on the GPU already, then the download of the particle state the program writes to
disk, as the driver's main loop does between two dumps.  Scenes are the repository's
own workloads (elastic sphere collision, dam break, axial bar, twisted column with
obstacles and heat, heated block, batched dam breaks), from a few thousand particles,
where a step is a dozen short launches, to the nine million of the headline workload,
in both precisions, all three B-spline orders, USL and MUSL, with and without
temperature, lattice-like and disordered particles, walls and periodic faces, through
the fused step, the batched step and the one-by-one step functions.

A mixed-precision run's state and results carry FP32 rounding, so the program keeps
them as FP32; an FP64 run's are FP64.
"""
import math

import numpy as np
import torch

from exagoop_b200 import native as nt
from exagoop_b200 import scenes

DEV = "cuda:0"
# literal constants of the particle generator (volume of a sphere of the lattice radius)
FOURBYTHREE, PI = 1.3333333333, 3.141592654


def listed():
    return [
        # 1-D validation runs: a few thousand particles, linear shape functions, many
        # steps; launch latency is all there is
        dict(name="bar 8k fp64 linear", kind="bar", n=64, order=1, fp64=True, steps=200),
        # a small dam break of a parameter study, FP64 against the reference's numbers
        dict(name="dam 15k fp64", kind="dam", nx=32, ny=16, nz=16, order=2, fp64=True, jitter=0.25, steps=100),
        # a reference-style main loop that calls the step functions one by one
        dict(name="spheres 140k step calls", kind="spheres", n=64, order=3, fp64=False, jitter=0.1, calls=True, steps=20),
        # thermo-mechanical block, MUSL, thermal walls of every kind, ragged grid
        dict(name="heated block 290k fp64 musl", kind="block", nx=45, ny=30, nz=38, order=2, fp64=True, musl=True,
             steps=40),
        # a middle-sized collision on a grid that is no multiple of a tile
        dict(name="spheres 540k mixed", kind="spheres", n=100, order=3, fp64=False, jitter=0.1, steps=150),
        # a dam break under way: particles at random, periodic in y
        dict(name="dam 0.9M mixed periodic", kind="dam", nx=123, ny=64, nz=61, order=2, fp64=False, jitter=1.0,
             periodic=True, steps=150),
        # the collision in FP64
        dict(name="spheres 1.1M fp64", kind="spheres", n=128, order=3, fp64=True, jitter=0.1, steps=100),
        # the column at its benchmark size: heat, obstacles, rigid particles
        dict(name="column 1.6M mixed heat", kind="column", nx=64, ny=64, nz=384, order=2, fp64=False, steps=60),
        # a batch of uneven dam breaks
        dict(name="batch of 16 dams mixed", kind="batch", scenes=16, lo=32, hi=64, order=2, fp64=False, steps=100),
        # the second benchmark workload
        dict(name="dam 8M mixed", kind="dam", nx=256, ny=128, nz=128, order=2, fp64=False, jitter=0.25, steps=300),
        # the headline workload
        dict(name="spheres 9M mixed", kind="spheres", n=256, order=3, fp64=False, jitter=0.1, steps=300),
    ]


def draw(rng):
    """One more run of the same kinds: sizes spread over their logarithm."""
    kind = rng.choice(["bar", "dam", "dam", "spheres", "spheres", "block", "column", "batch"])
    fp64 = rng.random() < 0.4
    np_ = math.exp(rng.uniform(math.log(1.5e4), math.log(4e6)))
    if kind == "bar":
        c = dict(kind=kind, n=rng.randint(40, 400), order=1, fp64=fp64)
        return dict(c, steps=rng.randint(100, 200))
    if kind == "batch":
        c = dict(kind=kind, scenes=rng.randint(3, 24), lo=rng.randint(20, 32), hi=rng.randint(40, 64),
                 order=rng.choice([2, 2, 3]), fp64=fp64)
        return dict(c, steps=rng.randint(30, 80))
    steps = max(20, min(150, int(1.5e8 / np_)))
    if kind == "spheres":
        # 0.067 of the cube's cells are filled, 8 particles each
        c = dict(kind=kind, n=int((np_ / 8 / 0.067) ** (1 / 3)), order=rng.choice([3, 3, 2]), fp64=fp64,
                 jitter=rng.choice([0.0, 0.1, 0.25]))
        if rng.random() < 0.25 and np_ < 5e5:
            return dict(c, calls=True, steps=rng.randint(5, 20))
        return dict(c, steps=steps)
    if kind == "dam":
        a = (np_ / 8 / 0.24 / 2) ** (1 / 3)  # a long tank, a quarter of it water
        ny = max(24, int(a))
        c = dict(kind=kind, nx=int(2 * a) + rng.randint(0, 7), ny=ny, nz=int(a) + rng.randint(0, 7),
                 order=rng.choice([2, 2, 3, 1]), fp64=fp64, jitter=rng.choice([0.25, 1.0]), musl=rng.random() < 0.2)
        if rng.random() < 0.3:
            c = dict(c, ny=ny // 8 * 8, periodic=True)
        return dict(c, steps=steps)
    if kind == "block":
        a = (min(np_, 6e5) / 8 / 0.7) ** (1 / 3)
        return dict(kind=kind, nx=int(1.2 * a), ny=max(8, int(0.8 * a)), nz=int(a), order=rng.choice([2, 3]), fp64=fp64,
                    musl=rng.random() < 0.5, steps=rng.randint(10, 40))
    n = max(16, int(64 * (min(np_, 1.6e6) / 1.57e6) ** (1 / 3)))
    return dict(kind=kind, nx=n, ny=n, nz=6 * n, order=2, fp64=fp64, steps=rng.randint(20, 60))


# ------------------------------------------------------------------ scenes
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64)


def _lattice(lo, hi, dx, ppc=2):
    """Points at (k + 1/2) / ppc of a cell in the box [lo, hi), x fastest: [3, n]."""
    ax = []
    for d in range(3):
        h = dx[d] / ppc
        n = int(math.floor((hi[d] - lo[d]) / h + 1e-9))
        ax.append(lo[d] + 0.5 * h + h * torch.arange(n, device=DEV, dtype=torch.float64))
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    return torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)])


def _fluid(sc, block, jitter, g):
    """Water in the low corner of a tank: Tait K = 2e6, gamma = 7, rho = 1000, mu = 1e-3."""
    dx, size = sc["dx"], sc["size"]
    pos = _lattice((0, 0, 0), block, dx)
    pos += (2 * jitter) * (_rand(g, *pos.shape) - 0.5) * torch.tensor(dx, device=DEV)[:, None]
    for d in range(3):
        if sc["periodic"][d]:
            pos[d] = torch.remainder(pos[d], size[d])
        pos[d].clamp_(1e-9 * size[d], size[d] * (1 - 1e-9))
    vel = torch.zeros_like(pos)
    return dict(sc, pos=pos, vel=vel, rho0=1000.0, model=1, K=2e6, gamma=7.0, visc=1e-3, E=0.0, nu=0.0)


def _box(n, size, order, alpha=0.99, gravity=(0.0, 0.0, 0.0), cfl=0.1):
    return dict(n=tuple(n), size=tuple(size), dx=tuple(size[d] / n[d] for d in range(3)), order=order, alpha=alpha,
                gravity=gravity, cfl=cfl, timestep=None, periodic=(0, 0, 0), slip=[[2, 2], [2, 2], [2, 2]], heat=False)


def _scene(case, seed):
    """Grid, parameters and particles of a case, as plain values and FP64 tensors."""
    g = _gen(seed)
    kind = case["kind"]
    if kind == "bar":
        n, dx = case["n"], 1.0 / case["n"]
        sc = _box((n, 4, 4), (1.0, 4 * dx, 4 * dx), 1)
        sc["timestep"] = 0.1 * dx / 10.0  # c = sqrt(E / rho) = 10
        sc["slip"][0][0] = 1
        pos = _lattice((0, 0, 0), sc["size"], sc["dx"])
        vel = torch.zeros_like(pos)
        vel[0] = 0.1 * torch.sin(0.5 * math.pi * pos[0]) * (1 + 0.01 * (_rand(g, pos.shape[1]) - 0.5))
        return dict(sc, pos=pos, vel=vel, rho0=1.0, model=0, E=100.0, nu=0.0, K=0.0, gamma=0.0, visc=0.0)
    if kind == "dam":
        n = (case["nx"], case["ny"], case["nz"])
        size = tuple(k / 256.0 for k in n)
        sc = _box(n, size, case["order"], gravity=(0.0, 0.0, -9.81))
        if case.get("periodic"):
            sc["periodic"] = (0, 1, 0)
        return _fluid(sc, (0.4 * size[0], size[1], 0.6 * size[2]), case["jitter"], g)
    if kind == "spheres":
        n = case["n"]
        sc = _box((n, n, n), (1.0, 1.0, 1.0), case["order"])
        h = 0.5 / n
        lo = [math.floor(v / (2 * h)) * 2 * h for v in (0.1, 0.3, 0.3)]
        hi = [math.ceil(v / (2 * h)) * 2 * h for v in (0.9, 0.7, 0.7)]
        pos = _lattice(lo, hi, sc["dx"])
        r2 = [sum((pos[d] - c[d]) ** 2 for d in range(3)) for c in ((0.3, 0.5, 0.5), (0.7, 0.5, 0.5))]
        left, right = r2[0] < 0.04, r2[1] < 0.04
        keep = left | right
        sign = torch.where(left, 1.0, -1.0)[keep].double()
        pos = pos[:, keep].contiguous()
        pos += (2 * case["jitter"] / n) * (_rand(g, *pos.shape) - 0.5)
        vel = 1e-3 * (_rand(g, *pos.shape) - 0.5)
        vel[0] += 0.1 * sign
        return dict(sc, pos=pos, vel=vel, rho0=1000.0, model=0, E=1e3, nu=0.3, K=0.0, gamma=0.0, visc=0.0)
    if kind == "block":
        n = (case["nx"], case["ny"], case["nz"])
        size = tuple(0.05 * k for k in n)
        sc = _box(n, size, case["order"], alpha=0.95, gravity=(0.0, 0.0, -9.81), cfl=0.2)
        sc["heat"] = True
        pos = _lattice((0, 0, 0), (size[0], size[1], 0.7 * size[2]), sc["dx"])
        pos += 0.4 * (_rand(g, *pos.shape) - 0.5) * torch.tensor(sc["dx"], device=DEV)[:, None]
        for d in range(3):
            pos[d].clamp_(1e-9 * size[d], size[d] * (1 - 1e-9))
        m = pos.shape[1]
        vel = 0.02 * torch.randn(3, m, generator=g, device=DEV, dtype=torch.float64)
        return dict(sc, pos=pos, vel=vel, rho0=2000.0, model=0, E=1e6, nu=0.25, K=0.0, gamma=0.0, visc=0.0,
                    T=280 + 40 * _rand(g, m), cp=900.0, kc=50.0, Q=1e5 * (0.5 + _rand(g, m)))
    # twisted column standing on a noslip base among spherical obstacles
    n, size, col = (case["nx"], case["ny"], case["nz"]), (0.2, 0.2, 1.2), (0.1, 0.1, 0.6)
    sc = _box(n, size, case["order"])
    sc["slip"][2][0] = 1
    sc["heat"] = True
    pos = _lattice((0.05, 0.05, 0.0), (0.15, 0.15, 0.6), sc["dx"])
    m = pos.shape[1]
    vel = torch.zeros_like(pos)
    vel[0], vel[1] = -10.0 * (pos[1] - 0.1), 10.0 * (pos[0] - 0.1)
    rng = np.random.default_rng(4321)
    spheres = []
    while len(spheres) < 20:
        r = rng.uniform(0.02, 0.05)
        c = rng.uniform([r, r, r], [size[0] - r, size[1] - r, size[2] - r])
        if not (abs(c[0] - 0.1) < 0.05 + r and abs(c[1] - 0.1) < 0.05 + r and c[2] < col[2] + r):
            spheres.append((tuple(float(v) for v in c), float(r)))
    return dict(sc, pos=pos, vel=vel, rho0=1000.0, model=0, E=1e5, nu=0.3, K=0.0, gamma=0.0, visc=0.0,
                T=300.0 + 1e-2 * torch.randn(m, generator=g, device=DEV, dtype=torch.float64), cp=1000.0, kc=1.0, Q=None,
                phase=(_rand(g, m) < 0.05).to(torch.int32), obstacles=spheres)


def _volume(sc):
    r = (sc["dx"][0] * sc["dx"][1] * sc["dx"][2] / 8 / (FOURBYTHREE * PI)) ** (1.0 / 3.0)
    return r, FOURBYTHREE * PI * r ** 3


def _scenes(case, seed):
    """The scenes of a case: one, or a batch's."""
    if case["kind"] != "batch":
        return [_scene(case, seed)]
    sides = [int(round(case["lo"] + (case["hi"] - case["lo"]) * k / 4)) for k in range(5)]
    out = []
    for i, (n, f) in enumerate(scenes.batched_scene_sizes(case["scenes"], tuple(sides), (0.1, 0.4), 2024)):
        sc = _box((n, n, n), (1.0, 1.0, 1.0), case["order"], gravity=(0.0, 0.0, -9.81))
        out.append(_fluid(sc, (2.0 * f, 1.0, 0.5), 0.25, _gen(seed * 1000 + i)))
    return out


# ------------------------------------------------------------------ the program
def _specs(case, sc):
    s = scenes.base_specs((0, 0, 0), sc["size"], sc["n"], sc["order"],
                          nt.PREC_FP64 if case["fp64"] else nt.PREC_MIXED)
    s.alpha_pic_flip, s.cfl = sc["alpha"], sc["cfl"]
    s.stress_update_scheme = 1 if case.get("musl") else 0
    s.autotune = 0  # production runs pin the launch variants: no timing runs in the middle of a job
    if sc["timestep"]:
        s.fixed_timestep, s.timestep = 1, sc["timestep"]
    for d in range(3):
        s.gravity[d], s.periodic[d] = sc["gravity"][d], sc["periodic"][d]
        if sc["periodic"][d]:
            s.bclo[d] = s.bchi[d] = nt.BC_PERIODIC
        else:
            s.bclo[d], s.bchi[d] = sc["slip"][d]
    if sc["heat"]:
        s.use_temp = 1
        if case["kind"] == "block":
            s.bclo_temp[0], s.T_wall_lo[0] = nt.BCT_ISOTHERMAL, 350.0
            s.bchi_temp[0], s.h_hi[0], s.Tinf_hi[0] = nt.BCT_CONVECTION, 20.0, 290.0
            s.bclo_temp[1], s.flux_lo[1] = nt.BCT_USERFLUX, 500.0
            s.bclo_temp[2], s.T_wall_lo[2] = nt.BCT_ISOTHERMAL, 280.0
            s.bchi_temp[2], s.h_hi[2], s.Tinf_hi[2] = nt.BCT_CONVECTION, 5.0, 300.0
    if sc.get("obstacles"):
        s.num_bodies = 1
        s.bodies[0].mom_bc = nt.BC_NOSLIP
    return s


_kept = {}


def _buffers(sizes):
    """The program's page-locked particle arrays, kept from one run to the next of the same sizes."""
    if _kept.get("sizes") != sizes:
        _kept.clear()
        _kept.update(sizes=sizes, parts=[nt.Particles(n, pinned=True) for n in sizes])
    return _kept["parts"]


def _fill(p, sc):
    """A scene's particles into host arrays, in the layout of the reference's particle fields."""
    n = p.n
    r, vol = _volume(sc)
    rd = torch.zeros(nt.EXG_NREAL, n, device=DEV, dtype=torch.float64)
    rd[nt.R_RADIUS] = r
    rd[nt.R_VEL:nt.R_VEL + 3] = sc["vel"]
    for k in (0, 4, 8):
        rd[nt.R_DEFGRAD + k] = 1.0
    rd[nt.R_VOLUME] = rd[nt.R_VOL_INIT] = vol
    rd[nt.R_MASS] = sc["rho0"] * vol
    rd[nt.R_DENSITY] = sc["rho0"]
    rd[nt.R_JACOBIAN] = 1.0
    for f, k in ((nt.R_E, "E"), (nt.R_NU, "nu"), (nt.R_BULK, "K"), (nt.R_GAMMA, "gamma"), (nt.R_VISC, "visc")):
        rd[f] = sc[k]
    if sc["heat"]:
        rd[nt.R_TEMPERATURE], rd[nt.R_SPHEAT], rd[nt.R_THERMCOND] = sc["T"], sc["cp"], sc["kc"]
        if sc["Q"] is not None:
            rd[nt.R_HEATSRC] = sc["Q"]
    ints = torch.zeros(nt.EXG_NINT, n, device=DEV, dtype=torch.int32)
    if sc.get("phase") is not None:
        ints[nt.I_PHASE] = sc["phase"]
    ints[nt.I_RIGID_ID] = -1
    ints[nt.I_MODEL] = sc["model"]
    torch.from_numpy(p.pos).copy_(sc["pos"])
    torch.from_numpy(p.rdata).copy_(rd)
    torch.from_numpy(p.idata).copy_(ints)


def prepare(case, seed):
    scs = _scenes(case, seed)
    parts = _buffers([sc["pos"].shape[1] for sc in scs])
    if case["kind"] == "batch":
        job = nt.Batch([_specs(case, sc) for sc in scs])
        ctxs = job.scenes
    else:
        job = nt.Context(_specs(case, scs[0]))
        ctxs = [job]
    for ctx, p, sc in zip(ctxs, parts, scs):
        _fill(p, sc)
        if sc.get("obstacles"):
            ctx.build_levelset(0, [nt.LsShape.sphere(c, r) for c, r in sc["obstacles"]])
        ctx.upload(p)
        ctx.Initialise_Internal_Forces()
    torch.cuda.empty_cache()
    return dict(case=case, job=job, ctxs=ctxs, parts=parts, time=0.0)


FIELDS = (("vel", nt.R_VEL, 3), ("vel_prime", nt.R_VEL_PRIME, 3), ("strainrate", nt.R_STRAINRATE, 6),
          ("strain", nt.R_STRAIN, 6), ("stress", nt.R_STRESS, 6), ("F", nt.R_DEFGRAD, 9), ("volume", nt.R_VOLUME, 1),
          ("density", nt.R_DENSITY, 1), ("J", nt.R_JACOBIAN, 1), ("pressure", nt.R_PRESSURE, 1))
HEAT = (("T", nt.R_TEMPERATURE, 1), ("heatflux", nt.R_HEATFLUX, 3))


def run(state):
    case, job = state["case"], state["job"]
    if case.get("calls"):
        for _ in range(case["steps"]):
            _step_by_calls(job, state)
    else:
        job.step(case["steps"])
    for ctx, p in zip(state["ctxs"], state["parts"]):
        ctx.download_into(p)
    fields = FIELDS + (HEAT if case["kind"] in ("block", "column") else ())
    rows = [{"pos": p.pos, **{k: p.rdata[a:a + m] for k, a, m in fields}} for p in state["parts"]]
    kept = torch.float64 if case["fp64"] else torch.float32
    if len(rows) == 1 and case["fp64"]:
        return rows[0]
    n = [p.n for p in state["parts"]]
    out = {}
    for k in rows[0]:
        out[k] = torch.empty(rows[0][k].shape[0], sum(n), dtype=kept)
        at = 0
        for r, m in zip(rows, n):
            out[k][:, at:at + m].copy_(torch.from_numpy(r[k]))
            at += m
    return out


def _step_by_calls(ctx, state):
    """One USL step as the reference's main loop writes it."""
    ctx.Redistribute()
    dt = ctx.Calculate_time_step()
    ctx.Reset_Nodaldata_to_Zero()
    ctx.P2G_Momentum(1, 1, 1)
    ctx.backup_current_velocity()
    ctx.Nodal_Time_Update_Momentum(dt)
    ctx.Apply_Nodal_BCs(dt, state["time"])
    ctx.G2P_Momentum(1, 1, dt)
    ctx.Update_MP_Positions(dt)
    ctx.Update_MP_Volume()
    ctx.Calculate_MP_Stress_Strain(state["time"], dt)
    state["time"] += dt


def _counts(case):
    """Particles of a case, without making them all where they are many."""
    if case["kind"] == "spheres":
        return int(2 * 4 / 3 * math.pi * 0.2 ** 3 * 8 * case["n"] ** 3)
    if case["kind"] == "batch":
        sides = tuple(int(round(case["lo"] + (case["hi"] - case["lo"]) * k / 4)) for k in range(5))
        return sum(scenes.batched_scene_particle_counts(case["scenes"], sides, (0.1, 0.4), 2024))
    if case["kind"] == "bar":
        return case["n"] * 128
    n, f = case["nx"] * case["ny"] * case["nz"], {"dam": 0.24, "block": 0.7, "column": 0.125}[case["kind"]]
    return int(8 * f * n)


def work(case):
    """Per step the particles' state read once and written once and the deposit's and the
    gather's multiply-adds (10 and 15 per node of the stencil); at the end the download."""
    n, w = _counts(case), 8 if case["fp64"] else 4
    heat = case["kind"] in ("block", "column")
    # read: x, J and v, strain, F, stress, volumes, mass, pressure; write: also v', strain rate, density
    step = 24 + 8 + w * (3 + 6 + 9 + 6 + 4) + 24 + 8 + w * (6 + 12 + 6 + 9 + 3) + (16 + 8 * w if heat else 0)
    stencil = {1: 8, 2: 27, 3: 64}[case["order"]]
    rows = 3 + sum(m for _, _, m in FIELDS) + (4 if heat else 0)
    return {"bytes": float(n) * (case["steps"] * step + 8 * rows), "flops": float(n) * case["steps"] * stencil * 50}


# ------------------------------------------------------------------ the same in plain FP64
# B-spline pieces by shape type (1 at a wall, 2 and 4 next to one, 3 inside), highest power first
_O6, _O3, _T3, _F3 = 0.16666666666667, 0.333333333333, 0.6666666666667, 1.3333333333
_Z = [0.0] * 4
_CUB = [[_Z] * 4,
        [[_O6, 1, 2, _F3], [-_O6, 0, 1, 1], [_O6, 0, -1, 1], [-_O6, 1, -2, _F3]],
        [_Z, [-_O3, -1, 0, _T3], [0.5, -1, 0, _T3], [-_O6, 1, -2, _F3]],
        [[_O6, 1, 2, _F3], [-0.5, -1, 0, _T3], [0.5, -1, 0, _T3], [-_O6, 1, -2, _F3]],
        [[_O6, 1, 2, _F3], [-0.5, -1, 0, _T3], [_O3, -1, 0, _T3], _Z]]
_QUAD = [[_Z] * 5,
         [[0, _T3, 2, 1.5], [0, -_F3, 0, 1], [0, -_F3, 0, 1], [0, _T3, -2, 1.5], _Z],
         [[0, 4 / 3, 8 / 3, 4 / 3], [0, -7 / 6, 1 / 6, 17 / 24], [0, 0.5, -1.5, 1.125], _Z, _Z],
         [[0, 0.5, 1.5, 1.125], [0, -1, 0, 0.75], [0, 0.5, -1.5, 1.125], _Z, _Z],
         [[0, 0.5, 1.5, 1.125], [0, -7 / 6, -1 / 6, 17 / 24], [0, 4 / 3, -8 / 3, 4 / 3], _Z, _Z]]
_QMAP = [[4] * 6, [0, 0, 1, 2, 3, 3], [0, 1, 1, 2, 2, 4], [0, 0, 1, 1, 2, 2], [0, 0, 1, 1, 2, 4]]  # 4: outside


def _axis(sc, x, d):
    """Weights, derivatives and nodes of one axis: [n, W] each."""
    order, nc, dx, per = sc["order"], sc["n"][d], sc["dx"][d], sc["periodic"][d]
    cell = torch.floor(x / dx).long()
    off = torch.arange(2, device=DEV) if order == 1 else torch.arange(-1, 3, device=DEV)
    node = cell[:, None] + off
    z = x[:, None] / dx - node
    if order == 1:
        w = torch.where(off == 0, 1 - z, z + 1)
        dw = torch.where(off == 0, -1.0, 1.0).double().expand_as(w) / dx
    else:
        ty = torch.full_like(node, 3)
        if not per:
            ty = torch.where((node == 0) | (node == nc), 1, ty)
            ty = torch.where(node == 1, 2, ty)
            ty = torch.where(node == nc - 1, 4, ty)
        if order == 3:
            c = torch.tensor(_CUB, device=DEV, dtype=torch.float64)[ty, (torch.floor(z).long() + 2).clamp(0, 3)]
        else:
            raw = torch.floor((z + torch.where(ty == 2, 1.0, 1.5)) * 2).long()
            q = torch.tensor(_QMAP, device=DEV)[ty, raw.clamp(0, 5)]
            q = torch.where((raw < 0) | (raw > 5), 4, q)
            c = torch.tensor(_QUAD, device=DEV, dtype=torch.float64)[ty.where(q < 4, torch.zeros_like(ty)), q]
        w = ((c[..., 0] * z + c[..., 1]) * z + c[..., 2]) * z + c[..., 3]
        dw = ((3 * c[..., 0] * z + 2 * c[..., 1]) * z + c[..., 2]) / dx
    if per:
        node = torch.remainder(node, nc)
    else:
        inside = (node >= 0) & (node <= nc)
        w, dw, node = w * inside, dw * inside, node.clamp(0, nc)
    return w, dw, node


def _rows(sc, ax):
    """For each (z, y) of the stencil the nodes of an x row and N, dN/dx, dN/dy, dN/dz there."""
    (wx, dx, ix), (wy, dy, iy), (wz, dz, iz) = ax
    nx, ny = sc["n"][0] + 1, sc["n"][1] + 1
    for k in range(wz.shape[1]):
        for j in range(wy.shape[1]):
            idx = (iz[:, k:k + 1] * ny + iy[:, j:j + 1]) * nx + ix
            yz, dyz, ydz = wy[:, j:j + 1] * wz[:, k:k + 1], dy[:, j:j + 1] * wz[:, k:k + 1], wy[:, j:j + 1] * dz[:, k:k + 1]
            yield idx, wx * yz, dx * yz, wx * dyz, wx * ydz


_SYM = ((0, 1, 2), (1, 3, 4), (2, 4, 5))  # packed XX XY XZ YY YZ ZZ


def _deposit(sc, q, ax, force):
    nodes = (sc["n"][0] + 1) * (sc["n"][1] + 1) * (sc["n"][2] + 1)
    grid = torch.zeros(nodes, 7, device=DEV, dtype=torch.float64)
    mv = q["m"] * q["v"]
    for idx, N, gx, gy, gz in _rows(sc, ax):
        ch = [q["m"] * N] + [mv[d][:, None] * N for d in range(3)]
        for d in range(3):
            if force:
                s = [-(q["vol"] * q["sig"][_SYM[d][e]])[:, None] for e in range(3)]
                ch.append(s[0] * gx + s[1] * gy + s[2] * gz + (q["m"] * sc["gravity"][d]) * N)
            else:
                ch.append(torch.zeros_like(N))
        grid.index_add_(0, idx.reshape(-1), torch.stack(ch, -1).reshape(-1, 7))
    return grid


def _node_walls(sc, v):
    """Slip or no-slip walls of the nodal velocities [nz, ny, nx, 3]; on an edge the last direction decides."""
    v0 = v.clone()
    for d in range(3):
        if sc["periodic"][d]:
            continue
        for side in range(2):
            at = [slice(None)] * 3
            at[2 - d] = -1 if side else 0
            u = v0[tuple(at)].clone()
            if sc["slip"][d][side] == 1:
                u.zero_()
            else:
                u[..., d] = 0.0
            v[tuple(at)] = u
    return v


def _gather(sc, ax, grid, want):
    n = ax[0][0].shape[0]
    val = torch.zeros(n, grid.shape[1], device=DEV, dtype=torch.float64)
    grad = torch.zeros(n, 3, 3, device=DEV, dtype=torch.float64)
    for idx, N, gx, gy, gz in _rows(sc, ax):
        u = grid[idx]
        val += (u * N[..., None]).sum(1)
        if want:
            for e, g in enumerate((gx, gy, gz)):
                grad[:, :, e] += (u[..., :3] * g[..., None]).sum(1)
    return val, grad


def _stress(sc, q):
    if sc["model"] == 0:
        E, nu, e = sc["E"], sc["nu"], q["eps"]
        c1, c2 = E / (1 + nu) / (1 - 2 * nu), E / (1 + nu)
        q["sig"] = torch.stack([c1 * ((1 - nu) * e[0] + nu * (e[3] + e[5])), c2 * e[1], c2 * e[2],
                                c1 * ((1 - nu) * e[3] + nu * (e[0] + e[5])), c2 * e[4],
                                c1 * ((1 - nu) * e[5] + nu * (e[0] + e[3]))])
    else:
        q["p"] = sc["K"] * ((1 / q["J"]) ** sc["gamma"] - 1)
        tr = (q["sr"][0] + q["sr"][3] + q["sr"][5]) / 3
        q["sig"] = 2 * sc["visc"] * q["sr"]
        for k in (0, 3, 5):
            q["sig"][k] += -2 * sc["visc"] * tr - q["p"]


def _strainrate(L):
    return torch.stack([0.5 * (L[:, a, b] + L[:, b, a]) for a in range(3) for b in range(a, 3)])


def _normalised(grid):
    m = grid[:, :1]
    return torch.where(m >= 1e-18, grid[:, 1:4] / m.clamp_min(1e-300), torch.zeros_like(grid[:, 1:4]))


def _exact_step(sc, q, musl):
    shape = (sc["n"][2] + 1, sc["n"][1] + 1, sc["n"][0] + 1, 3)
    if sc["timestep"]:
        dt = sc["timestep"]
    else:
        mod = sc["K"] if sc["model"] else sc["E"] * (1 - sc["nu"]) / ((1 + sc["nu"]) * (1 - 2 * sc["nu"]))
        speed = torch.sqrt(mod / q["rho"]) + torch.sqrt((q["v"] ** 2).sum(0))
        dt = min(max(sc["cfl"] * min(sc["dx"]) / float(speed.max()), 1e-12), 1.0)
    ax = [_axis(sc, q["x"][d], d) for d in range(3)]
    grid = _deposit(sc, q, ax, True)
    m = grid[:, :1]
    old = _normalised(grid)
    new = torch.where(m >= 1e-18, old + grid[:, 4:] / m.clamp_min(1e-300) * dt, torch.zeros_like(old))
    new = _node_walls(sc, new.reshape(shape)).reshape(-1, 3)
    delta = torch.where(m > 0, new - old, torch.zeros_like(old))
    val, L = _gather(sc, ax, torch.cat([new, delta], 1), not musl)
    a = sc["alpha"]
    q["vp"] = val[:, :3].T.contiguous()
    q["v"] = a * q["v"] + a * val[:, 3:].T + (1 - a) * q["vp"]
    if musl:
        new = _node_walls(sc, _normalised(_deposit(sc, q, ax, False)).reshape(shape)).reshape(-1, 3)
        _, L = _gather(sc, ax, new, True)
    F = q["F"].T.reshape(-1, 3, 3)
    F = F + dt * (L @ F)
    q["F"] = F.reshape(-1, 9).T.contiguous()
    q["sr"] = _strainrate(L)
    q["x"] = q["x"] + dt * q["vp"]
    rin = q["v"].clone()
    for d in range(3):
        if sc["periodic"][d]:
            q["x"][d] = torch.remainder(q["x"][d], sc["size"][d])
            continue
        for side, out in ((0, q["x"][d] < 0), (1, q["x"][d] > sc["size"][d])):
            q["x"][d] = torch.where(out, 2 * side * sc["size"][d] - q["x"][d], q["x"][d])
            for e in range(3):
                hit = 0.0 if e == d or sc["slip"][d][side] == 1 else rin[e]
                q["v"][e] = torch.where(out, hit, q["v"][e])
    q["J"] = torch.linalg.det(F)
    q["vol"] = q["vol0"] * q["J"]
    q["rho"] = q["m"] / q["vol"]
    q["eps"] = q["eps"] + dt * q["sr"]
    _stress(sc, q)


def exact(case, seed):
    """The pass in FP64 with torch alone.  The two heated scenes and the two largest have no such value here
    (thermal sweeps and obstacles; minutes of scatter-adds)."""
    if case["kind"] in ("block", "column") or _counts(case) * case["steps"] * (64 if case["order"] > 1 else 8) > 1.1e10:
        return None
    outs = []
    for sc in _scenes(case, seed):
        n = sc["pos"].shape[1]
        _, vol = _volume(sc)
        eye = torch.eye(3, device=DEV, dtype=torch.float64).reshape(9, 1).expand(9, n).contiguous()
        zero = lambda k: torch.zeros(k, n, device=DEV, dtype=torch.float64)  # noqa: E731
        q = dict(x=sc["pos"].clone(), v=sc["vel"].clone(), vp=zero(3), eps=zero(6), sig=zero(6), F=eye, p=zero(1)[0],
                 J=torch.ones(n, device=DEV, dtype=torch.float64), vol0=vol, m=sc["rho0"] * vol)
        q["vol"], q["rho"] = vol * q["J"], sc["rho0"] * q["J"]
        ax = [_axis(sc, q["x"][d], d) for d in range(3)]
        _, L = _gather(sc, ax, _normalised(_deposit(sc, q, ax, False)), True)
        q["sr"] = _strainrate(L)
        _stress(sc, q)
        for _ in range(case["steps"]):
            _exact_step(sc, q, bool(case.get("musl")))
        outs.append({"pos": q["x"], "vel": q["v"], "vel_prime": q["vp"], "strainrate": q["sr"], "strain": q["eps"],
                     "stress": q["sig"], "F": q["F"], "volume": q["vol"][None], "density": q["rho"][None], "J": q["J"][None],
                     "pressure": q["p"][None]})
    return {k: torch.cat([o[k] for o in outs], 1) for k in outs[0]}
