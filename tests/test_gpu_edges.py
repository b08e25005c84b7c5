"""Edge cases of the step path through the C ABI: an empty particle set, a
single particle, particles exactly on nodes, cell faces, tile faces and the
lower domain faces (binning ties and the ends of the B-spline supports), and
a particle count above the 32-bit index range.  Parity against the FP64
oracle at the tolerance of the other parity tests; binning bit-exact."""
import numpy as np
import pytest

from exagoop_b200 import native as nt, scenes
import orc
import parity

pytestmark = pytest.mark.gpu

TOL64 = 1e-10
FIELDS = [("vel", nt.R_VEL, 3), ("vel_prime", nt.R_VEL_PRIME, 3), ("strainrate", nt.R_STRAINRATE, 6),
          ("strain", nt.R_STRAIN, 6), ("stress", nt.R_STRESS, 6), ("defgrad", nt.R_DEFGRAD, 9),
          ("volume", nt.R_VOLUME, 1), ("density", nt.R_DENSITY, 1), ("jacobian", nt.R_JACOBIAN, 1),
          ("pressure", nt.R_PRESSURE, 1)]


def check(g, r, tol=TOL64):
    for name, e in parity.field_errors(g, r, FIELDS).items():
        assert e < tol, f"{name}: max rel err {e:.3e}"
    e = np.abs(g.pos - r.pos).max()
    assert e < tol * max(1.0, np.abs(r.pos).max()), f"position: max abs err {e:.3e}"


def unit_box(order, n=16):
    # dx = 1/16: node, face and tile coordinates are exact binary fractions
    s = scenes.base_specs((0.0, 0.0, 0.0), (1.0, 1.0, 1.0), (n, n, n), order)
    s.gravity[2] = -2.0
    return s, [1.0 / n] * 3


def elastic(pos, dx, seed, speed=0.2):
    # Initialise_Internal_Forces sets the stress from the strain, so the
    # particles carry a strain (a lone particle with none translates
    # rigidly and its strain rate is rounding noise about zero)
    rng = np.random.default_rng(seed)
    p = scenes.make_particles(pos, dx, (2, 2, 2), 1000.0, 0, E=5e3, nu=0.3)
    n = pos.shape[1]
    p.rdata[nt.R_VEL:nt.R_VEL + 3] = rng.normal(0, speed, (3, n))
    p.rdata[nt.R_STRAIN:nt.R_STRAIN + 6] = rng.normal(0, 1e-3, (6, n))
    return p


def run_both(s, p, nsteps):
    ctx = nt.Context(s)
    ctx.upload(p)
    o = orc.Oracle(s)
    o.upload(p)
    ctx.Initialise_Internal_Forces()
    o.init_internal_forces()
    ctx.step(nsteps)
    assert o.step(nsteps) == 0
    g, r = ctx.download(), o.download()
    ctx.close()
    return g, r


def test_empty_particle_set_is_not_ready_and_recovers():
    s, dx = unit_box(2)
    ctx = nt.Context(s)
    ctx.upload(nt.Particles(0))
    for call in (lambda: ctx.step(1), lambda: ctx.P2G_Momentum(1, 1, 1)):
        with pytest.raises(nt.ExgError) as e:
            call()
        assert e.value.code == -11  # EXG_ERR_NOT_READY
    # the reference's minimum over no particles is the largest double, so
    # its dt is CFL x that clamped to dt_max_limit
    assert ctx.Calculate_time_step() == s.dt_max_limit
    assert ctx.download().n == 0
    # the context stays usable: a later upload steps as a fresh context does
    pos = np.random.default_rng(4).uniform(0.3, 0.7, (3, 500))
    p = elastic(pos, dx, 4)
    ctx.upload(p)
    ctx.Initialise_Internal_Forces()
    ctx.step(5)
    fresh = nt.Context(s)
    fresh.upload(p)
    fresh.Initialise_Internal_Forces()
    fresh.step(5)
    a, b = ctx.download(), fresh.download()
    assert np.array_equal(a.pos, b.pos) and np.array_equal(a.rdata, b.rdata)
    ctx.close()
    fresh.close()


@pytest.mark.parametrize("order", [1, 2, 3])
def test_single_particle(order):
    s, dx = unit_box(order)
    p = elastic(np.array([[0.4137], [0.5521], [0.2906]]), dx, 7)
    g, r = run_both(s, p, 20)
    check(g, r)


@pytest.mark.parametrize("order", [1, 2, 3])
def test_particles_on_nodes_faces_and_tile_faces(order):
    # every coordinate from {k dx, (k + 1/2) dx}: nodes and cell faces (the
    # cubic and linear bins' edges), cell centres (the quadratic nearest-node
    # ties), the tile faces at 8 dx and the lower domain faces at 0
    s, dx = unit_box(order)
    ks = np.arange(0, 32) / 32.0
    g3 = np.stack(np.meshgrid(ks, ks, ks, indexing="ij")).reshape(3, -1)
    rng = np.random.default_rng(11)
    pos = g3[:, rng.choice(g3.shape[1], 6000, replace=False)]
    p = elastic(pos, dx, 11, speed=0.02)
    ctx = nt.Context(s)
    ctx.upload(p)
    o = orc.Oracle(s)
    o.upload(p)
    keys, perm = ctx.sort_keys()
    okeys, operm = o.sort_keys(ctx.tile())
    assert np.array_equal(keys, okeys) and np.array_equal(perm, operm)
    ctx.close()
    # linear basis: a particle on node i weighs node i + 1 by 0 but with a
    # full gradient, the reference's cell-crossing instability; on this
    # sparse lattice J turns negative by the second step in the oracle
    # too, so the linear case is compared after the step that starts from
    # the exact positions
    g, r = run_both(s, p, 1 if order == 1 else 10)
    check(g, r)


def test_particle_count_above_int32_is_rejected():
    # refused before any array is read, so the pointers may be null
    s, _ = unit_box(2)
    ctx = nt.Context(s)
    soa = nt.ParticleSoA(1 << 31, None, None, None)
    rc = ctx.L.exg_particles_upload(ctx.h, nt.C.byref(soa))
    assert rc == -8  # EXG_ERR_ARG
    assert b"2^31" in ctx.L.exg_last_error(ctx.h)
    ctx.close()


def rel_l2(g, r):
    out = {}
    for name, f, k in [("vel", nt.R_VEL, 3), ("stress", nt.R_STRESS, 6), ("jacobian", nt.R_JACOBIAN, 1)]:
        a, b = g.rdata[f:f + k], r.rdata[f:f + k]
        out[name] = np.linalg.norm(a - b) / np.linalg.norm(b)
    return out


@pytest.mark.parametrize("order", [1, 2, 3])
def test_mixed_precision_edges(order):
    # the same single particle and lattice through the FP32 kernels (mixed
    # state): binning bit-exact (positions stay FP64), velocity and stress
    # within 1e-4 relative L2 of the FP64 oracle, J within 1e-6
    s, dx = unit_box(order)
    s.precision = nt.PREC_MIXED
    s64 = s.copy()
    s64.precision = nt.PREC_FP64
    ks = np.arange(0, 32) / 32.0
    g3 = np.stack(np.meshgrid(ks, ks, ks, indexing="ij")).reshape(3, -1)
    rng = np.random.default_rng(12)
    cases = [(elastic(np.array([[0.4137], [0.5521], [0.2906]]), dx, 7), 20),
             (elastic(g3[:, rng.choice(g3.shape[1], 6000, replace=False)], dx, 12, speed=0.02),
              1 if order == 1 else 10)]
    for p, nsteps in cases:
        ctx = nt.Context(s)
        ctx.upload(p)
        o = orc.Oracle(s64)
        o.upload(p)
        keys, perm = ctx.sort_keys()
        okeys, operm = o.sort_keys(ctx.tile())
        assert np.array_equal(keys, okeys) and np.array_equal(perm, operm)
        ctx.Initialise_Internal_Forces()
        o.init_internal_forces()
        ctx.step(nsteps)
        assert o.step(nsteps) == 0
        e = rel_l2(ctx.download(), o.download())
        ctx.close()
        assert e["vel"] < 1e-4 and e["stress"] < 1e-4 and e["jacobian"] < 1e-6, (p.n, e)


# More step paths from the same lattice start (coordinates k dx / 2): a
# periodic axis with particles on its face (the wrap of bins and nodes),
# per-axis orders (the non-factorized P2G and the generic G2P window), and
# the thermal path (temperature deposit, thermal G2P, heat flux)
LATTICE_PATHS = {
    "periodic_x": dict(order=2, periodic=0),
    "orders_2_3_3": dict(order=(2, 3, 3)),
    "thermal": dict(order=2, thermal=True),
    "neo_hookean": dict(order=3, model=2),
    "tait_fluid": dict(order=2, model=1),
    "musl": dict(order=3, musl=True),
    "partial_slip_moving_walls": dict(order=2, walls=True),
}


def lattice_scene(order=2, periodic=None, thermal=False, model=0, musl=False, walls=False, seed=21):
    s, dx = unit_box(order if isinstance(order, int) else 2)
    if musl:
        s.stress_update_scheme = 1
    if walls:
        for d in range(3):
            s.bclo[d] = s.bchi[d] = nt.BC_PARTIALSLIP
            s.wall_mu_lo[d] = s.wall_mu_hi[d] = 0.3
            s.wall_vel_lo[3 * d + (d + 1) % 3] = 0.05
    if not isinstance(order, int):
        for d in range(3):
            s.order[d] = order[d]
    if periodic is not None:
        # a periodic axis needs three tiles: twice the length at the same dx
        s.phi[periodic], s.ncells[periodic] = 2.0, 32
        s.periodic[periodic] = 1
        s.bclo[periodic] = s.bchi[periodic] = nt.BC_PERIODIC
    # with friction walls, particles on a face that move outwards leave the
    # domain in the reference as here (EXG_ERR_DOMAIN): keep off the faces
    ks = np.arange(1 if walls else 0, 31 if walls else 32) / 32.0
    g3 = np.stack(np.meshgrid(ks, ks, ks, indexing="ij")).reshape(3, -1)
    rng = np.random.default_rng(seed)
    pos = g3[:, rng.choice(g3.shape[1], 6000, replace=False)]
    if model == 0:
        p = elastic(pos, dx, seed, speed=0.02)
    else:
        # neo-Hookean solid (model 2) or Tait fluid (model 1: K, gamma 7,
        # viscosity), with the same velocities
        p = (scenes.make_particles(pos, dx, (2, 2, 2), 1000.0, 2, E=5e3, nu=0.3) if model == 2 else
             scenes.make_particles(pos, dx, (2, 2, 2), 1000.0, 1, K=2e3, gamma=7.0, visc=1e-3))
        p.rdata[nt.R_VEL:nt.R_VEL + 3] = np.random.default_rng(seed).normal(0, 0.02, (3, p.n))
        if model == 2:
            p.rdata[nt.R_STRAIN:nt.R_STRAIN + 6] = np.random.default_rng(seed + 1).normal(0, 1e-3, (6, p.n))
    if thermal:
        s.use_temp = 1
        for d in range(3):
            s.bclo_temp[d] = s.bchi_temp[d] = nt.BCT_ADIABATIC
        p.rdata[nt.R_TEMPERATURE] = 300.0 + rng.uniform(-20.0, 20.0, p.n)
        p.rdata[nt.R_SPHEAT] = 900.0
        p.rdata[nt.R_THERMCOND] = 50.0
        p.rdata[nt.R_HEATSRC] = 1e5 * (1.0 + rng.uniform(-0.5, 0.5, p.n))
    return s, p


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("case", list(LATTICE_PATHS))
def test_lattice_start_paths(case, precision):
    s, p = lattice_scene(**LATTICE_PATHS[case])
    s64 = s.copy()
    if precision == "mixed":
        s.precision = nt.PREC_MIXED
    ctx = nt.Context(s)
    ctx.upload(p)
    o = orc.Oracle(s64)
    o.upload(p)
    ctx.Initialise_Internal_Forces()
    o.init_internal_forces()
    ctx.step(10)
    assert o.step(10) == 0
    g, r = ctx.download(), o.download()
    ctx.close()
    if precision == "fp64":
        check(g, r)
    else:
        e = rel_l2(g, r)
        assert e["vel"] < 1e-4 and e["stress"] < 1e-4 and e["jacobian"] < 1e-6, e
    if s.use_temp:
        T = r.rdata[nt.R_TEMPERATURE]
        eT = np.linalg.norm(g.rdata[nt.R_TEMPERATURE] - T) / np.linalg.norm(T)
        assert eT < (1e-12 if precision == "fp64" else 1e-5), eT


def test_no_memory_for_the_staging_array(monkeypatch):
    # the P2G's staging array grows with the upload; where its memory is not
    # to be had (here: a limit between what 2 and 6000 particles need), the
    # calls that would use it report that, and a later upload recovers
    s, dx = unit_box(3)
    rng = np.random.default_rng(3)
    few, many = (elastic(rng.uniform(0.1, 0.9, (3, n)), dx, 3) for n in (2, 6000))
    monkeypatch.setenv("EXG_P2G_STAGING_MAX", str(1 << 20))
    ctx = nt.Context(s)
    ctx.upload(few)
    ctx.Initialise_Internal_Forces()
    ctx.step(4)  # two of them replayed from graphs
    with pytest.raises(nt.ExgError, match="staging"):
        ctx.upload(many)
    for call in (lambda: ctx.step(1), lambda: ctx.P2G_Momentum(1, 1, 1), lambda: ctx.autotune()):
        with pytest.raises(nt.ExgError, match="staging"):
            call()
    ctx.upload(few)
    ctx.Initialise_Internal_Forces()
    ctx.step(4)
    fresh = nt.Context(s)
    fresh.upload(few)
    fresh.Initialise_Internal_Forces()
    fresh.step(4)
    a, b = ctx.download(), fresh.download()
    assert np.array_equal(a.pos, b.pos) and np.array_equal(a.rdata, b.rdata)
    ctx.close()
    fresh.close()


@pytest.mark.parametrize("precision", [nt.PREC_FP64, nt.PREC_MIXED])
@pytest.mark.parametrize("case", ["cubic", "quadratic", "thermal"])
def test_least_staging(case, precision, monkeypatch):
    # where the staging of split tiles does not fit, tiles stay whole and
    # their staging is as large as the node blocks themselves: n values of 8
    # (FP64 12) bytes; every split gives the same bits
    s, p = lattice_scene(order=2 if case == "quadratic" else 3, thermal=case == "thermal")
    s.precision = precision
    s.autotune = 0
    edge = 8 + (2 if case == "quadratic" else 3)
    values = -(-(11 if case == "thermal" else 7) * edge ** 3 // 4) * 4
    tiles = 3 ** 3
    out = []
    for limit in (None, tiles * values * (12 if precision == nt.PREC_FP64 else 8)):
        if limit is not None:
            monkeypatch.setenv("EXG_P2G_STAGING_MAX", str(limit))
        ctx = nt.Context(s)
        ctx.upload(p)
        ctx.Initialise_Internal_Forces()
        ctx.step(5)
        out.append(ctx.download())
        ctx.P2G_Momentum(1, 1, 1)
        out.append([ctx.nodes(c) for c in (nt.N_MASS, nt.N_VEL, nt.N_VEL + 1, nt.N_FRC, nt.N_FRC + 2)])
        ctx.close()
    assert np.array_equal(out[0].pos, out[2].pos) and np.array_equal(out[0].rdata, out[2].rdata)
    assert np.array_equal(out[1], out[3])


def test_least_staging_in_a_batch(monkeypatch):
    # a scene without memory for the common split takes the whole batch to the
    # least one
    items = [lattice_scene(order=3, seed=k) for k in (1, 2)]
    items = [(s, elastic(p.pos[:, :n], (1 / 16.,) * 3, 5, speed=0.02)) for (s, p), n in zip(items, (6000, 40))]
    values = -(-7 * 11 ** 3 // 4) * 4
    ref = []
    for s, p in items:
        ctx = nt.Context(s)
        ctx.upload(p)
        ctx.Initialise_Internal_Forces()
        ctx.step(5)
        ref.append(ctx.download())
        ctx.close()
    monkeypatch.setenv("EXG_P2G_STAGING_MAX", str(27 * values * 12))
    b = nt.Batch([s for s, _ in items])
    for sc, (_, p) in zip(b.scenes, items):
        sc.upload(p)
        sc.Initialise_Internal_Forces()
    b.step(2)
    b.step(3)
    for sc, r in zip(b.scenes, ref):
        g = sc.download()
        assert np.array_equal(g.pos, r.pos) and np.array_equal(g.rdata, r.rdata)
    b.close()
