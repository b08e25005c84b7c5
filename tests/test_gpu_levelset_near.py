"""Particles look at the level-set bodies only near them: fields whose negative
nodes are a sphere, lone nodes, or corners of the domain, among positive values
of a grid spacing, of nearly nothing and of very much, with and without a
periodic axis.  One step against the FP64 oracle within 1e-10 of each field's max
norm (the suite's tolerance); particles are placed at random, so that one is within rounding of a
zero of the sampled field with a probability below 1e-10."""
import numpy as np
import pytest

from exagoop_b200 import native as nt, scenes
import orc

pytestmark = pytest.mark.gpu


def field(kind, n, rng):
    k, j, i = np.meshgrid(*[np.arange(n + 1)] * 3, indexing="ij")
    dx = 1.0 / n
    if kind == "sphere":
        return (np.sqrt((i - 0.4 * n) ** 2 + (j - 0.5 * n) ** 2 + (k - 0.6 * n) ** 2) - 2.3) * dx
    phi = np.full(i.shape, 0.7 * dx)
    if kind == "corners":
        phi[[0, 0, -1, -1], [0, -1, 0, -1], [0, -1, -1, 0]] = -2.0 * dx
        return phi
    phi[rng.random(phi.shape) < 0.02] = -3.0 * dx
    phi[rng.random(phi.shape) < 0.05] = 1e-9 * dx
    phi[rng.random(phi.shape) < 0.02] = 1e7 * dx
    return phi


@pytest.mark.parametrize("periodic", [0, 1])
@pytest.mark.parametrize("kind", ["sphere", "nodes", "corners"])
def test_levelset_near(kind, periodic):
    n = 12
    dx = 1.0 / n
    rng = np.random.default_rng(5 + periodic)
    s = scenes.base_specs((0, 0, 0), (1, 1, 1), (n, n, n), 2, nt.PREC_FP64)
    s.num_bodies = 1
    s.bodies[0].mom_bc = nt.BC_SLIP
    s.autotune = 0
    phi = field(kind, n, rng)
    if periodic:
        s.periodic[1], s.tile = 1, 4
        s.bclo[1] = s.bchi[1] = nt.BC_PERIODIC
        phi[:, -1] = phi[:, 0]
    phi = np.ascontiguousarray(phi).ravel()
    p = scenes.make_particles(rng.uniform(0.02, 0.98, (3, 6 * n ** 3)), (dx,) * 3, (2, 2, 2), 1000.0, 0, E=1e3, nu=0.3)
    p.rdata[nt.R_VEL:nt.R_VEL + 3] = rng.normal(0, 1, (3, p.n))
    ctx, o = nt.Context(s), orc.Oracle(s)
    for c in (ctx, o):
        c.upload(p)
        c.set_levelset(0, phi)
    ctx.Initialise_Internal_Forces()
    o.init_internal_forces()
    ctx.step(1)
    assert o.step(1) == 0
    g, r = ctx.download(), o.download()
    for f, k in [(nt.R_VEL, 3), (nt.R_STRESS, 6), (nt.R_DEFGRAD, 9)]:
        a, b = g.rdata[f:f + k], r.rdata[f:f + k]
        assert np.abs(a - b).max() <= 1e-10 * np.abs(b).max(), f
    assert np.abs(g.pos - r.pos).max() <= 1e-10
