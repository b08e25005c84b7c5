"""The row-walking P2G at the sizes where its walk and its work split can go
wrong: one particle per row, rows of more particles than are staged at once,
crowded cells, empty cells between occupied ones, tiles of edge 4 and 8,
and few enough particles that tiles are split into items of
one plane.  Nodal mass, velocity and force against the FP64 oracle: FP64 within
1e-10 of the field's max norm (the suite's tolerance for an exact fixed-point
sum of FP64 terms), mixed within 2e-6: each node sums at most a few hundred
FP32 terms, each of relative rounding 6e-8 or less, and the terms of a force
component do not exceed its max norm by more than a small factor."""
import numpy as np
import pytest

from exagoop_b200 import native as nt, scenes
import orc

pytestmark = pytest.mark.gpu


def particles(kind, n, dx, rng):
    """Positions of one distribution in the unit cells of an n^3 grid."""
    if kind == "sparse":      # one particle in every fifth cell
        c = np.stack(np.meshgrid(*[np.arange(2, n - 2)] * 3, indexing="ij")).reshape(3, -1)[:, ::5]
        pos = c + rng.uniform(0.05, 0.95, c.shape)
    elif kind == "crowded":   # one row with 70 particles in one cell, 33 in the next but one
        pos = np.concatenate([rng.uniform(0.05, 0.95, (3, 70)) + np.array([[3], [4], [5]]),
                              rng.uniform(0.05, 0.95, (3, 33)) + np.array([[5], [4], [5]]),
                              rng.uniform(0.05, 0.95, (3, 1)) + np.array([[7], [4], [5]])], axis=1)
    else:                     # everywhere, faces included: about 3 a cell
        pos = rng.uniform(0.0, n, (3, 3 * n ** 3))
    return np.ascontiguousarray(pos) * dx


@pytest.mark.parametrize("precision", [nt.PREC_FP64, nt.PREC_MIXED])
@pytest.mark.parametrize("order", [1, 2, 3])
@pytest.mark.parametrize("tile", [4, 8])
@pytest.mark.parametrize("kind", ["sparse", "crowded", "filled"])
def test_p2g_rows(kind, tile, order, precision):
    n = 13
    dx = 1.0 / n
    rng = np.random.default_rng(17 * order + tile)
    s = scenes.base_specs((0, 0, 0), (1, 1, 1), (n, n, n), order, precision)
    s.gravity[2] = -9.81
    s.tile = tile
    s.autotune = 0
    p = scenes.make_particles(particles(kind, n, dx, rng), (dx,) * 3, (2, 2, 2), 1000.0, 0, E=1e3, nu=0.3)
    p.rdata[nt.R_VEL:nt.R_VEL + 3] = rng.normal(0, 1, (3, p.n))
    p.rdata[nt.R_STRESS:nt.R_STRESS + 6] = rng.normal(0, 1e3, (6, p.n))
    p.idata[nt.I_PHASE, ::11] = 1
    ctx = nt.Context(s)
    ctx.upload(p)
    ctx.P2G_Momentum(1, 1, 1)
    o = orc.Oracle(s)
    o.upload(p)
    o.p2g_momentum(1, 1, 1)
    tol = 1e-10 if precision == nt.PREC_FP64 else 2e-6
    m = o.nodes(nt.N_MASS)
    heavy = m >= 1e-6 * m.max()
    for comp in [nt.N_MASS] + [nt.N_VEL + d for d in range(3)] + [nt.N_FRC + d for d in range(3)]:
        a, b = ctx.nodes(comp), o.nodes(comp)
        if nt.N_VEL <= comp < nt.N_FRC:  # momenta everywhere, velocities where the node is not light
            assert np.abs((a - b) * m).max() <= tol * max(np.abs(b * m).max(), 1e-300), comp
            a, b = a[heavy], b[heavy]
            tol_c = tol * 10 if precision == nt.PREC_MIXED else tol
        else:
            tol_c = tol
        assert np.abs(a - b).max() <= tol_c * max(np.abs(b).max(), 1e-300), comp
    ctx.close()


def test_pile_up_in_one_row():
    """Four million particles in one cell beside a particle in every tile: the
    warp that walks the row takes longer than the bound on the other warps'
    waits for its buffer, which counts only while nothing moves.  The nodal
    sums are the particles' (an interior cubic stencil sums to 1): relative
    1e-9, above the rounding of an FP64 sum of four million terms."""
    n, big = 64, 4_000_000
    rng = np.random.default_rng(5)
    cells = np.stack(np.meshgrid(*[np.arange(4, n, 8)] * 3, indexing="ij")).reshape(3, -1)
    pos = np.concatenate([np.array([[20], [28], [36]]) + rng.uniform(0.01, 0.99, (3, big)), cells + 0.5], axis=1) / n
    s = scenes.base_specs((0, 0, 0), (1, 1, 1), (n, n, n), 3, nt.PREC_FP64)
    s.gravity[2] = -9.81
    s.autotune = 0
    p = scenes.make_particles(pos, (1.0 / n,) * 3, (2, 2, 2), 1000.0, 0, E=1e3, nu=0.3)
    p.rdata[nt.R_VEL] = 0.25
    ctx = nt.Context(s)
    ctx.upload(p)
    ctx.P2G_Momentum(1, 1, 1)
    m, total = ctx.nodes(nt.N_MASS), p.rdata[nt.R_MASS].sum()
    assert abs(m.sum() / total - 1.0) < 1e-9
    assert abs((m * ctx.nodes(nt.N_VEL)).sum() / (0.25 * total) - 1.0) < 1e-9
    assert abs(ctx.nodes(nt.N_FRC + 2).sum() / (-9.81 * total) - 1.0) < 1e-9
    ctx.close()
