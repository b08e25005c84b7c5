"""The P2G at every split of a tile into items: whole, halves, quarters (single
planes are what the small grids of the other tests get).  The split follows the
particle count: n / (8 T^3) tiles are halved until they are 444 items; FP64
cubic with tile 8 never takes whole ones, whose two node blocks do not fit.
Nodal sums against the FP64 oracle: FP64 within 1e-10 of the field's max norm
(exact fixed-point sums of FP64 terms), mixed within 2e-6 (a few hundred FP32
terms a node, each of relative rounding 6e-8 or less)."""
import numpy as np
import pytest

from exagoop_b200 import native as nt, scenes
import orc

pytestmark = pytest.mark.gpu

# tile, particles, orders: whole, halves, quarters; whole, halves (with temperature)
SPLITS = [(8, 1_850_000, (2, 3)), (8, 1_000_000, (2, 3)), (8, 500_000, (1, 3)),
          (4, 240_000, (1, 2, 3)), (4, 120_000, (1, 2, 3))]


@pytest.mark.parametrize("precision", [nt.PREC_FP64, nt.PREC_MIXED])
@pytest.mark.parametrize("tile, count, order", [(t, n, o) for t, n, orders in SPLITS for o in orders])
def test_p2g_splits(tile, count, order, precision):
    n = int(round((count / 4) ** (1.0 / 3.0)))  # four particles a cell
    dx = 1.0 / n
    rng = np.random.default_rng(order + tile)
    s = scenes.base_specs((0, 0, 0), (1, 1, 1), (n, n, n), order, precision)
    s.gravity[2] = -9.81
    s.tile = tile
    s.autotune = 0
    s.use_temp = int(tile == 4)
    p = scenes.make_particles(rng.uniform(0.0, 1.0, (3, count)), (dx,) * 3, (2, 2, 1), 1000.0, 0, E=1e3, nu=0.3)
    p.rdata[nt.R_VEL:nt.R_VEL + 3] = rng.normal(0, 1, (3, count))
    p.rdata[nt.R_STRESS:nt.R_STRESS + 6] = rng.normal(0, 1e3, (6, count))
    p.rdata[nt.R_TEMPERATURE] = 300.0 + rng.uniform(-20.0, 20.0, count)
    p.rdata[nt.R_SPHEAT], p.rdata[nt.R_THERMCOND], p.rdata[nt.R_HEATSRC] = 900.0, 50.0, 1e5
    p.rdata[nt.R_HEATFLUX:nt.R_HEATFLUX + 3] = rng.normal(0, 100.0, (3, count))
    ctx = nt.Context(s)
    ctx.upload(p)
    o = orc.Oracle(s, 8)
    o.upload(p)
    tol = 1e-10 if precision == nt.PREC_FP64 else 2e-6

    def same(a, b, what):
        assert np.abs(a - b).max() <= tol * np.abs(b).max(), what

    ctx.P2G_Momentum(1, 1, 1)
    o.p2g_momentum(1, 1, 1)
    m = o.nodes(nt.N_MASS)
    same(ctx.nodes(nt.N_MASS), m, "mass")
    for d in range(3):
        same(ctx.nodes(nt.N_VEL + d) * m, o.nodes(nt.N_VEL + d) * m, f"momentum {d}")
        same(ctx.nodes(nt.N_FRC + d), o.nodes(nt.N_FRC + d), f"force {d}")
    if s.use_temp:
        ctx.P2G_Temperature(1, 1, 1)
        o.p2g_temperature(1, 1, 1)
        for c in (nt.N_MASS_SPHEAT, nt.N_MASS_SPHEAT_TEMP, nt.N_SOURCE_TEMP):
            same(ctx.nodes(c), o.nodes(c), f"component {c}")
    ctx.close()
