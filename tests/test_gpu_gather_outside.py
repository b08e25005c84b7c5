"""The gathers of the step functions (G2P_Momentum, G2P_Temperature) for
particles on the high faces and outside the domain, where a program that moves
particles without Redistribute has them: a node outside a non-periodic domain
contributes nothing, a periodic axis wraps however far outside the particle is.
Reference: the sum over the in-domain nodes of compute_bounds with the oracle's
basis functions on the GPU's nodal fields.  FP64 within 1e-10 of the largest
node value (of its gradient over a cell); mixed within 2e-6: sums of at most 64
terms whose FP32 weights sum to at most 1 (gradients: 8 / dx), each rounded a
handful of times."""
import ctypes as C

import numpy as np
import pytest

from exagoop_b200 import native as nt, scenes
import orc

pytestmark = pytest.mark.gpu

N, DT = 24, 1e-3


def ptr(a):
    return a.ctypes.data_as(C.POINTER(C.c_double if a.dtype == np.float64 else C.c_int))


def bounds(iv, order, periodic):
    if order == 1:
        return range(0, 2)
    if periodic:
        return range(-1, 3)
    return range(0 if iv == 0 else -1, 2 if iv == N - 1 else 3)


def gathers(o, s, x, fields):
    """Sums of N f and grad N f over the in-domain nodes, per field."""
    order, per = s.order[0], [bool(s.periodic[d]) for d in range(3)]
    cell = np.floor((x - 0.0) * N).astype(np.int32)
    val, grad = np.zeros(len(fields)), np.zeros((len(fields), 3))
    for n in bounds(cell[2], order, per[2]):
        for m in bounds(cell[1], order, per[1]):
            for l in bounds(cell[0], order, per[0]):
                st = np.array([l, m, n], dtype=np.int32)
                node = [int(k) % N if p else int(k) for k, p in zip(cell + st, per)]
                if min(node) < 0 or max(node) > N:
                    continue
                g = np.zeros(3)
                w = o.L.orc_fn_basis_and_grad(o.h, ptr(st), ptr(cell), ptr(x), ptr(g))
                for k, f in enumerate(fields):
                    v = f[(node[2] * (N + 1) + node[1]) * (N + 1) + node[0]]
                    val[k] += w * v
                    grad[k] += g * v
    return val, grad


@pytest.mark.parametrize("precision", [nt.PREC_FP64, nt.PREC_MIXED])
@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("order", [1, 2, 3])
def test_gathers_outside(order, periodic, precision):
    dx = 1.0 / N
    s = scenes.base_specs((0, 0, 0), (1, 1, 1), (N, N, N), order, precision)
    s.autotune = 0
    s.use_temp = 1
    s.alpha_pic_flip = 0.95
    if periodic:
        s.periodic[0] = 1
        s.bclo[0] = s.bchi[0] = nt.BC_PERIODIC
    rng = np.random.default_rng(order)

    def fill(pos):
        p = scenes.make_particles(np.ascontiguousarray(pos), (dx,) * 3, (2, 2, 2), 1000.0, 0, E=1e3, nu=0.3)
        p.rdata[nt.R_VEL:nt.R_VEL + 3] = rng.normal(0, 1, (3, p.n))
        p.rdata[nt.R_STRESS:nt.R_STRESS + 6] = rng.normal(0, 1e3, (6, p.n))
        p.rdata[nt.R_TEMPERATURE] = 300.0 + rng.uniform(-20.0, 20.0, p.n)
        p.rdata[nt.R_SPHEAT], p.rdata[nt.R_THERMCOND], p.rdata[nt.R_HEATSRC] = 900.0, 50.0, 1e7
        return p

    ctx = nt.Context(s)
    ctx.upload(fill(rng.uniform(0.0, 1.0, (3, 8 * N ** 3))))
    ctx.P2G_Momentum(1, 1, 1)
    ctx.backup_current_velocity()
    ctx.Nodal_Time_Update_Momentum(DT)
    ctx.P2G_Temperature(1, 1, 1)
    ctx.backup_current_temperature()
    ctx.Nodal_Time_Update_Temperature(DT)
    ctx.store_delta_temperature()
    fields = [ctx.nodes(c) for c in [nt.N_VEL, nt.N_VEL + 1, nt.N_VEL + 2, nt.N_DVEL, nt.N_DVEL + 1, nt.N_DVEL + 2,
                                     nt.N_DELTA_TEMPERATURE, nt.N_TEMPERATURE]]
    # one axis on or past a face, the others inside; several axes; far outside
    off = [1.0, 1.0 + 0.3 * dx, 1.0 + 1.2 * dx, 1.0 + 2.7 * dx, -0.3 * dx, -1.2 * dx, -3.5 * dx, 1.0 - 1e-9]
    probes = [np.where(np.arange(3) == d, q, rng.uniform(0.1, 0.9, 3)) for q in off for d in range(3)]
    probes += [np.full(3, q) for q in off] + [np.array([q, 0.31, 0.47]) for q in (2.3, -1.6, 3.0)]
    p = fill(np.array(probes).T)
    ctx.upload(p)
    ctx.G2P_Momentum(1, 1, DT)
    ctx.G2P_Temperature(1, 1)
    g = ctx.download()
    ctx.close()
    o = orc.Oracle(s)
    tol = 1e-10 if precision == nt.PREC_FP64 else 2e-6
    top = [np.abs(f).max() for f in fields]
    sym = [(0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2)]
    for i, x in enumerate(probes):
        val, grad = gathers(o, s, x, fields)
        for d in range(3):
            assert abs(g.rdata[nt.R_VEL_PRIME + d, i] - val[d]) <= tol * top[d], (i, d)
            v = 0.95 * p.rdata[nt.R_VEL + d, i] + 0.95 * val[3 + d] + 0.05 * val[d]
            assert abs(g.rdata[nt.R_VEL + d, i] - v) <= tol * (top[d] + top[3 + d] + 5.0), (i, d)
        for c, (a, b) in enumerate(sym):
            e = 0.5 * (grad[a, b] + grad[b, a])
            assert abs(g.rdata[nt.R_STRAINRATE + c, i] - e) <= tol * 8.0 / dx * max(top[:3]), (i, a, b)
        dT = g.rdata[nt.R_TEMPERATURE, i] - p.rdata[nt.R_TEMPERATURE, i]
        assert abs(dT - val[6]) <= tol * top[6] + 1e-12 * 300.0, i
        if precision == nt.PREC_FP64:  # FP32 nodes hold T less a reference that a cut-off gradient does not cancel
            for d in range(3):
                assert abs(g.rdata[nt.R_HEATFLUX + d, i] + 50.0 * grad[7, d]) <= tol * 50.0 * 8.0 / dx * top[7], (i, d)
