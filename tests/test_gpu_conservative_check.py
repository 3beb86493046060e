"""The conservative path's admissibility check (rhs_function.c:380-420), bit for bit against the
oracle, on states whose cells are refused at some of their nodes and accepted at others: every
face, both Gauss points, every order, and Kapila's test of alpha_1 alone (only alpha_1 = 1 passes)."""
import numpy as np
import pytest

import cases
import oracle as O

pytestmark = pytest.mark.gpu


def _same(hp, orc, cfg, U):
    with hp.Solver(cases.to_pkg(cfg)) as s:
        R, dt, st = s.rhs_function_prim(0.0, U)
    with np.errstate(all="ignore"):
        Ro, dto, sto = orc.rhs(cfg, U)
    assert (st != hp.OK) == (sto != 0)
    if sto != 0:
        return
    nan = np.isnan(Ro)
    assert np.array_equal(nan, np.isnan(R))
    assert R[~nan].tobytes() == Ro[~nan].tobytes()
    assert dt == dto or (np.isnan(dt) and np.isnan(dto))


def _euler(nx, ny, along, order):
    """Velocity jumps along one axis (or both), pressures that the jumps' kinetic energy outweighs
    at the faces of some cells."""
    cfg = O.Config(system=O.EULER, order=order, nx=nx, ny=ny, conservative=1, **cases.EULER_EOS)
    r = np.random.default_rng(17 + order)
    j, i = np.mgrid[0:ny, 0:nx]
    phase = {"x": i, "y": j, "both": i + 2 * j}[along]
    rho = 1.0 + 0.9 * np.sin(1.7 * phase + 0.1 * r.random((ny, nx)))
    u, v = 3.0 * np.cos(1.1 * phase), 2.0 * np.sin(0.9 * phase)
    p = 0.02 + 0.05 * r.random((ny, nx))
    Q = np.stack([rho, rho * u, rho * v, p / (cfg.gamma1 - 1) + 0.5 * rho * (u * u + v * v)], -1)
    return cfg, np.ascontiguousarray(Q.reshape(-1))


def _bn(nx, ny, along, order):
    cfg = O.Config(system=O.BN, order=order, nx=nx, ny=ny, conservative=1, bn_fixed_p2=1, **cases.KAPILA_EOS)
    r = np.random.default_rng(23 + order)
    j, i = np.mgrid[0:ny, 0:nx]
    phase = {"x": i, "y": j, "both": i + 2 * j}[along]
    a = 0.5 + 0.45 * np.sin(1.3 * phase)
    out = []
    for al, rr, p, g, pi in ((a, 1000.0, 1e5, cfg.gamma1, cfg.pi1), (1 - a, 1.0, 40.0, cfg.gamma2, cfg.pi2)):
        rho = rr * (1.0 + 0.8 * np.sin(1.7 * phase + 0.1 * r.random((ny, nx))))
        u, v = 9.0 * np.cos(1.1 * phase), 7.0 * np.sin(0.9 * phase)
        p = p * (0.5 + r.random((ny, nx)))
        out += [al * rho, al * rho * u, al * rho * v, al * ((p + g * pi) / (g - 1) + 0.5 * rho * (u * u + v * v))]
    return cfg, np.ascontiguousarray(np.stack(out + [a], -1).reshape(-1))


@pytest.mark.parametrize("order", [1, 2, 3])
@pytest.mark.parametrize("along", ["x", "y", "both"])
@pytest.mark.parametrize("state", [_euler, _bn])
@pytest.mark.parametrize("nx,ny", [(37, 21), (131, 40), (250, 9)])
def test_cells_refused_at_some_nodes(hp, orc, state, along, order, nx, ny):
    _same(hp, orc, *state(nx, ny, along, order))


@pytest.mark.parametrize("order", [1, 2, 3])
@pytest.mark.parametrize("viscous", [0, 1])
@pytest.mark.parametrize("trace", [0.0, 1e-30])
def test_kapila_regions_of_pure_liquid(hp, orc, order, viscous, trace):
    """alpha_1 = 1 exactly in part of the grid: those cells pass the test of alpha_1 and go on to the
    others, their neighbours do not."""
    nx, ny = 67, 33
    cfg = O.Config(system=O.KAPILA, order=order, nx=nx, ny=ny, conservative=1, viscous=viscous, mu1=0.4, mu2=0.05, **cases.KAPILA_EOS)
    r = np.random.default_rng(5)
    j, i = np.mgrid[0:ny, 0:nx]
    a = np.where((i > 20) & (i < 45) & (j > 8) & (j < 25), 1.0, 0.5 + 0.4 * np.sin(0.3 * i) * np.cos(0.2 * j))
    r1, r2 = 1000.0 * (1 + 0.1 * r.random((ny, nx))), np.where(a < 1.0, 1.0, trace)
    u, v, p = r.uniform(-1, 1, (ny, nx)), r.uniform(-1, 1, (ny, nx)), 1e5 * (1 + 0.1 * r.random((ny, nx)))
    g1, g2 = cfg.gamma1 - 1, cfg.gamma2 - 1
    q1 = np.where(a < 1.0, (1 - a) * r2, trace)
    rho = a * r1 + q1
    e = (p * (a * g2 + (1 - a) * g1) + a * cfg.gamma1 * cfg.pi1 * g2 + (1 - a) * cfg.gamma2 * cfg.pi2 * g1) / (g1 * g2)
    Q = np.stack([a * r1, q1, rho * u, rho * v, e + 0.5 * rho * (u * u + v * v), a], -1)
    _same(hp, orc, cfg, np.ascontiguousarray(Q.reshape(-1)))
