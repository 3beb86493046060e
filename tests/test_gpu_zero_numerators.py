"""Zero numerators in the branch-free divisions (csrc/hype_div.cuh drops the sign of a zero's
quotient): momenta and partial densities that are +0 or -0, bit for bit against the oracle."""
import numpy as np
import pytest

import cases
import oracle as O

pytestmark = pytest.mark.gpu

NAMES = ["bn_13x21_periodic_N1", "bn_23x19_fixed_p2", "bn_12x10_N3", "kapila_19x17_N1", "kapila_11x10_N0", "kapila_37x23_rough_mixed_bc",
         "euler_21x19_reflective_N1", "euler_16x16"]


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("where", ["all", "some"])
@pytest.mark.parametrize("zero", [0.0, -0.0])
def test_zero_momenta(hp, orc, name, where, zero):
    _, cfg, kind, seed = cases.case_by_name(name)
    nv = cases.to_pkg(cfg).nvar
    U = cases.state(cfg, kind, seed).reshape(cfg.ny, cfg.nx, nv).copy()
    take = np.ones((cfg.ny, cfg.nx), bool) if where == "all" else np.add.outer(np.arange(cfg.ny), np.arange(cfg.nx)) % 3 == 0
    for c in {4: (1, 2), 6: (2, 3), 9: (1, 2, 5, 6)}[nv]:
        U[take, c] = zero
    U = np.ascontiguousarray(U.reshape(-1))
    Ro, dto, sto = orc.rhs(cfg, U)
    with hp.Solver(cases.to_pkg(cfg)) as s:
        R, dt, st = s.rhs_function_prim(0.0, U)
    assert (st != hp.OK) == (sto != 0)
    if sto == 0:
        assert R.tobytes() == Ro.tobytes() and dt == dto


@pytest.mark.parametrize("order", [0, 1, 2])
def test_zero_partial_density(hp, orc, order):
    """Kapila with an absent phase: its partial density is zero in part of the grid."""
    cfg = O.Config(system=O.KAPILA, order=order, nx=41, ny=23, **cases.KAPILA_EOS)
    j, i = np.mgrid[0:23, 0:41]
    a = np.where(i < 20, 0.75, 0.25)
    rho1, rho2 = 1000.0, 1.0
    u, v, p = 0.5 * np.sin(0.3 * i), np.zeros_like(a), 1e5 + 10.0 * j
    g1, g2 = cfg.gamma1 - 1, cfg.gamma2 - 1
    q = [a * rho1, (1 - a) * rho2 * np.where(j < 12, 1.0, 0.0)]
    rho = q[0] + q[1]
    e = (p * (a * g2 + (1 - a) * g1) + a * cfg.gamma1 * cfg.pi1 * g2) / (g1 * g2)
    U = np.ascontiguousarray(np.stack([q[0], q[1], rho * u, -v, e + 0.5 * rho * u * u, a], -1).reshape(-1))
    with np.errstate(all="ignore"):
        Ro, dto, sto = orc.rhs(cfg, U)
    with hp.Solver(cases.to_pkg(cfg)) as s:
        R, dt, st = s.rhs_function_prim(0.0, U)
    assert (st != hp.OK) == (sto != 0)
    if sto == 0:
        nan = np.isnan(Ro)
        assert np.array_equal(nan, np.isnan(R)) and R[~nan].tobytes() == Ro[~nan].tobytes()
