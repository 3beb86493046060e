"""The tile's point values and its quick admissibility test (csrc/hype_stage_tile.cuh,
System<SYS>::pad_quick) where they can go wrong, bit for bit against the oracle.

 * Values on both sides of the ranges pad_quick accepts: densities and pressures scaled far
   out of them, negative pressures, alpha_1 at 0 and 1, gammas and P_inf that quick_eos refuses.
   Most of these cells take the exact check, some of them the minmod fallback.
 * Cells that are not finite: their neighbours' results carry the same NaNs.
 * Strips that leave warps, or all but a few threads of the last warp, without a cell.
"""
import numpy as np
import pytest

import cases
import oracle as O

pytestmark = pytest.mark.gpu


def _same(hp, orc, cfg, U):
    with hp.Solver(cases.to_pkg(cfg)) as s:
        R, dt, st = s.rhs_function_prim(0.0, U)
    Ro, dto, sto = orc.rhs(cfg, U)
    assert (st != hp.OK) == (sto != 0)
    if sto != 0:      # the oracle ends at an inadmissible face, its RHS is incomplete
        return
    nan = np.isnan(Ro)
    assert np.array_equal(nan, np.isnan(R))
    assert R[~nan].tobytes() == Ro[~nan].tobytes()
    assert dt == dto or (np.isnan(dt) and np.isnan(dto))


def _kapila(order, nx, ny, scale_r=1.0, scale_p=1.0, alpha=None, **eos):
    cfg = O.Config(system=O.KAPILA, order=order, nx=nx, ny=ny, **{**cases.KAPILA_EOS, **eos})
    r = np.random.default_rng(nx * 131 + ny)
    a = np.clip(np.where(r.random((ny, nx)) < 0.5, 0.03, 0.97) + 0.02 * r.standard_normal((ny, nx)), 1e-3, 1 - 1e-3)
    if alpha is not None:
        a[ny // 2, nx // 3:nx // 2] = alpha
    r1, r2 = scale_r * 1000 * r.uniform(0.5, 2, (ny, nx)), scale_r * r.uniform(0.5, 2, (ny, nx))
    p = scale_p * r.uniform(0.1, 1.0, (ny, nx))
    u, v = r.uniform(-1, 1, (ny, nx)), r.uniform(-1, 1, (ny, nx))
    g1, g2 = cfg.gamma1 - 1, cfg.gamma2 - 1
    rho = a * r1 + (1 - a) * r2
    e = (p * (a * g2 + (1 - a) * g1) + a * cfg.gamma1 * cfg.pi1 * g2 + (1 - a) * cfg.gamma2 * cfg.pi2 * g1) / (g1 * g2)
    Q = np.stack([a * r1, (1 - a) * r2, rho * u, rho * v, e + 0.5 * rho * (u * u + v * v), a], -1)
    return cfg, np.ascontiguousarray(Q.reshape(-1))


@pytest.mark.parametrize("order", [2, 3])
@pytest.mark.parametrize("kw", [
    dict(scale_r=2.0 ** 40, scale_p=2.0 ** 30), dict(scale_r=2.0 ** -45, scale_p=1.0), dict(scale_p=2.0 ** -24, pi1=0.0),
    dict(scale_p=-1e5), dict(scale_p=1e5, alpha=0.0), dict(scale_p=1e5, alpha=1.0), dict(scale_p=1e5, gamma1=2000.0),
    dict(scale_p=10.0, pi1=-0.5),
], ids=["dense", "thin", "low_p", "tension", "alpha0", "alpha1", "gamma", "pi_neg"])
def test_kapila_out_of_the_quick_range(hp, orc, order, kw):
    with np.errstate(all="ignore"):
        _same(hp, orc, *_kapila(order, 41, 23, **kw))


@pytest.mark.parametrize("system", ["kapila", "bn", "euler"])
@pytest.mark.parametrize("value", [np.nan, np.inf, 0.0, -1.0])
def test_bad_cells(hp, orc, system, value):
    name = {"kapila": "kapila_37x23_rough_mixed_bc", "bn": "bn_23x19_fixed_p2", "euler": "euler_16x16"}[system]
    _, cfg, kind, seed = cases.case_by_name(name)
    U = cases.state(cfg, kind, seed).copy()
    nv = cases.to_pkg(cfg).nvar
    U[(cfg.nx * (cfg.ny // 2) + cfg.nx // 2) * nv] = value      # a partial density
    _same(hp, orc, cfg, U)


@pytest.mark.parametrize("nx", [3, 15, 16, 33, 124, 125, 131, 249, 373])
def test_strip_widths(hp, orc, nx):
    for order in (1, 2):
        _same(hp, orc, *_kapila(order, nx, 9, scale_p=1e5))


@pytest.mark.parametrize("name", ["bn_23x19_fixed_p2", "bn_13x21_periodic_N1", "bn_12x10_N3", "euler_21x19_reflective_N1", "euler_16x16"])
@pytest.mark.parametrize("scale", [2.0 ** -60, 2.0 ** 60, 2.0 ** -170, 2.0 ** 170])
def test_scaled_units(hp, orc, name, scale):
    """Densities, momenta and energies in other units: past 2^100 or below 2^-100 the Riemann
    solver's branch-free divisions hand over to the compiler's."""
    _, cfg, kind, seed = cases.case_by_name(name)
    U = cases.state(cfg, kind, seed).reshape(-1, cases.to_pkg(cfg).nvar).copy()
    k = 8 if U.shape[1] == 9 else U.shape[1]
    U[:, :k] *= scale
    cfg.pi1, cfg.pi2 = cfg.pi1 * scale, cfg.pi2 * scale
    _same(hp, orc, cfg, U.reshape(-1))


def test_repeated_batches_give_the_same_bits(hp):
    """Warps of a block run up to most of a row apart; whatever their order, neighbouring columns'
    fluxes are read before the next row's coefficients replace them."""
    grids = [(hp.Config(nx=nx, ny=ny, cfl=0.4, bc_bottom=hp.BC_REFLECTIVE, bc_top=hp.BC_REFLECTIVE, **cases.KAPILA_EOS), k)
             for k, (nx, ny) in enumerate([(476, 435), (380, 486), (409, 300), (230, 290)])]
    states = [hp.initial_state(c, "shock_bubble", seed=k, nbubbles=4) for c, k in grids]
    seen = set()
    with hp.Batch(max_instances=len(grids), max_cells=512 * 512) as b:
        for _ in range(8):
            ids = [b.add(c, U, 0.0, 1e30, 12) for (c, _), U in zip(grids, states)]
            b.advance(12)
            b.sync()
            seen.add(b"".join(b.get_state(i).tobytes() for i in ids))
            for i in ids:
                b.remove(i)
    assert len(seen) == 1
    lone = []
    for (c, _), U in zip(grids, states):
        with hp.Solver(c) as s:
            s.set_state(U)
            s.solve(0.0, 1e30, 12)
            lone.append(s.get_state().tobytes())
    assert seen == {b"".join(lone)}


@pytest.mark.parametrize("ny", [3, 4, 7, 16, 33, 150])
def test_run_heights(hp, orc, ny):
    """The estimated tile shapes: short grids take row runs of one to a few rows."""
    for order in (1, 2, 3):
        _same(hp, orc, *_kapila(order, 131, ny, scale_p=1e5))


@pytest.mark.parametrize("system", ["kapila", "bn", "euler"])
@pytest.mark.parametrize("precision", ["mixed", "fast"])
@pytest.mark.parametrize("nx,ny", [(64, 64), (131, 5), (37, 200)])
def test_shapes_of_the_other_forms(hp, system, precision, nx, ny):
    """The right-hand side does not depend on the tile shape: the estimated one against those the
    autotuner tries and keeps, and against row bands of a host call."""
    kind, eos = {"kapila": ("shock_bubble", cases.KAPILA_EOS), "bn": ("bn_discs", cases.KAPILA_EOS),
                 "euler": ("euler_quadrants", cases.EULER_EOS)}[system]
    cfg = hp.Config(system={"kapila": hp.KAPILA_5EQN, "bn": hp.BAER_NUNZIATO, "euler": hp.EULER}[system], nx=nx, ny=ny, cfl=0.4,
                    precision={"mixed": hp.PREC_MIXED, "fast": hp.PREC_FP64_FAST}[precision], flags=hp.FLAG_BN_FIX_P2, **eos)
    U = hp.initial_state(cfg, kind, seed=5)
    got = []
    with hp.Solver(cfg) as s:
        for tune in (False, True):
            if tune:
                s.autotune(1)
            s.set_state(U)
            n, t, dt, st = s.solve(0.0, 1e30, 3)
            got.append((n, t, dt, st, s.get_state().tobytes(), s.rhs_function_prim(0.0, U)[0].tobytes()))
    assert got[0] == got[1] and got[0][3] == hp.OK


@pytest.mark.parametrize("nx,ny", [(18000, 16), (2600, 12), (300, 41), (700, 130)])
@pytest.mark.parametrize("bc", [O.TRANSMISSIVE, O.PERIODIC])
def test_bands_of_host_calls(hp, orc, nx, ny, bc):
    """Row bands of host right-hand sides and host steps on wide, short grids: every band has the
    rows its neighbours' stencils read."""
    cfg, U = _kapila(2, nx, ny, scale_p=1e5)
    cfg.bc_left = cfg.bc_right = cfg.bc_bottom = cfg.bc_top = bc
    _same(hp, orc, cfg, U)
    out = np.empty_like(U)
    with hp.Solver(cases.to_pkg(cfg)) as s:
        s.set_state(U)
        s.begin(0.0, 1e30, 2)
        s.advance(1)
        st = s.wait()
        state = s.get_state()
        s.set_state(U)
        s.begin(0.0, 1e30, 2)
        assert s.advance_host(U, out, 1) == st and out.tobytes() == state.tobytes()


@pytest.mark.parametrize("system", ["kapila", "bn", "euler"])
@pytest.mark.parametrize("order", [0, 1, 2, 3])
@pytest.mark.parametrize("nx,ny", [(3, 3), (64, 5), (65, 7), (126, 4), (131, 9), (260, 6)])
@pytest.mark.parametrize("ends", ["walls", "periodic"])
def test_device_calls_read_cell_major_arrays(hp, orc, system, order, nx, ny, ends):
    """hype_rhs_prim_device loads the caller's cell-major rows by TMA where they start on 16-byte
    boundaries (an odd Baer-Nunziato width does not, nor does an array moved by 8 bytes) and
    converts the array to planes elsewhere: the oracle's bits either way."""
    import torch
    kind, eos, nv = {"kapila": ("bubble", cases.KAPILA_EOS, 6), "bn": ("discs", cases.KAPILA_EOS, 9),
                     "euler": ("quadrants", cases.EULER_EOS, 4)}[system]
    lr, bt = ((O.REFLECTIVE, O.TRANSMISSIVE), (O.TRANSMISSIVE, O.REFLECTIVE)) if ends == "walls" else ((O.PERIODIC,) * 2,) * 2
    cfg = O.Config(system={"kapila": O.KAPILA, "bn": O.BN, "euler": O.EULER}[system], order=order, nx=nx, ny=ny, bc_left=lr[0],
                   bc_right=lr[1], bc_bottom=bt[0], bc_top=bt[1], **eos)
    if system == "bn":
        cfg.bn_fixed_p2 = 1
    U = cases.state(cfg, kind, 7)
    Ro, dto, sto = orc.rhs(cfg, U)
    room = torch.zeros(U.size + 1, dtype=torch.float64, device="cuda")
    with hp.Solver(cases.to_pkg(cfg)) as s:
        for shift in (0, 1):
            dU, dR = room[shift:shift + U.size], torch.full((U.size,), np.nan, dtype=torch.float64, device="cuda")
            dU.copy_(torch.from_numpy(U))
            torch.cuda.synchronize()
            dt, st = s.rhs_function_prim_device(0.0, dU.data_ptr(), dR.data_ptr())
            assert (st != hp.OK) == (sto != 0)
            if sto == 0:
                assert dR.cpu().numpy().tobytes() == Ro.tobytes() and dt == dto


@pytest.mark.parametrize("order", [1, 2, 3])
def test_liquid_under_tension(hp, orc, order):
    """Negative pressures above -P_inf in an almost pure liquid: the trace gas's p + pi_2 is negative,
    the quick range refuses every cell and the mixture's denominators may cancel."""
    cfg, U = _kapila(order, 67, 21, scale_p=-1e5)
    U = U.reshape(-1, 6)
    a0, a1 = U[:, 5].copy(), 1.0 - 1e-6 * (1.0 + np.arange(U.shape[0]) % 7)
    U[:, 0] *= a1 / a0
    U[:, 1] *= (1.0 - a1) / (1.0 - a0)
    U[:, 5] = a1
    rho = U[:, 0] + U[:, 1]
    U[:, 2:4] = 0.01 * rho[:, None] * np.sin(np.arange(2 * U.shape[0]).reshape(-1, 2))
    g1, g2 = cfg.gamma1 - 1, cfg.gamma2 - 1
    p = -1e3 * (1.0 + (np.arange(U.shape[0]) % 13))
    U[:, 4] = (p * (a1 * g2 + (1 - a1) * g1) + a1 * cfg.gamma1 * cfg.pi1 * g2) / (g1 * g2) + 0.5 * (U[:, 2] ** 2 + U[:, 3] ** 2) / rho
    _same(hp, orc, cfg, np.ascontiguousarray(U.reshape(-1)))
