"""hype_rhs_prim_device on the arrays its callers may pass: a result over its own input, wholly
or in part, on rows that TMA can load as they are and on rows that it cannot."""
import numpy as np
import pytest

import cases
import oracle as O

pytestmark = pytest.mark.gpu

SYSTEMS = {"kapila": (O.KAPILA, "bubble", cases.KAPILA_EOS), "bn": (O.BN, "discs", cases.KAPILA_EOS),
           "euler": (O.EULER, "quadrants", cases.EULER_EOS)}


def _case(system, nx, ny, ends=O.TRANSMISSIVE, order=2):
    sys_id, kind, eos = SYSTEMS[system]
    cfg = O.Config(system=sys_id, order=order, nx=nx, ny=ny, bc_left=ends, bc_right=ends, bc_bottom=ends, bc_top=ends, **eos)
    if system == "bn":
        cfg.bn_fixed_p2 = 1
    return cfg, cases.state(cfg, kind, 11)


@pytest.mark.parametrize("system", ["kapila", "bn", "euler"])
@pytest.mark.parametrize("nx,ny", [(300, 200), (131, 90)])
@pytest.mark.parametrize("ends", [O.TRANSMISSIVE, O.PERIODIC], ids=["open", "periodic"])
@pytest.mark.parametrize("precision", ["fp64", "fast"])
def test_result_over_its_input(hp, orc, system, nx, ny, ends, precision):
    """dRHS == dU, and dRHS a few elements or half an array before or behind dU: what a call with
    arrays of their own gives, on an aligned input and on one moved by 8 bytes.  Strips and row
    runs read their neighbours' cells, so a launch may not store what it still loads."""
    import torch
    cfg, U = _case(system, nx, ny, ends)
    pc = cases.to_pkg(cfg)
    pc.precision = {"fp64": hp.PREC_FP64, "fast": hp.PREC_FP64_FAST}[precision]
    n = U.size
    room = torch.empty(3 * n + 8, dtype=torch.float64, device="cuda")
    with hp.Solver(pc) as s:
        def call(at, to):
            room.fill_(float("nan"))
            room[at:at + n].copy_(torch.from_numpy(U))
            torch.cuda.synchronize()
            dt, st = s.rhs_function_prim_device(0.0, room.data_ptr() + 8 * at, room.data_ptr() + 8 * to)
            assert st == hp.OK
            return room[to:to + n].cpu().numpy().tobytes(), dt
        first = n + n % 2
        apart = call(first + 1, 0)   # by way of planes: the performance form's two kernels round differently
        if precision == "fp64":
            Ro, dto, _ = orc.rhs(cfg, U)
            assert apart == (Ro.tobytes(), dto)
            assert call(first, 0) == apart
        for at in (first, first + 1):
            for to in (at, at + 2, at - 2, at + n // 2, at - n // 2):
                assert call(at, to) == apart


@pytest.mark.parametrize("system", ["kapila", "bn", "euler"])
@pytest.mark.parametrize("order", [0, 1, 2, 3])
@pytest.mark.parametrize("nx,ny", [(3, 3), (65, 7), (126, 4), (131, 9), (260, 30)])
@pytest.mark.parametrize("ends", [O.TRANSMISSIVE, O.REFLECTIVE, O.PERIODIC], ids=["open", "walls", "periodic"])
def test_performance_form(hp, orc, system, order, nx, ny, ends):
    """The performance form's device calls, reading the caller's rows (aligned arrays) or by way of
    planes (arrays moved by 8 bytes): both within its bar of the reference's arithmetic, and by way
    of planes the host call's bits."""
    import torch
    from test_gpu_fast import TOL, assert_within, field_errors, sensitivity
    cfg, U = _case(system, nx, ny, ends, order)
    Ro, dto, sto = orc.rhs(cfg, U)
    pc = cases.to_pkg(cfg)
    pc.precision = hp.PREC_FP64_FAST
    room = torch.zeros(U.size + 1, dtype=torch.float64, device="cuda")
    got = []
    with hp.Solver(pc) as s:
        for shift in (0, 1):
            dU, dR = room[shift:shift + U.size], torch.full((U.size,), np.nan, dtype=torch.float64, device="cuda")
            dU.copy_(torch.from_numpy(U))
            torch.cuda.synchronize()
            dt, st = s.rhs_function_prim_device(0.0, dU.data_ptr(), dR.data_ptr())
            assert (st != hp.OK) == (sto != 0)
            got.append((dR.cpu().numpy(), dt))
        R, dt, st = s.rhs_function_prim(0.0, U)
    if sto != 0:
        return
    assert R.tobytes() == got[1][0].tobytes() and dt == got[1][1]
    for R, dt in got:
        err = field_errors(R, Ro, cfg.system)
        kappa = sensitivity(lambda X: orc.rhs(cfg, X)[0], U, cfg.system) if err.max() > TOL else 0.0 * err
        assert_within(err, kappa, (system, order, nx, ny))
        assert abs(dt - dto) <= TOL * dto
