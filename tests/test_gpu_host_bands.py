"""Host right-hand sides, whose row bands depend on the grid and on whether the arrays are pinned
(downloads then begin with an upload) or pageable (four bands): every way gives the device call's
bits and dt, the result over its own input too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(40, 3), (33, 17), (300, 200), (512, 512), (1024, 600), (257, 1100)])
@pytest.mark.parametrize("ends", ["open", "periodic"])
@pytest.mark.parametrize("form", ["kapila", "bn", "mixed"])
def test_host_calls_equal_the_device_call(hp, nx, ny, ends, form):
    torch = pytest.importorskip("torch")
    bc = hp.BC_PERIODIC if ends == "periodic" else hp.BC_TRANSMISSIVE
    kw = {"bn": dict(system=hp.BAER_NUNZIATO, flags=hp.FLAG_BN_FIX_P2), "mixed": dict(system=hp.KAPILA_5EQN, precision=hp.PREC_MIXED),
          "kapila": dict(system=hp.KAPILA_5EQN)}[form]
    c = hp.Config(order=2, nx=nx, ny=ny, y_max=ny / nx, cfl=0.4, bc_left=bc, bc_right=bc, bc_bottom=bc, bc_top=bc, **kw)
    U = hp.initial_state(c, "bn_discs" if form == "bn" else "shock_bubble", seed=nx + ny)
    with hp.Solver(c) as s:
        dU = torch.from_numpy(U.copy()).cuda()
        dR = torch.empty_like(dU)
        dt = s.rhs_function_prim_device(0.0, dU.data_ptr(), dR.data_ptr())[0]
        want = dR.cpu().numpy().tobytes()
        for pinned in (False, True):
            for alias in (False, True):
                a = torch.from_numpy(U.copy())
                a = (a.pin_memory() if pinned else a).numpy()
                r = a if alias else np.full_like(U, np.nan)
                if pinned and not alias:
                    r = torch.full((U.size,), float("nan"), dtype=torch.float64).pin_memory().numpy()
                for _ in range(1 if alias else 2):   # the second call over buffers in use
                    _, dt_h, st = s.rhs_function_prim(0.0, a, r)
                    assert st == hp.OK and dt_h == dt, (pinned, alias)
                    assert r.tobytes() == want, (pinned, alias)
