"""Results do not depend on the tile shape: a periodic grid and the same grid repeated side by side
and on top of itself have the same values cell by cell, in launches of other shapes."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("system", ["kapila", "bn", "euler"])
@pytest.mark.parametrize("precision", ["fp64", "mixed", "fast"])
def test_repeated_periodic_grids(hp, system, precision):
    kind, eos = {"kapila": ("shock_bubble", cases.KAPILA_EOS), "bn": ("bn_discs", cases.KAPILA_EOS),
                 "euler": ("euler_quadrants", cases.EULER_EOS)}[system]

    def cfg(nx, ny):     # cells of 1/64 at every size
        return hp.Config(system={"kapila": hp.KAPILA_5EQN, "bn": hp.BAER_NUNZIATO, "euler": hp.EULER}[system], nx=nx, ny=ny,
                         x_min=0.0, x_max=nx / 64, y_min=0.0, y_max=ny / 64, cfl=0.4, flags=hp.FLAG_BN_FIX_P2,
                         precision={"fp64": hp.PREC_FP64, "mixed": hp.PREC_MIXED, "fast": hp.PREC_FP64_FAST}[precision],
                         bc_left=hp.BC_PERIODIC, bc_right=hp.BC_PERIODIC, bc_bottom=hp.BC_PERIODIC, bc_top=hp.BC_PERIODIC, **eos)
    nx, ny = 64, 24
    U = hp.initial_state(cfg(nx, ny), kind, seed=9).reshape(ny, nx, -1)
    want, shapes = None, set()
    for a, b in ((1, 1), (1, 11), (9, 1), (24, 50)):
        c = cfg(a * nx, b * ny)
        V = np.ascontiguousarray(np.tile(U, (b, a, 1)).reshape(-1))
        with hp.Solver(c) as s:
            info = s.launch_info()
            shapes.add((info["threads"], -(-b * ny // info["grid"][1])))
            R, dt, st = s.rhs_function_prim(0.0, V)
            s.set_state(V)
            n, t, dt2, st2 = s.solve(0.0, 1e30, 2)
            S = s.get_state()
        assert st == st2 == hp.OK and n == 2
        got = []
        for X in (R, S):
            X = X.reshape(b, ny, a, nx, -1)
            assert all(X[j, :, i].tobytes() == X[0, :, 0].tobytes() for j in range(b) for i in range(a))
            got.append(X[0, :, 0].tobytes())
        got += [dt, dt2, t]
        want = want or got
        assert got == want
    assert len(shapes) > 2
    if system == "kapila":      # the other systems' tiles are estimated faster at 64 columns throughout
        assert {w // 2 for w, _ in shapes} == {64, 128}
