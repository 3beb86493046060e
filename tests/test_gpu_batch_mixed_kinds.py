"""Mixed Baer-Nunziato and Euler batches in a process that made no solver before.

Their kinds once took the shared memory and block counts of another path's
kernels: a Baer-Nunziato batch could not start unless a mixed solver had set
its kernels up, and an Euler one ran one block per SM.  Every grid of the batch
equals its lone mixed solver bit for bit, for both tile widths.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

CHILD = """
import sys
import numpy as np
import __graft_entry__ as g
hp = g._import_package()
system, kind, kw = {"bn": (hp.BAER_NUNZIATO, "bn_discs", dict(flags=hp.FLAG_BN_FIX_P2)),
                    "euler": (hp.EULER, "euler_quadrants", dict(gamma1=1.4, pi1=0.0))}[sys.argv[1]]
cells, rows = int(sys.argv[2]), int(sys.argv[3])
sizes = [(40, 24), (63, 97), (130, 70), (257, 33)]
cfgs = [hp.Config(system=system, order=2, nx=nx, ny=ny, y_max=ny / nx, cfl=0.4, precision=hp.PREC_MIXED, **kw) for nx, ny in sizes]
U = [hp.initial_state(c, kind, seed=k) for k, c in enumerate(cfgs)]
got = []
with hp.Batch(max_instances=8, max_cells=512 * 512) as b:
    ids = [b.add(c, u, 0.0, 1e30, 5) for c, u in zip(cfgs, U)]
    if cells:
        b.set_tiling(cells, rows)
    b.advance(5)
    b.sync()
    got = [b.get_state(i) for i in ids]
for c, u, x in zip(cfgs, U, got):
    with hp.Solver(c) as s:
        s.set_state(u)
        s.solve(0.0, 1e30, 5)
        assert s.get_state().tobytes() == x.tobytes(), (c.nx, c.ny)
print("equal")
"""


@pytest.mark.parametrize("system", ["bn", "euler"])
@pytest.mark.parametrize("cells,rows", [(0, 0), (64, 16), (128, 32)])
def test_batch_before_any_solver(system, cells, rows):
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([HERE, os.path.dirname(HERE)]))
    p = subprocess.run([sys.executable, "-c", CHILD, system, str(cells), str(rows)], env=env, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and "equal" in p.stdout, p.stderr[-2000:]
