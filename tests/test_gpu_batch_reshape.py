"""A batch that takes another tile shape because members left goes on without waiting for the
steps that are queued, and with the same bits."""
import time

import pytest

import cases

pytestmark = pytest.mark.gpu


def test_advance_after_leaves_does_not_wait(hp):
    def cfg(n):
        return hp.Config(system=hp.KAPILA_5EQN, order=2, nx=n, ny=n, cfl=0.4, **cases.KAPILA_EOS)
    small = [hp.initial_state(cfg(100), "shock_bubble", seed=k, nbubbles=2) for k in (1, 2)]
    large = hp.initial_state(cfg(1000), "shock_bubble", seed=3)
    with hp.Batch(max_instances=16, max_cells=1000 * 1000) as b:
        keep = [b.add(cfg(100), U, 0.0, 1e30, 1 << 30) for U in small]
        go = [b.add(cfg(1000), large, 0.0, 1e30, 1 << 30) for _ in range(12)]
        b.advance(2)
        b.sync()
        tall = b.tiling()
        b.advance(25)
        for i in go:
            b.remove(i)
        t = time.perf_counter()
        b.advance(20)
        called = time.perf_counter() - t
        b.sync()
        done = time.perf_counter() - t
        print("advance returned after %.4f s, its steps were done after %.4f s" % (called, done), tall, b.tiling())
        assert b.tiling() != tall and b.tiling()[1] < tall[1]     # two small grids: short row runs
        assert done > 0.1 and called < 0.3 * done                  # 25 steps of 12 large grids were ahead
        got = [b.get_state(i).tobytes() for i in keep]
    for U, state in zip(small, got):
        with hp.Solver(cfg(100)) as s:
            s.set_state(U)
            s.solve(0.0, 1e30, 47)
            assert s.get_state().tobytes() == state


def test_shapes_change_back_and_forth(hp):
    """Members that come and go by turns: every advance may take another shape; the step graphs that
    are replaced go when their launches are done, the results stay."""
    def cfg(nx, ny):
        return hp.Config(system=hp.KAPILA_5EQN, order=2, nx=nx, ny=ny, cfl=0.4, **cases.KAPILA_EOS)
    U = hp.initial_state(cfg(96, 80), "shock_bubble", seed=1, nbubbles=2)
    V = hp.initial_state(cfg(640, 600), "shock_bubble", seed=2, nbubbles=2)
    seen = set()
    with hp.Batch(max_instances=8, max_cells=640 * 600) as b:
        i = b.add(cfg(96, 80), U, 0.0, 1e30, 1 << 30)
        n = 0
        for k in range(12):
            j = b.add(cfg(640, 600), V, 0.0, 1e30, 1 << 30)
            for steps in (3, 40):
                b.advance(steps)
                n += steps
                seen.add(b.tiling())
                if steps == 3:
                    b.remove(j)
        b.sync()
        assert len(seen) > 1
        got = b.get_state(i).tobytes()
    with hp.Solver(cfg(96, 80)) as s:
        s.set_state(U)
        s.solve(0.0, 1e30, n)
        assert s.get_state().tobytes() == got
