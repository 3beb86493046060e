"""What the autotuners report is what they leave installed."""
import pytest

import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(64, 64), (251, 7), (500, 333), (40, 900), (1500, 700)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_solver_reports_the_shape_in_use(hp, nx, ny, precision):
    cfg = hp.Config(system=hp.KAPILA_5EQN, order=2, nx=nx, ny=ny, cfl=0.4, **cases.KAPILA_EOS,
                    precision={"fp64": hp.PREC_FP64, "mixed": hp.PREC_MIXED}[precision])
    with hp.Solver(cfg) as s:
        s.set_state(hp.initial_state(cfg, "shock_bubble", seed=1))
        for reps in (1, 3):
            cells, waves = s.autotune(reps)
            info = s.launch_info()
            tiles = info["grid"][0] * info["grid"][1]
            import torch
            slots = torch.cuda.get_device_properties(0).multi_processor_count * info["blocks_per_sm"]
            assert info["threads"] == 2 * cells
            # tiles of more than 8 rows are not cut further for more waves
            assert (tiles + slots - 1) // slots == waves or (tiles <= slots * waves and info["grid"][1] == max(1, ny // 8))


def test_batch_reports_the_shape_in_use(hp):
    def cfg(nx, ny):
        return hp.Config(system=hp.KAPILA_5EQN, order=2, nx=nx, ny=ny, cfl=0.4, **cases.KAPILA_EOS)
    with hp.Batch(max_instances=8, max_cells=512 * 512) as b:
        assert b.tiling() == (0, 0)
        for sizes in ([(90, 70)], [(300, 200), (128, 500)]):
            for nx, ny in sizes:
                b.add(cfg(nx, ny), hp.initial_state(cfg(nx, ny), "shock_bubble", seed=nx), 0.0, 1e30, 10)
            b.set_tiling(64, 48)
            assert b.tiling() == (64, 48)
            reported = b.autotune(2)
            cells, rows = b.tiling()
            items = b.info()["work_items"]
            b.set_tiling(*reported)
            if (cells, rows) == reported:
                assert b.info()["work_items"] == items
            assert b.tiling() == reported
