"""The autotuner changes no setting that makes no difference to the launch it
times: small launches choose their blocks and gather batches themselves, and a
choice among equals would be chance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4096, 50000])
@pytest.mark.parametrize("block,force_block,gather", [(128, 0, 2), (256, 96, 3), (1024, 0, 2)])
def test_settings_without_effect_stay(gpu_lib, n, block, force_block, gather):
    import fluidsim
    from fluidsim import scenes
    pos, vel, bound = scenes.fill_box_scene(np.random.default_rng(n), n, 0.5, (1.0, 1.0, 1.0))
    p = scenes.SimParams(radius=0.35, bound=bound, **scenes.DAM_CONSTANTS)
    sim = fluidsim.FluidSimulation(p)
    sim.InitializeData(n, pos, vel)
    sim.set_tuning(block=block, force_block=force_block, gather=gather)
    best, ms = sim.autotune(1.0 / 120.0, 2, steps_per_trial=2)
    sim.close()
    assert ms > 0.0
    if n > 28800:  # the force kernels run in blocks of the tuning, and gather 4 or 8
        assert best["gather"] in (gather, 8)
    elif best["particles_per_warp"] == 32:
        assert (best["force_block"], best["gather"]) == (force_block, gather)
        if best["cell_tile"] == 1:
            assert best["block"] == block


def test_a_tuning_that_cannot_run_is_left(gpu_lib):
    import fluidsim
    from fluidsim import scenes
    sc = scenes.dam_break_16k()
    sim = fluidsim.FluidSimulation(sc["params"])
    sim.InitializeData(sc["pos"].shape[0], sc["pos"], sc["vel"])
    sim.set_tuning(block=1024, cell_tile=256)  # more registers than such a block has
    best, ms = sim.autotune(sc["dt"], 3, steps_per_trial=1)
    assert ms > 0.0 and best["block"] <= 512
    sim.Update(sc["dt"], 3)
    assert sim.status() == 0
    sim.close()
