"""The largest blocks of the neighbour kernels take every size of launch: those
that would gather more list entries at once (and so more registers a thread) in
the default blocks, and those of another register cap. The results are the
default tuning's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33000, 50000, 90000, 210000, 250000, 620000])
@pytest.mark.parametrize("lanes", [32, 16])
def test_largest_blocks_equal_default(gpu_lib, n, lanes):
    import fluidsim
    from fluidsim import scenes
    pos, vel, bound = scenes.fill_box_scene(np.random.default_rng(n), n, 0.5, (1.0, 1.0, 1.0))
    p = scenes.SimParams(radius=0.35, bound=bound, **scenes.DAM_CONSTANTS)
    outs = []
    for block in (128, 1024):
        sim = fluidsim.FluidSimulation(p)
        sim.InitializeData(n, pos, vel)
        sim.set_tuning(block=block, force_block=block, particles_per_warp=lanes)
        sim.Update(1.0 / 120.0, 2)
        assert sim.status() == 0
        outs.append(sim.download())
        sim.close()
    for a, b in zip(*outs):
        assert np.array_equal(a, b)
