"""Every gather batch the tuning takes steps in every block it takes: where a
block's threads leave a kernel of that batch too few registers, a smaller batch
runs. The results are the default tuning's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [50000, 350000])
@pytest.mark.parametrize("lanes", [32, 16])
@pytest.mark.parametrize("table", [0, 1])
def test_gathers_in_large_blocks(gpu_lib, n, lanes, table):
    import fluidsim
    from fluidsim import scenes
    pos, vel, bound = scenes.fill_box_scene(np.random.default_rng(n), n, 0.5, (1.0, 1.0, 1.0))
    p = scenes.SimParams(radius=0.35, bound=bound, **scenes.DAM_CONSTANTS)

    def run(**tuning):
        sim = fluidsim.FluidSimulation(p)
        sim.InitializeData(n, pos, vel)
        sim.set_tuning(particles_per_warp=lanes, table=table, **tuning)
        sim.Update(1.0 / 120.0, 1)
        assert sim.status() == 0
        out = sim.download()
        sim.close()
        return out

    want = run()
    for gather in (2, 3, 4, 8):
        for block in (512, 544, 768, 1024):
            for a, b in zip(run(gather=gather, force_block=block), want):
                assert np.array_equal(a, b), (gather, block)
