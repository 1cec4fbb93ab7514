"""Launches of many waves run the viscosity pass at more warps an SM (another
register cap, the same code), those of a little more than one wave also the
density pass, and some of a few waves gather three list entries at once: scenes
in a batch beside a filler of such a size step bit for bit as alone, where the
launch is small. Clouds from a lone particle to lists that overflow, under each
form of the key tables."""
import numpy as np
import pytest

from test_gpu_latency_forms import cloud

pytestmark = pytest.mark.gpu

# particles: between 40 and 48 warps an SM; two waves of 32; two of 48; more than three of 40
FILLERS = [205000, 250000, 430000, 600000]


@pytest.mark.parametrize("fill", FILLERS)
@pytest.mark.parametrize("table", [0, 1, 2])
def test_large_launch_equals_alone(gpu_lib, table, fill):
    import fluidsim
    from fluidsim import scenes
    dt = 1.0 / 240.0
    scs = [cloud(n, side, 7 + n) for n, side in [(1, 1.0), (33, 1.0), (1500, 0.9), (4097, 3.6)]]
    pos, vel, bound = scenes.fill_box_scene(np.random.default_rng(5), fill, 0.5, (1.0, 1.0, 1.0))
    filler = scenes.SimParams(radius=0.35, bound=bound, **scenes.DAM_CONSTANTS)
    b = fluidsim.Batch(fill + sum(s[1].shape[0] for s in scs), len(scs) + 1)
    b.set_tuning(table=table)
    b.add(filler, pos, vel, dt)
    ids = [b.add(*s, dt) for s in scs]
    for _ in range(2):
        b.step(2)
    assert b.status() == 0
    for sid, (p, pos, vel) in zip(ids, scs):
        sim = fluidsim.FluidSimulation(p)
        sim.InitializeData(pos.shape[0], pos, vel)
        sim.set_tuning(table=table)
        for _ in range(2):
            sim.Update(dt, 2)
        want = sim.download()
        sim.close()
        for g, w in zip(b.download(sid), want):
            assert np.array_equal(g, w), pos.shape[0]
    b.close()
