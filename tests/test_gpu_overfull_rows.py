"""Small launches of scenes too dense for their queues: a row of the density walk
with more hits than its queue, lists that overflow, more neighbours than the
sums have room for, runs too long to be counted first. The bits are those of
the same scene in a large launch, beside a filler."""
import numpy as np
import pytest

from test_gpu_latency_forms import FILLER, cloud, filler

pytestmark = pytest.mark.gpu

# (particles, side of the cube): about 45, 64, 200, 340, 360, 600 neighbours,
# then runs of more than 1,024 candidates, spread and at one point
CLOUDS = [(1000, 1.6), (1500, 1.6), (1500, 1.1), (1500, 0.85), (1600, 0.85), (2500, 0.85),
          (5000, 0.75), (1300, 0.0)]


@pytest.mark.parametrize("table", [0, 1, 2])
def test_small_launch_equals_large(gpu_lib, table):
    import fluidsim
    dt = 1.0 / 240.0
    fp, fpos, fvel = filler()
    scs = [cloud(n, side, 300 + k) for k, (n, side) in enumerate(CLOUDS)]
    b = fluidsim.Batch(FILLER + sum(s[1].shape[0] for s in scs), len(scs) + 1)
    b.set_tuning(table=table)
    b.add(fp, fpos, fvel, dt)
    ids = [b.add(*s, dt) for s in scs]
    for _ in range(2):
        b.step(1)
    assert b.status() == 0
    for sid, (p, pos, vel) in zip(ids, scs):
        sim = fluidsim.FluidSimulation(p)
        sim.InitializeData(pos.shape[0], pos, vel)
        sim.set_tuning(table=table)
        for _ in range(2):
            sim.Update(dt, 1)
        want = sim.download()
        sim.close()
        for g, w in zip(b.download(sid), want):
            assert np.array_equal(g, w), pos.shape[0]
    b.close()
