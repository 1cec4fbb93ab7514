"""Batches of more tiny scenes than the latency forms hold tiles take the plain
forms, the density walk one candidate at a time: every scene steps bit for bit
as alone, where its launch is a latency form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 7, 8, 9, 31, 33, 40]  # 15 a scene on average


@pytest.mark.parametrize("count", [700, 2100])
@pytest.mark.parametrize("table", [0, 1, 2])
def test_tiny_scenes_equal_alone(gpu_lib, table, count):
    import fluidsim
    from test_gpu_latency_forms import cloud
    dt = 1.0 / 240.0
    scs = [cloud(n, 0.5, 50 + n) for n in SIZES]
    b = fluidsim.Batch(count * sum(SIZES), count)
    b.set_tuning(table=table)
    ids = [b.add(*scs[k % len(scs)], dt) for k in range(count)]
    for _ in range(2):
        b.step(2)
    assert b.status() == 0
    for k, (p, pos, vel) in enumerate(scs):
        sim = fluidsim.FluidSimulation(p)
        sim.InitializeData(pos.shape[0], pos, vel)
        sim.set_tuning(table=table)
        for _ in range(2):
            sim.Update(dt, 2)
        want = sim.download()
        sim.close()
        for sid in (ids[k], ids[count - len(scs) + (k - count) % len(scs)]):
            for g, w in zip(b.download(sid), want):
                assert np.array_equal(g, w), pos.shape[0]
    b.close()
