"""Small launches take the latency forms of the neighbour kernels (several
warps a tile, ordered sums through shared memory), large ones the plain forms
(a lane a particle). Both must give the same bits: a scene stepped alone (a
small launch) against the same scene in a batch beside a filler that makes
the launch a large one. Sizes at the edges of the eight-particle groups and of
the tiles; clouds dense enough to overflow the per-row queues (16 hits) and
the neighbour lists (64); grid and bucket key tables."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FILLER = 70000  # particles: more than the latency forms take


def cloud(n, side, seed):
    """n particles, uniform in a cube of `side` off the origin, in a 6^3 box."""
    from fluidsim import scenes
    rng = np.random.default_rng(seed)
    pos = (rng.uniform(-0.5 * side, 0.5 * side, (n, 3)) - 0.7).astype(np.float32)
    vel = rng.uniform(-1.0, 1.0, (n, 3)).astype(np.float32)
    p = scenes.SimParams(radius=0.35, bound=(6.0, 6.0, 6.0), **scenes.DAM_CONSTANTS)
    return p, pos, vel


def filler():
    from fluidsim import scenes
    rng = np.random.default_rng(3)
    pos, vel, bound = scenes.fill_box_scene(rng, FILLER, 0.5, (1.0, 1.0, 1.0))
    return scenes.SimParams(radius=0.35, bound=bound, **scenes.DAM_CONSTANTS), pos, vel


# (particles, side of the cube): sparse, then 10, 40 and 200 neighbours
CLOUDS = [(1, 1.0), (7, 0.8), (8, 0.8), (9, 0.8), (31, 1.0), (33, 1.0), (257, 1.2),
          (1000, 2.4), (1500, 1.5), (1500, 0.9), (4096, 3.6), (28801, 5.0)]


@pytest.mark.parametrize("table", [0, 1, 2])
def test_small_launch_equals_large(gpu_lib, table):
    import fluidsim
    dt = 1.0 / 240.0
    fp, fpos, fvel = filler()
    scs = [cloud(n, side, 100 + k) for k, (n, side) in enumerate(CLOUDS)]
    b = fluidsim.Batch(FILLER + sum(s[1].shape[0] for s in scs), len(scs) + 1)
    b.set_tuning(table=table)
    b.add(fp, fpos, fvel, dt)
    ids = [b.add(*s, dt) for s in scs]
    for _ in range(2):
        b.step(2)
    assert b.status() == 0
    most = 0
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
        # r^2 - weighted count of neighbours: the densest clouds overflow the lists
        d2 = ((pos[None, 0] - pos) ** 2).sum(1)
        most = max(most, int((d2 < 0.35 ** 2).sum()))
    b.close()
    assert most > 65
