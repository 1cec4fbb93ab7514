"""A coincident pair is pushed along y only (the reference's fallback
direction). With a pressure that overflows, y is lost and flagged, and x and z
stay what they are in every form of the force kernels: a scene alone (a small
launch) against the same scene beside a filler (a large one)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("table", [0, 1])
@pytest.mark.parametrize("mult", [500.0, 3e38])
def test_coincident_pair(gpu_lib, table, mult):
    import fluidsim
    from fluidsim import scenes
    dt = 1.0 / 240.0
    pos = np.array([[0.1, 0.2, 0.3], [0.1, 0.2, 0.3], [2.0, 2.0, 2.0]], np.float32)
    vel = np.array([[0.5, 0.25, -0.5], [0.5, 0.25, -0.5], [1.0, 0.0, -1.0]], np.float32)
    p = scenes.SimParams(radius=0.35, bound=(6.0, 6.0, 6.0),
                         **dict(scenes.DAM_CONSTANTS, pressure_mult=mult))
    fpos, fvel, bound = scenes.fill_box_scene(np.random.default_rng(3), 70000, 0.5,
                                              (1.0, 1.0, 1.0))
    b = fluidsim.Batch(70003, 2)
    b.set_tuning(table=table)
    b.add(scenes.SimParams(radius=0.35, bound=bound, **scenes.DAM_CONSTANTS), fpos, fvel, dt)
    sid = b.add(p, pos, vel, dt)
    b.step(1)
    want = b.download(sid)
    b.close()
    sim = fluidsim.FluidSimulation(p)
    sim.InitializeData(3, pos, vel)
    sim.set_tuning(table=table)
    sim.Update(dt, 1)
    got = sim.download()
    assert (sim.status() != 0) == (mult > 1e30)
    sim.close()
    if mult > 1e30:
        assert not np.isfinite(want[1][:2, 1]).any()
    assert np.isfinite(want[1][:, [0, 2]]).all()
    for g, w in zip(got, want):
        assert np.array_equal(g, w, equal_nan=True)
        assert np.array_equal(np.signbit(g), np.signbit(w))
