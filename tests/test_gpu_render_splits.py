"""The threads a splat is drawn by follow the image's pixels per particle: at
sizes of each rule's range (1, 2, 4, 8 threads, a warp), with a camera beside
the fluid and one within it (splats of many rows, near clipping), the image and
the depth match the oracle's bit for bit."""
import numpy as np
import pytest

from fluidsim import render

pytestmark = pytest.mark.gpu

# 1, 3.8, 12, 30 and 210 pixels a particle at 1,000 particles
SIZES = [(33, 31), (64, 60), (110, 110), (200, 151), (500, 421)]


@pytest.fixture(scope="module")
def scene_1k(gpu_lib):
    import fluidsim
    from fluidsim import scenes
    sc = scenes.batched_scenes(count=1, seed=21, lo=1000, hi=1000)[0]
    sim = fluidsim.FluidSimulation(sc["params"])
    sim.InitializeData(sc["pos"].shape[0], sc["pos"], sc["vel"])
    for _ in range(6):
        sim.Update(sc["dt"], 3)
    yield sim, sc["params"].bound
    sim.close()


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("near", [False, True])
def test_split_splats_match_oracle(scene_1k, oracle_mod, size, near):
    sim, bound = scene_1k
    assert sim.download()[0].shape[0] == 1000
    pos, vel, _ = sim.download()
    middle = pos.mean(0)
    eye = middle + (np.float32(0.1) if near else np.asarray(bound, np.float32))
    v = render.view(tuple(map(float, eye)), tuple(map(float, middle - eye)), *size)
    img, depth = sim.render(v)
    want_img, want_depth = oracle_mod.render(pos, vel, v)
    assert (want_depth < 1.0).any()
    assert np.array_equal(depth, want_depth)
    assert np.array_equal(img, want_img)
