"""Neighbour lists of slots past 2^26 lie beyond 2^32 entries (64 a slot). A dense
scene (lists that fill and overflow) behind fillers that take the slots before
it must step bit for bit as alone. The engine holds about 47 GB of HBM."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LARGEST = 2**24 - 1  # particles a scene may have
FILLERS = 4


def test_lists_past_2_32(gpu_lib):
    import fluidsim
    from fluidsim import scenes
    from test_gpu_wide_lists import dense_scene
    sc = dense_scene()
    n = sc["pos"].shape[0]
    assert (FILLERS * LARGEST + n - 1) * 64 > 2**32
    sim = fluidsim.FluidSimulation(sc["params"])
    sim.InitializeData(n, sc["pos"], sc["vel"])
    for _ in range(2):
        sim.Update(sc["dt"], 1)
    want = sim.download()
    sim.close()
    # about 1.4 neighbours a particle: their lists use the first entries of a slot
    bound = 0.5 * np.ceil(np.cbrt(LARGEST))
    rng = np.random.default_rng(17)
    pos = (rng.random((LARGEST, 3), dtype=np.float32) - np.float32(0.5)) * np.float32(0.98 * bound)
    filler = scenes.SimParams(radius=0.35, bound=(bound,) * 3, **scenes.DAM_CONSTANTS)
    b = fluidsim.Batch(FILLERS * LARGEST + n, FILLERS + 1)
    for _ in range(FILLERS):
        b.add(filler, pos, np.zeros_like(pos), sc["dt"])
    sid = b.add(sc["params"], sc["pos"], sc["vel"], sc["dt"])
    for _ in range(2):
        b.step(1)
    assert b.status() == 0
    got = b.download(sid)
    b.close()
    for g, w in zip(got, want):
        assert np.array_equal(g, w)
