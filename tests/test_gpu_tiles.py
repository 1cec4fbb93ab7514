"""The tile tables a layout change writes on the device: scenes of sizes around
a tile's 32 slots, with removed scenes between live ones and more scenes than
one launch's parameters hold, step bit for bit as each does alone."""
import numpy as np
import pytest

from test_gpu_batch import alone

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 32, 33, 64, 65, 127, 500]


@pytest.mark.parametrize("count", [1, 2, 9, 300])
def test_layout_changes_match_scenes_alone(gpu_lib, count):
    import fluidsim
    from fluidsim import scenes
    pool = scenes.batched_scenes(count=8, seed=3, lo=500, hi=900)

    def scene(k):
        s = dict(pool[k % 8])
        n = SIZES[(3 * k) % 8]
        s["pos"], s["vel"] = s["pos"][:n].copy(), s["vel"][:n].copy()
        return s

    b = fluidsim.Batch(2 * count * max(SIZES), 2 * count)
    live = {}
    for k in range(count):
        s = scene(k)
        live[b.add(s["params"], s["pos"], s["vel"], s["dt"])] = (s, 2)
    b.step(2)
    for sid in list(live)[1::3]:  # holes between live scenes
        b.remove(sid)
        del live[sid]
    for k in range(count // 4 + 1):  # and scenes that fill some of them
        s = scene(k + 5)
        live[b.add(s["params"], s["pos"], s["vel"], s["dt"])] = (s, 1)
    b.step(2)
    assert b.status() == 0
    ids = sorted(live)
    for sid in ids[:6] + ids[-6:]:
        s, steps = live[sid]
        for g, r in zip(b.download(sid), alone(s, steps, substeps=2)):
            assert np.array_equal(g, r)
    b.close()
