"""The reorder of grid tables ranks by particle index alone, that of bucket tables
by (cell, index), and only the latter writes the cell arrays: scenes whose cells
hold from one to hundreds of particles (cells ending on, before and behind a
tile's edge, cells filling several tiles) give the same result bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_cell", [1, 5, 16, 17, 33, 48, 64, 65, 300])
@pytest.mark.parametrize("count", [1, 3])
def test_grid_order_equals_bucket_order(gpu_lib, per_cell, count):
    import fluidsim
    from fluidsim import scenes
    rng = np.random.default_rng(per_cell)
    p = scenes.SimParams(radius=0.35, bound=(6.0, 6.0, 6.0), **scenes.DAM_CONSTANTS)
    cells = np.stack(np.meshgrid(*[np.arange(-3, 3)] * 3), -1).reshape(-1, 3)[:max(2, 6000 // per_cell)]
    outs = []
    scs = []
    for k in range(count):  # about per_cell particles a cell, in shuffled order
        at = np.repeat(cells, per_cell, 0)[: len(cells) * per_cell - k]
        pos = ((at + rng.uniform(0.05, 0.95, at.shape)) * 0.35).astype(np.float32)
        rng.shuffle(pos)
        scs.append((pos, rng.uniform(-0.5, 0.5, pos.shape).astype(np.float32)))
    for table in (1, 2):
        b = fluidsim.Batch(sum(s[0].shape[0] for s in scs), count)
        b.set_tuning(table=table)
        ids = [b.add(p, pos, vel, 1.0 / 240.0) for pos, vel in scs]
        for _ in range(2):
            b.step(2)
        assert b.status() == 0
        outs.append([x for sid in ids for x in b.download(sid)])
        b.close()
    for a, c in zip(*outs):
        assert np.array_equal(a, c)
