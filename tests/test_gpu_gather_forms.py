"""The plain force kernels under every gather batch, with one and two lanes a
particle, on full and overflowing lists. Small launches choose batches of their
own, so the dense scene steps beside a filler of a size whose launches take the
batch that is asked for: more tiles than one wave of the densest form, and a
wave more at the registers of three entries than at those of two. A batch only
changes which loads are in flight: the bits are those of batches of two, and
with one lane those of the scene alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("table", [0, 1])
@pytest.mark.parametrize("lanes", [32, 16])
def test_gathers_bit_equal(gpu_lib, lanes, table):
    import torch
    import fluidsim
    from fluidsim import scenes
    from test_gpu_wide_lists import dense_scene
    sc = dense_scene()
    n = sc["pos"].shape[0]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    fill = 72 * 32 * sms - n  # 72 warps an SM: two waves of 40 or 48, three of 32
    fpos, fvel, bound = scenes.fill_box_scene(np.random.default_rng(9), fill, 0.5,
                                              (1.0, 1.0, 1.0))
    filler = scenes.SimParams(radius=0.35, bound=bound, **scenes.DAM_CONSTANTS)
    outs = {}
    for gather in (2, 3, 4, 8):
        b = fluidsim.Batch(fill + n, 2)
        b.set_tuning(gather=gather, particles_per_warp=lanes, table=table)
        b.add(filler, fpos, fvel, sc["dt"])
        sid = b.add(sc["params"], sc["pos"], sc["vel"], sc["dt"])
        for _ in range(2):
            b.step(2)
        assert b.status() == 0
        outs[gather] = b.download(sid)
        b.close()
    if lanes == 32:
        sim = fluidsim.FluidSimulation(sc["params"])
        sim.InitializeData(n, sc["pos"], sc["vel"])
        sim.set_tuning(table=table)
        for _ in range(2):
            sim.Update(sc["dt"], 2)
        outs["alone"] = sim.download()
        sim.close()
    for key, out in outs.items():
        for g, w in zip(out, outs[2]):
            assert np.array_equal(g, w), key
