"""A device upload captured by the caller has not run when the next step is
called. Whether the graph is dropped, launched once, or launched again before
later steps with other rows in its buffers, every step gives what plain uploads
of the rows the engine then holds give, bit for bit."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RELAXED = 2


@pytest.mark.parametrize("use", ["dropped", "launched", "launched again"])
@pytest.mark.parametrize("n", [1000, 4096])  # the histogram cleared by a memset, by a kernel
def test_step_after_a_captured_upload(gpu_lib, n, use):
    import torch
    import fluidsim
    from fluidsim import scenes
    rt = ctypes.CDLL("libcudart.so.13")
    sc = scenes.batched_scenes(count=1, seed=n, lo=n, hi=n)[0]
    rng = np.random.default_rng(n)
    vel = sc["vel"]
    # other states: the particles in another order, so every stale key is wrong
    x, y, z = (sc["pos"][rng.permutation(n)] for _ in range(3))
    stream = torch.cuda.Stream()
    st = ctypes.c_void_p(stream.cuda_stream)

    def fresh():
        sim = fluidsim.FluidSimulation(sc["params"], stream=stream.cuda_stream)
        sim.InitializeData(n, sc["pos"], vel)
        sim.Update(sc["dt"], 2)
        sim.upload(x, vel)
        return sim

    ref = fresh()
    for rows in {"dropped": [], "launched": [y], "launched again": [y, z]}[use]:
        ref.upload(rows, vel)
        ref.Update(sc["dt"], 2)
    if use == "dropped":
        ref.Update(sc["dt"], 2)
    want = ref.download()
    ref.close()

    sim = fresh()
    dpos, dvel = torch.from_numpy(y).cuda(), torch.from_numpy(vel).cuda()
    torch.cuda.synchronize()
    graph, ex = ctypes.c_void_p(), ctypes.c_void_p()
    assert rt.cudaStreamBeginCapture(st, RELAXED) == 0
    assert gpu_lib.sph_upload_device(sim.handle, ctypes.c_void_p(dpos.data_ptr()),
                                     ctypes.c_void_p(dvel.data_ptr()), st) == 0
    assert rt.cudaStreamEndCapture(st, ctypes.byref(graph)) == 0
    assert rt.cudaGraphInstantiate(ctypes.byref(ex), graph, ctypes.c_ulonglong(0)) == 0
    if use != "dropped":
        assert rt.cudaGraphLaunch(ex, st) == 0
    sim.Update(sc["dt"], 2)
    if use == "launched again":
        torch.cuda.synchronize()
        dpos.copy_(torch.from_numpy(z))
        torch.cuda.synchronize()
        assert rt.cudaGraphLaunch(ex, st) == 0
        sim.Update(sc["dt"], 2)
    got = sim.download()
    assert sim.status() == 0
    sim.close()
    rt.cudaGraphExecDestroy(ex)
    rt.cudaGraphDestroy(graph)
    for g, w in zip(got, want):
        assert np.array_equal(g, w)
