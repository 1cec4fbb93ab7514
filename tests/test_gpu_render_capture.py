"""A render into a stream that is being captured is refused, and its kernels
never run: the next frame must start from a cleared key buffer, whether the
refused call had to grow the buffers or not."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RELAXED = 2


@pytest.mark.parametrize("first", [None, (64, 48), (200, 100)])
def test_frame_after_a_refused_capture(gpu_lib, first):
    import torch
    import fluidsim
    from fluidsim import render, scenes
    rt = ctypes.CDLL("libcudart.so.13")
    sc = scenes.dam_break_16k()

    def fresh(stream=None):
        sim = fluidsim.FluidSimulation(sc["params"], stream=stream)
        sim.InitializeData(sc["pos"].shape[0], sc["pos"], sc["vel"])
        return sim

    def view(size):
        return render.view((2.0, 3.0, 9.0), (-2.0, -1.5, -1.0), *size)

    ref = fresh()
    want = ref.render(view((200, 100)))
    ref.close()
    stream = torch.cuda.Stream()
    sim = fresh(stream.cuda_stream)
    if first:
        sim.render(view(first))
    torch.cuda.synchronize()
    v = view((200, 100))
    img = np.empty((100, 200, 4), np.uint8)
    st = ctypes.c_void_p(stream.cuda_stream)
    assert rt.cudaStreamBeginCapture(st, RELAXED) == 0
    rc = gpu_lib.sph_render(sim.handle, ctypes.byref(v), ctypes.c_void_p(img.ctypes.data),
                            None, st)
    graph = ctypes.c_void_p()
    ended = rt.cudaStreamEndCapture(st, ctypes.byref(graph))
    rt.cudaGetLastError()
    assert rc != 0 and ended != 0
    got = sim.render(v)
    sim.close()
    assert (want[1] < 1.0).sum() > 100
    for g, w in zip(got, want):
        assert np.array_equal(g, w)
