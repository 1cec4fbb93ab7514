"""An error that another call left behind (here a refused cudaSetDevice, in the
runtime the library loaded) is not taken for a failure of the library's own
launches."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CALLS = ["first step", "step", "upload", "device upload", "download", "pinned download",
         "device download", "render", "lookup", "debug export", "batch step"]


@pytest.mark.parametrize("call", CALLS)
def test_call_after_an_error(gpu_lib, call):
    import torch
    import fluidsim
    from fluidsim import render, scenes
    rt = ctypes.CDLL("libcudart.so.13")
    n = 2000
    sc = scenes.batched_scenes(count=1, seed=4, lo=n, hi=n)[0]
    sim = fluidsim.FluidSimulation(sc["params"])
    sim.InitializeData(n, sc["pos"], sc["vel"])
    b = fluidsim.Batch(n, 1)
    b.add(sc["params"], sc["pos"], sc["vel"], sc["dt"])
    dev = [torch.from_numpy(sc[k]).cuda() for k in ("pos", "vel")]
    out = [torch.zeros((n, k), device="cuda") for k in (3, 3, 2)]
    pinned = [torch.zeros((n, k), pin_memory=True) for k in (3, 3, 2)]
    ints = [torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(4)]

    def ptrs(ts):
        return [ctypes.c_void_p(t.data_ptr()) for t in ts]

    if call != "first step":
        if call == "debug export":
            sim.debug_enable()
        sim.Update(sc["dt"], 1)
    torch.cuda.synchronize()
    assert rt.cudaSetDevice(9999) != 0
    try:
        if call in ("first step", "step"):
            sim.Update(sc["dt"], 1)
        elif call == "upload":
            sim.upload(sc["pos"], sc["vel"])
        elif call == "device upload":
            assert gpu_lib.sph_upload_device(sim.handle, *ptrs(dev), None) == 0
        elif call == "download":
            sim.download()
        elif call == "pinned download":
            assert gpu_lib.sph_download(sim.handle, *ptrs(pinned), None) == 0
        elif call == "device download":
            assert gpu_lib.sph_download_device(sim.handle, *ptrs(out), None) == 0
        elif call == "render":
            sim.render(render.view((2.0, 3.0, 9.0), (0.0, 0.0, 0.0), 64, 48))
        elif call == "lookup":
            assert gpu_lib.sph_spatial_lookup_static(
                ptrs(dev)[0], n, ctypes.c_float(0.35), *ptrs(ints), None) == 0
        elif call == "debug export":
            sim.debug_export()
            sim.debug_export_layout()
        else:
            b.step(2)
    finally:
        rt.cudaGetLastError()
    assert np.isfinite(sim.download()[0]).all()
    sim.close()
    b.close()
