"""sph_upload_device predicts the next step's first substep in the import, as
pinned host uploads do. Whatever happens between the upload and the step --
nothing, another dt, a setting, a second upload -- and for rows that are not
16-byte aligned (the plain import), the step gives what a host upload of the
same rows gives, bit for bit; densities read before a step are zero."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("between", ["nothing", "dt", "setting", "again"])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [1, 33, 1031, 4096])
def test_device_upload_equals_host_upload(gpu_lib, n, offset, between):
    import torch
    import fluidsim
    from fluidsim import scenes
    sc = scenes.batched_scenes(count=1, seed=n, lo=n, hi=n)[0]
    pos, vel = sc["pos"], sc["vel"]
    rng = np.random.default_rng(n)
    other = (pos + rng.uniform(-0.02, 0.02, pos.shape)).astype(np.float32)

    def device_rows(a):
        flat = torch.zeros(3 * n + offset, dtype=torch.float32, device="cuda")
        flat[offset:] = torch.from_numpy(a.reshape(-1)).cuda()
        return flat[offset:]

    def run(on_device):
        sim = fluidsim.FluidSimulation(sc["params"])
        sim.InitializeData(n, pos, vel)
        sim.Update(sc["dt"], 3)
        rows = [device_rows(a) for a in (other, vel, pos)]
        torch.cuda.synchronize()

        def upload(k, a):
            if on_device:
                assert gpu_lib.sph_upload_device(
                    sim.handle, ctypes.c_void_p(rows[k].data_ptr()),
                    ctypes.c_void_p(rows[1].data_ptr()), None) == 0
            else:
                sim.upload(a, vel)
        if between == "again":
            upload(2, pos)
        upload(0, other)
        assert not sim.download()[2].any()
        if between == "setting":
            sim.setGravityScale(3.0)
        dt = sc["dt"] * (0.5 if between == "dt" else 1.0)
        for _ in range(2):
            sim.Update(dt, 3)
        out = sim.download()
        assert sim.status() == 0
        sim.close()
        return out

    for a, b in zip(run(True), run(False)):
        assert np.array_equal(a, b)
