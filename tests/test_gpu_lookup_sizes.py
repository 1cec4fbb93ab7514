"""sph_spatial_lookup_static at the edges of its sorting passes: rounds of 32
entries a warp, 8,192 entries a round of the cluster, the largest size; keys
that differ in the low byte, the high byte, both or not at all."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [0.1, 1.5, 60.0])
@pytest.mark.parametrize("n", [1, 31, 33, 255, 1025, 8191, 8192, 8193, 20000, 65535, 65536])
def test_lookup_sizes(gpu_lib, oracle_mod, n, side):
    import torch
    from oracle import layout
    rng = np.random.default_rng(n)
    pred = rng.uniform(-side, side, (n, 3)).astype(np.float32)
    want = layout.reference_lookup(pred, np.float32(0.35))
    d = torch.from_numpy(pred).cuda()
    outs = [torch.full((n,), -1, dtype=torch.int32, device="cuda") for _ in range(4)]
    for _ in range(2):  # the second call finds the first one's working memory
        rc = gpu_lib.sph_spatial_lookup_static(
            ctypes.c_void_p(d.data_ptr()), n, ctypes.c_float(0.35),
            *[ctypes.c_void_p(o.data_ptr()) for o in outs],
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0
    torch.cuda.synchronize()
    for o, k in zip(outs, ("hash", "key", "sorted_ids", "start")):
        assert np.array_equal(o.cpu().numpy().view(np.uint32), want[k]), k
