"""sph_spatial_lookup_static of up to 512 particles takes one block: sizes at the
edges of its warps and of its last group of four entries, to the largest and one
past it, with keys all alike, mixed and mostly apart."""
import pytest

import test_gpu_lookup_sizes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [0.1, 1.5, 60.0])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 31, 32, 33, 34, 127, 129, 500, 509, 511, 512, 513])
def test_small_lookups(gpu_lib, oracle_mod, n, side):
    test_gpu_lookup_sizes.test_lookup_sizes(gpu_lib, oracle_mod, n, side)
