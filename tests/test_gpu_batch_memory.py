"""The device memory a batch takes per particle is what the server's split of a
budget counts with."""
import gc

import pytest

from amsc_b200 import serving
from amsc_b200.batch import Batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,per_particle", [("fp64", serving.BYTES_PER_PARTICLE),
                                                    ("fp32", serving.BYTES_PER_PARTICLE_F32)])
def test_bytes_per_particle(cuda_lib, precision, per_particle):
    import torch
    gc.collect()

    def taken(cap):
        # (capacities at which every array is a multiple of the driver's 2 MB)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        with Batch(cap, 1 << 20, 4, precision=precision):
            return free - torch.cuda.mem_get_info()[0]

    taken(1 << 20)
    small, large = 1 << 22, 1 << 24
    slope = (taken(large) - taken(small)) / (large - small)
    assert 0.9 * per_particle < slope < 1.01 * per_particle
