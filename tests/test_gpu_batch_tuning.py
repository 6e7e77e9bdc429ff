"""The threshold above which a batch's meshes get a thread-block cluster: the
default follows the batch, and every size that is asked for is taken as it
is."""
import numpy as np
import pytest
import torch

import rtbvh_gb300 as rb
from gpu_helpers import to_cuda
from rtbvh_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("meshes,size", [(400, 4200), (12, 4200)])
def test_cluster_threshold(meshes, size):
    tris = scenes.incoherent(meshes * size, seed=meshes, median=0.05)
    rays, _ = scenes.incoherent_rays(64 * meshes, seed=5)
    b = rb.Batch(to_cuda(tris), np.arange(meshes + 1) * size, to_cuda(rays), np.arange(meshes + 1) * 64)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    default = max(4096, meshes * size * 10 // (14 * sms))
    assert (default > 4096) == (meshes == 400)
    assert b.tuning["cluster_min_prims"] == default
    want = b.run().clone()
    for asked, got in ((4096, 4096), (4095, 4095), (0, default), (default, default), (2, 2)):
        b.set_tuning(cluster_min_prims=asked)
        assert b.tuning["cluster_min_prims"] == got
        assert torch.equal(b.run().view(torch.int32), want.view(torch.int32))
    assert b.status() == rb.ResultCode.Ok
    chosen = b.tune()["cluster_min_prims"]
    assert chosen in (default, 2048, 4096, 8192, 16384, 65536)
    assert b.tuning["cluster_min_prims"] == chosen
