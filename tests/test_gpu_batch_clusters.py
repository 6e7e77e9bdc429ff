"""Batches of meshes of one size: the blocks per mesh of the clustering follow
from the largest mesh's share (1, 2, 4 and 8 blocks), the trees do not."""
import numpy as np
import pytest

import rtbvh_gb300 as rb
from gpu_helpers import oracle_build, to_cuda, u32
from rtbvh_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("meshes,size", [(400, 4200), (150, 4200), (60, 4200), (12, 4200), (12, 20000), (3, 40001)])
def test_blocks_per_mesh(meshes, size):
    tris = scenes.incoherent(meshes * size, seed=meshes, median=0.05)
    off = np.arange(meshes + 1) * size
    rays, _ = scenes.incoherent_rays(meshes, seed=5)
    b = rb.Batch(to_cuda(tris), off, to_cuda(rays), np.arange(meshes + 1))
    b.run()
    assert b.status() == rb.ResultCode.Ok
    v = b.view()
    ints = rb.device_copy(v.nodes, (v.node_capacity, 8)).view(np.int32)
    for k in {0, 1, meshes // 2, meshes - 1}:
        o, base = int(off[k]), 2 * int(off[k]) - k
        on, _ = oracle_build(tris[o:o + size], "locb")
        want = on.copy()
        wi = want.view(np.int32)
        leaf = wi[:, 3] >= 0
        wi[leaf, 7] += o
        wi[~leaf, 7] += base
        assert np.array_equal(ints[base:base + len(on)].view(np.uint32), u32(want)), k
