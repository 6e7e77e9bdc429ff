"""LOCB builds of the exact sizes where the last levels change hands: up to 32
nodes one warp's, up to 256 one block's, above that the cluster's."""
import numpy as np
import pytest

import rtbvh_gb300 as rb
from gpu_helpers import gpu_build, oracle_build, to_cuda, u32
from rtbvh_gb300 import scenes
from test_gpu_locb_sizes import _scene

pytestmark = pytest.mark.gpu

SIZES = [31, 32, 33, 34, 63, 64, 65, 254, 256, 257, 258, 511, 512, 513]


@pytest.mark.parametrize("kind", ["soup", "ties"])
@pytest.mark.parametrize("n", SIZES)
def test_locb_edges(n, kind):
    tris = _scene(n, kind)
    g = gpu_build(tris, "locb")
    on, oi = oracle_build(tris, "locb")
    assert np.array_equal(u32(g.nodes()), u32(on))
    assert np.array_equal(g.indices(), oi)


@pytest.mark.parametrize("cluster_min", [2, 65536])
def test_locb_edges_in_a_batch(cluster_min):
    off = np.concatenate([[0], np.cumsum(SIZES)])
    parts = [_scene(n, "ties" if k % 2 else "soup") for k, n in enumerate(SIZES)]
    rays, _ = scenes.incoherent_rays(len(SIZES), seed=5)
    b = rb.Batch(to_cuda(np.concatenate(parts)), off, to_cuda(rays), np.arange(len(SIZES) + 1))
    b.set_tuning(cluster_min_prims=cluster_min)
    b.run()
    assert b.status() == rb.ResultCode.Ok
    v = b.view()
    ints = rb.device_copy(v.nodes, (v.node_capacity, 8)).view(np.int32)
    for k, n in enumerate(SIZES):
        o, base = int(off[k]), 2 * int(off[k]) - k
        want = oracle_build(parts[k], "locb")[0].copy()
        wi = want.view(np.int32)
        leaf = wi[:, 3] >= 0
        wi[leaf, 7] += o
        wi[~leaf, 7] += base
        assert np.array_equal(ints[base:base + len(want)].view(np.uint32), u32(want)), n
