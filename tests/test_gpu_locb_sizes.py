"""LOCB builds around the sizes where the clustering changes form: the last
128 nodes in one block, 2048 nodes per block of a cluster, and the levels in
global memory above that; single meshes and batches against the oracle."""
import numpy as np
import pytest

import oracle
import rtbvh_gb300 as rb
from gpu_helpers import gpu_build, oracle_build, to_cuda, u32
from rtbvh_gb300 import scenes

pytestmark = pytest.mark.gpu

SIZES = [3, 4, 15, 28, 29, 30, 57, 127, 128, 129, 130, 156, 200, 255, 300, 1000, 2047, 2048, 2049, 4097, 16385, 32767,
         32768, 32769, 33000, 70001]


def _scene(n, kind):
    if kind == "soup":
        return scenes.incoherent(n, seed=n)
    t = np.repeat(scenes.incoherent(max(1, n // 7), seed=n), 8, axis=0)[:n]  # equal boxes: ties everywhere
    return np.concatenate([t, t[: n - len(t)]]) if len(t) < n else t


@pytest.mark.parametrize("kind", ["soup", "ties"])
@pytest.mark.parametrize("n", SIZES)
def test_locb_sizes(n, kind):
    tris = _scene(n, kind)
    g = gpu_build(tris, "locb")
    on, oi = oracle_build(tris, "locb")
    assert np.array_equal(u32(g.nodes()), u32(on))
    assert np.array_equal(g.indices(), oi)


@pytest.mark.parametrize("cluster_min", [2048, 65536])
def test_locb_sizes_in_a_batch(cluster_min):
    sizes = [n for n in SIZES if n != 70001] + [1, 2, 40000]
    off = np.concatenate([[0], np.cumsum(sizes)])
    parts = [_scene(n, "ties" if k % 3 == 0 else "soup") for k, n in enumerate(sizes)]
    tris = np.concatenate(parts)
    rays, _ = scenes.incoherent_rays(64 * len(sizes), seed=5)
    b = rb.Batch(to_cuda(tris), off, to_cuda(rays), np.arange(len(sizes) + 1) * 64)
    b.set_tuning(cluster_min_prims=cluster_min)
    b.run()
    assert b.status() == rb.ResultCode.Ok
    v = b.view()
    nodes = rb.device_copy(v.nodes, (v.node_capacity, 8))
    ints = nodes.view(np.int32)
    for k, n in enumerate(sizes):
        base, o = 2 * int(off[k]) - k, int(off[k])
        on, _ = oracle_build(parts[k], "locb")
        want = on.copy()
        wi = want.view(np.int32)
        leaf = wi[:, 3] >= 0
        wi[leaf, 7] += o
        wi[~leaf, 7] += base
        got = ints[base:base + len(on)]
        assert np.array_equal(got.view(np.uint32), u32(want)), n


@pytest.mark.parametrize("n", [1000000, 1000001])
def test_locb_at_a_million(n):
    """More blocks per SM above a million primitives."""
    tris = _scene(n, "soup")
    g = gpu_build(tris, "locb")
    on, oi = oracle_build(tris, "locb")
    assert np.array_equal(u32(g.nodes()), u32(on))
    assert np.array_equal(g.indices(), oi)
