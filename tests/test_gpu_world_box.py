"""World boxes (the Morton grid of a LOCB build) where their reduction changes
form: one block or many, and rows and runs of a batch that meshes share. The
box's extreme triangle is the first or the last, so a primitive left out or
counted into a neighbour moves every key."""
import numpy as np
import pytest

import rtbvh_gb300 as rb
from gpu_helpers import gpu_build, oracle_build, to_cuda, u32
from rtbvh_gb300 import scenes

pytestmark = pytest.mark.gpu


def _scene(n, end, seed=0):
    t = scenes.incoherent(n, seed=n + seed)
    t[-1 if end else 0] += np.float32(3.0 if end else -3.0)
    return t


@pytest.mark.parametrize("end", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 1023, 1024, 1025, 8191, 8192, 8193, 8449, 70001])
def test_one_mesh(n, end):
    tris = _scene(n, end)
    g = gpu_build(tris, "locb")
    on, oi = oracle_build(tris, "locb")
    assert np.array_equal(u32(g.nodes()), u32(on))
    assert np.array_equal(g.indices(), oi)


@pytest.mark.parametrize("sizes", [[1] * 70 + [2, 3] * 40, [31, 1, 32, 32, 1, 33, 63, 65], [256, 256, 255, 1, 257, 300, 2048, 511],
                                   [9000, 7, 5000, 1, 1, 1, 20000]])
def test_batches(sizes):
    off = np.concatenate([[0], np.cumsum(sizes)])
    parts = [_scene(n, k & 1, seed=k) for k, n in enumerate(sizes)]
    rays, _ = scenes.incoherent_rays(len(sizes), seed=5)
    b = rb.Batch(to_cuda(np.concatenate(parts)), off, to_cuda(rays), np.arange(len(sizes) + 1))
    for _ in range(2):
        b.run()
        assert b.status() == rb.ResultCode.Ok
        v = b.view()
        idx = rb.device_copy(v.indices, (int(off[-1]),), np.uint32)
        for k, part in enumerate(parts):
            assert np.array_equal(idx[off[k]:off[k + 1]], oracle_build(part, "locb")[1] + off[k]), k
