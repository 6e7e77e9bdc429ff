"""Closest hits of the compact walk over the whole range of its slab
arithmetic: scenes near both ends of the coordinate range, directions whose
inverses reach the largest the walk takes, t_max from zero up -- against the
walk over the exact nodes."""
import numpy as np
import pytest

import rtbvh_gb300 as rb
from gpu_helpers import assert_same_nearest, gpu_build, to_cuda
from rtbvh_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["locb", "sah"])
@pytest.mark.parametrize("scale", [0.05, 1.0, 60.0, 127.0])
def test_compact_walk_at_the_ends_of_its_range(scale, kind):
    tris = (scenes.incoherent(6000, seed=71, median=0.03) * np.float32(scale)).astype(np.float32)
    tris = np.clip(tris, 0.0, 127.9).astype(np.float32)
    m = rb.Mbvh.construct(gpu_build(tris, kind))
    rng = np.random.default_rng(72)
    n = 65537
    c = tris.mean(axis=1)[rng.integers(0, len(tris), n)].astype(np.float64)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    axis = rng.integers(0, 3, n)
    small = rng.random(n) < 0.5
    d[small, axis[small]] = (10.0 ** -rng.uniform(3.0, 17.9, n) * rng.choice([-1.0, 1.0], n))[small]
    o = c - d * rng.uniform(0.0, 0.5 * scale, (n, 1))
    rays = np.concatenate([o, d], 1).astype(np.float32)
    t_max = (scale * 10.0 ** rng.uniform(-6.0, 1.0, n)).astype(np.float32)
    t_max[::31] = 0.0
    t_max[1::31] = np.float32(1e-30)
    t_max[2::31] = np.inf
    for limit in (None, to_cuda(t_max)):
        hits = m.intersect(to_cuda(rays), t_max=limit)[0].cpu().numpy()
        exact = m.intersect(to_cuda(rays), t_max=limit, exact_nodes=True)[0].cpu().numpy()
        assert_same_nearest(hits, exact, tris, rays)
    assert m.status() == rb.ResultCode.Ok
    assert (rb.hit_prims(hits) >= 0).sum() > n // 50
