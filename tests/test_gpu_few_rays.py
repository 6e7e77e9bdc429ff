"""Small launches walk with four lanes per ray: the same hits, bit for bit, as
the walks with one lane per ray that large launches take (a batch padded
beyond the threshold with more rays)."""
import numpy as np
import pytest
import torch

import rtbvh_gb300 as rb
from gpu_helpers import gpu_build, scene, to_cuda, u32
from rtbvh_gb300 import scenes

pytestmark = pytest.mark.gpu

LARGE = 200000  # more rays than any small launch


def _rays(tris, n, seed):
    rng = np.random.default_rng(seed)
    lo, hi = tris.reshape(-1, 3).min(0), tris.reshape(-1, 3).max(0)
    c = tris.mean(axis=1)[rng.integers(0, len(tris), n)].astype(np.float64)
    o = np.where(rng.random((n, 1)) < 0.5, rng.uniform(lo, hi, size=(n, 3)),
                 c + (hi - lo).max() * rng.normal(size=(n, 3)))
    d = c - o
    d[: n // 4] = rng.normal(size=(n // 4, 3))
    d /= np.maximum(np.linalg.norm(d, axis=1, keepdims=True), 1e-30)
    d[::41, 2] = 0.0  # non-finite inverses
    o[::97] *= 1e4  # beyond the compact walk's range
    return np.concatenate([o, d], 1).astype(np.float32), rng.uniform(0.05, 4.0, n).astype(np.float32)


MODES = [{}, {"exact_nodes": True}, {"any_hit": True}, {"any_hit": True, "exact_nodes": True}]


@pytest.mark.parametrize("mode", MODES, ids=["closest", "closest_exact", "any", "any_exact"])
@pytest.mark.parametrize("name,kind,scale", [("sphere", "sah", 1.0), ("teapot", "sah", 1.0), ("incoherent_20k", "locb", 1.0),
                                             ("sphere", "locb", 200.0), ("slivers", "sah", 1.0), ("slivers", "spatial", 1.0)])
def test_small_launches_equal_large_ones(name, kind, scale, mode):
    tris = scenes.slivers(3000) if name == "slivers" else scene(name)
    tris = (tris * np.float32(scale)).astype(np.float32)
    if kind == "spatial":
        g = rb.Builder(primitives=rb.Triangles(to_cuda(tris))).construct_spatial_sah(fixes=31)
    else:
        g = gpu_build(tris, kind)
    m = rb.Mbvh.construct(g)
    rays, t_max = _rays(tris, LARGE, 5)
    r, tm = to_cuda(rays), to_cuda(t_max)
    for limit in (None, tm):
        want = m.intersect(r, t_max=limit, **mode)[0].cpu().numpy()
        for first, count in ((0, 1), (1, 2), (3, 7), (10, 129), (200, 4097), (5000, 30011)):
            part = None if limit is None else limit[first:first + count].contiguous()
            got = m.intersect(r[first:first + count].contiguous(), t_max=part, **mode)[0].cpu().numpy()
            assert np.array_equal(u32(got), u32(want[first:first + count])), (first, count)
    assert m.status() == rb.ResultCode.Ok
    assert (rb.hit_prims(want) >= 0).any()


@pytest.mark.parametrize("step,count", [(35, 700001), (20, 700001), (35, 500001), (35, 8000003), (35, 10000019)])
def test_handed_on_rays_of_large_launches(step, count):
    """Rays that the compact walk hands on (about 3 % and every step-th), on
    both sides of the lines between four lanes and one: 1/16 of the launch,
    32,768 rays, 524,288 rays. The exact walk is theirs, bit for bit."""
    tris = scene("sphere")
    m = rb.Mbvh.construct(gpu_build(tris, "sah"))
    rays, _ = _rays(tris, 500001, 6)
    rays[::97, :3] *= np.float32(1e-4)  # back within range
    rays[:, :3] = np.clip(rays[:, :3], -100, 100)
    r = to_cuda(rays)[torch.arange(count, device="cuda") % 500001]
    r[::step, :3] += 300.0 * r[::step, 3:]  # beyond it
    got, work = m.intersect(r, walk_stats=True)
    handed = work[:, 2] > 0
    n = int(handed.sum())
    assert (n <= count // 16) == (step == 35) and (n > 32768) == (count > 600000) and (n > 524288) == (count > 9000000)
    want = m.intersect(r, exact_nodes=True)[0]
    assert torch.equal(got[handed].view(torch.int32), want[handed].view(torch.int32))
    # the others may take another of two triangles at the same t
    assert torch.equal(got[:, 0].view(torch.int32), want[:, 0].view(torch.int32))
    assert m.status() == rb.ResultCode.Ok


def test_small_batch_of_meshes():
    sizes = [1, 2, 300, 5000, 3]
    off = np.concatenate([[0], np.cumsum(sizes)])
    tris = scenes.incoherent(int(off[-1]), seed=9, median=0.1)
    roff = np.array([0, 70, 140, 5000, 15001, 15003])
    rays, _ = scenes.incoherent_rays(int(roff[-1]), seed=10)
    for any_hit in (False, True):
        b = rb.Batch(to_cuda(tris), off, to_cuda(rays), roff, any_hit=any_hit)
        got = b.run().clone()
        b.set_tuning(trace_ray_batch=32)  # an asked-for launch shape: one lane per ray
        assert torch.equal(got.view(torch.int32), b.run().view(torch.int32))
        assert b.status() == rb.ResultCode.Ok
