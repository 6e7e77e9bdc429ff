"""Any hit on grazing rays: nearly in a triangle's plane its determinant is just
above the test's 1e-5, t, u and v are rounding noise, and the reference accepts
the triangle although its grown box lies wholly behind the ray's origin. The
walks that skip slots report those hits too, bit for bit."""
import numpy as np
import pytest

import oracle
import rtbvh_gb300 as rb
from gpu_helpers import gpu_build, oracle_build, to_cuda, u32

pytestmark = pytest.mark.gpu


def _cross(a, b):
    """a x b with float32 roundings, products and differences one by one."""
    return np.stack([a[:, 1] * b[:, 2] - b[:, 1] * a[:, 2], a[:, 2] * b[:, 0] - b[:, 2] * a[:, 0],
                     a[:, 0] * b[:, 1] - b[:, 0] * a[:, 1]], 1)


def _dot(a, b):
    return (a[:, 0] * b[:, 0] + a[:, 1] * b[:, 1]) + a[:, 2] * b[:, 2]


def accepted_behind(tris, rays):
    """Rays whose triangle the reference's test accepts (float32, unbounded)
    while the slab test passes its box grown by 1e-4 with an exit t below 0."""
    with np.errstate(all="ignore"):
        o, d = rays[:, :3], rays[:, 3:]
        e1, e2 = tris[:, 1] - tris[:, 0], tris[:, 2] - tris[:, 0]
        h = _cross(d, e2)
        det = _dot(e1, h)
        f = np.float32(1.0) / det
        s = o - tris[:, 0]
        u = f * _dot(s, h)
        q = _cross(s, e1)
        v = f * _dot(d, q)
        t = f * _dot(e2, q)
        ok = (np.abs(det) >= np.float32(1e-5)) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1)
        ok &= (t > np.float32(1e-4)) & (t < np.float32(1e34))
        inv = np.float32(1.0) / d
        t0 = (tris.min(1) - np.float32(1e-4) - o) * inv
        t1 = (tris.max(1) + np.float32(1e-4) - o) * inv
        near, far = np.minimum(t0, t1).max(1), np.maximum(t0, t1).min(1)
        return ok & np.isfinite(inv).all(1) & (far >= near) & (far < 0)


def grazing(lo, hi, reach, n, seed, large=0):
    """48 scattered triangles with edges in [lo, hi], the first `large` of them
    ten times that size, and rays of the kind above: past a border point of a
    triangle, `reach` of its size beyond it at most, directions with
    determinants of 1e-5 to 3e-5."""
    rng = np.random.default_rng(seed)
    c = rng.uniform(-3.0 * hi, 3.0 * hi, (48, 1, 3))
    size = np.where(np.arange(48) < large, 10.0, 1.0)[:, None, None] * rng.uniform(lo, hi, (48, 3, 1))
    tris = (c + size * rng.normal(size=(48, 3, 3))).clip(-100.0, 100.0).astype(np.float32)
    k = rng.integers(0, 48, n)
    t = tris[k].astype(np.float64)
    e1, e2 = t[:, 1] - t[:, 0], t[:, 2] - t[:, 0]
    nrm = np.cross(e1, e2)
    area = np.linalg.norm(nrm, axis=1, keepdims=True)
    w = rng.dirichlet((1.0, 1.0, 1.0), n)
    edge = rng.random(n) < 0.7
    w[edge, rng.integers(0, 3, edge.sum())] = 0.0
    w /= w.sum(1, keepdims=True)
    p = (t * w[:, :, None]).sum(1)
    a = rng.uniform(0.0, 2.0 * np.pi, (n, 1))
    e = e1 / np.linalg.norm(e1, axis=1, keepdims=True)
    d = np.cos(a) * e + np.sin(a) * np.cross(nrm / area, e)
    d += rng.uniform(1.0, 3.0, (n, 1)) * rng.choice([-1.0, 1.0], (n, 1)) * 1e-5 / area * nrm / area
    far = reach * np.sqrt(area) * rng.random((n, 1)) ** 3
    rays = np.concatenate([p + far * d, d], 1).astype(np.float32)
    bad = accepted_behind(tris[k], rays)
    return tris, rays[bad], int(bad.sum())


@pytest.mark.parametrize("few", [True, False])
@pytest.mark.parametrize("kind", ["locb", "sah"])
@pytest.mark.parametrize("lo,hi,reach,large", [(0.3, 0.5, 0.001, 0), (0.5, 1.5, 0.01, 0), (2.0, 5.0, 0.1, 0), (8.0, 20.0, 1.0, 0),
                                               (0.2, 0.4, 0.1, 5), (0.2, 0.4, 0.1, 9)])
def test_grazing_any_hits_equal_the_walk_without_skips(lo, hi, reach, large, kind, few):
    """Scenes in which every triangle, all but a few or only some are small
    enough for the walks to skip slots."""
    tris, rays, bad = grazing(lo, hi, reach, 2000000 if hi < 1.0 else 400000, seed=11, large=large)
    assert bad >= 5
    if not few:  # more rays than small launches take
        rays = np.tile(rays, (70000 // len(rays) + 1, 1))
    m = rb.Mbvh.construct(gpu_build(tris, kind))
    r = to_cuda(rays)
    got = m.intersect(r, any_hit=True)[0].cpu().numpy()
    want = m.intersect(r, any_hit=True, exact_nodes=True)[0].cpu().numpy()
    assert np.array_equal(u32(got), u32(want))
    assert m.status() == rb.ResultCode.Ok


def test_one_grazed_triangle():
    """The oracle's hit at t = 0.0048 although the box ends at t = -0.0024."""
    tris = np.array([[[0.52354699, 1.79714823, -1.66983688], [0.25733528, 0.85064638, -0.58718336],
                      [-0.66274583, 0.56335968, -0.72492296]]], np.float32)
    rays = np.array([[-0.66169465, 0.56217307, -0.72279632, 0.40016645, -0.44511086, 0.80108875]], np.float32)
    on, oi = oracle_build(tris, "locb")
    want = oracle.trace("mbvh", oracle.mbvh(on), oi, tris, rays, any_hit=True)[0]
    assert want.view(np.int32)[0, 3] == 0 and accepted_behind(tris, rays).all()
    m = rb.Mbvh.construct(gpu_build(tris, "locb"))
    got = m.intersect(to_cuda(rays), any_hit=True)[0].cpu().numpy()
    assert np.array_equal(u32(got), u32(want))
