"""Any-hit walks that skip slots without a hit (wholly behind the origin, or
subtree boxes the ray cannot enter) against the exact walk that skips none:
the hits are the reference order's first ones, bit for bit."""
import numpy as np
import pytest

from gpu_helpers import gpu_build, scene, to_cuda, u32
import rtbvh_gb300 as rb

pytestmark = pytest.mark.gpu


def _rays(tris, n, seed):
    """Origins in the scene box, on surfaces (1e-4 off) and outside; some
    axis-parallel directions (non-finite inverse)."""
    rng = np.random.default_rng(seed)
    lo, hi = tris.reshape(-1, 3).min(0), tris.reshape(-1, 3).max(0)
    size = float((hi - lo).max())
    t = tris[rng.integers(0, len(tris), n)].astype(np.float64)
    w = rng.dirichlet((1.0, 1.0, 1.0), n)[:, :, None]
    nrm = np.cross(t[:, 1] - t[:, 0], t[:, 2] - t[:, 0])
    nrm /= np.maximum(np.linalg.norm(nrm, axis=1, keepdims=True), 1e-30)
    o = (t * w).sum(1) + 1e-4 * nrm
    o[: n // 3] = rng.uniform(lo, hi, size=(n // 3, 3))
    o[n // 3: n // 2] += size * rng.normal(size=(n // 2 - n // 3, 3))
    d = rng.normal(size=(n, 3))
    d[::97, 1] = 0.0
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.concatenate([o, d], 1).astype(np.float32)
    return rays, (size * rng.uniform(0.01, 2.0, n)).astype(np.float32)


@pytest.mark.parametrize("name", ["sphere", "teapot", "incoherent_20k"])
@pytest.mark.parametrize("kind", ["locb", "sah", "sah_refit"])
@pytest.mark.parametrize("scale", [1.0, 300.0])
def test_any_hit_equals_the_walk_without_skips(name, kind, scale):
    """scale 300 puts the scene beyond the range of the skips."""
    tris = (scene(name) * np.float32(scale)).astype(np.float32)
    g = gpu_build(tris, kind.split("_")[0])
    m = rb.Mbvh.construct(g)
    if kind == "sah_refit":
        g.refit(triangles=to_cuda(tris), mbvh=m)
    rays, t_max = _rays(tris, 32771, 3)
    r, tm = to_cuda(rays), to_cuda(t_max)
    for limit in (tm, None):
        got = m.intersect(r, t_max=limit, any_hit=True)[0].cpu().numpy()
        want = m.intersect(r, t_max=limit, any_hit=True, exact_nodes=True)[0].cpu().numpy()
        assert np.array_equal(u32(got), u32(want))
    assert m.status() == rb.ResultCode.Ok
    hits = rb.hit_prims(got) >= 0
    assert hits.sum() > len(rays) // 50 and (~hits).sum() > 0
