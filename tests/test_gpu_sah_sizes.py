"""Binned-SAH builds of the sizes where tasks change form (32 primitives: a
lane each; more: a warp; the breadth-first part above), small leaves, equal
and degenerate primitives: the tree in canonical form and its Mbvh against the
oracle."""
import numpy as np
import pytest

import oracle
import rtbvh_gb300 as rb
from gpu_helpers import canonical, gpu_build, oracle_build, u32
from rtbvh_gb300 import scenes

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 4, 7, 8, 9, 15, 16, 17, 31, 32, 33, 34, 63, 64, 65, 100, 255, 257, 600, 1023, 1025, 2049, 5000, 20011]


def _scene(n, kind):
    if kind == "soup":
        return scenes.incoherent(n, seed=n + 1, median=0.02)
    if kind == "sphere":
        return scenes.sphere_fast(max(3, int(np.sqrt(n)) + 1), max(2, int(np.sqrt(n)) // 2 + 1), seed=n)[:n]
    if kind == "flat":  # one axis has no extent: its bins are all alike
        t = scenes.incoherent(n, seed=n + 2, median=0.02)
        t[:, :, 1] = 0.0
        return t
    t = np.repeat(scenes.incoherent(max(1, n // 5), seed=n + 3, median=0.02), 6, axis=0)[:n]  # groups of equal ones
    return np.concatenate([t, np.zeros((n - len(t), 3, 3), np.float32)]) if len(t) < n else t


@pytest.mark.parametrize("kind", ["soup", "sphere", "flat", "equal"])
@pytest.mark.parametrize("ppl", [None, 4])
@pytest.mark.parametrize("n", SIZES)
def test_sah_sizes(n, ppl, kind):
    tris = _scene(n, kind)
    g = gpu_build(tris, "sah", ppl)
    on, oi = oracle_build(tris, "sah", ppl or 1)
    nodes, idx = g.nodes(), g.indices()
    assert len(nodes) == len(on)
    assert canonical(nodes, idx) == canonical(on, oi)
    assert np.array_equal(np.sort(idx), np.arange(len(tris)))
    assert np.array_equal(u32(rb.Mbvh.construct(g).quad_nodes()), u32(oracle.mbvh(nodes)))


@pytest.mark.parametrize("n,kind", [(1048577, "soup"), (1300003, "equal"), (1100000, "sphere")])
def test_sah_above_the_cooperative_size(n, kind):
    """Builds of more than 2^20 primitives launch the phases of a level one by
    one, the indices changing sides at every level."""
    tris = _scene(n, kind)
    g = gpu_build(tris, "sah")
    on, oi = oracle_build(tris, "sah")
    nodes, idx = g.nodes(), g.indices()
    assert len(nodes) == len(on)
    assert np.array_equal(np.sort(idx), np.arange(len(tris)))
    assert np.array_equal(u32(oracle.mbvh(nodes)), u32(oracle.mbvh(on)))


@pytest.mark.parametrize("n,kind", [(329727, "soup"), (329728, "soup"), (330001, "equal"), (340007, "sphere")])
def test_sah_subtrees_in_two_launches(n, kind):
    """From 329,728 primitives subtrees have more than 160 and are split first."""
    tris = _scene(n, kind)
    g = gpu_build(tris, "sah")
    on, oi = oracle_build(tris, "sah", 1)
    nodes, idx = g.nodes(), g.indices()
    assert len(nodes) == len(on)
    assert canonical(nodes, idx) == canonical(on, oi)


def test_sah_one_launch_above_a_million():
    tris = _scene(1100003, "sphere")
    g = gpu_build(tris, "sah")
    on, oi = oracle_build(tris, "sah", 1)
    nodes, idx = g.nodes(), g.indices()
    assert len(nodes) == len(on)
    assert canonical(nodes, idx) == canonical(on, oi)
