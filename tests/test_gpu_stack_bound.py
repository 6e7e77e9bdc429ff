"""Rays that need more than the 64 stack entries of a walk over the quad nodes:
a leaf that the node of the overflowing push tests before it still counts, and
small launches (four lanes per ray) report what large ones (one lane) do."""
import struct

import numpy as np
import pytest

import rtbvh_gb300 as rb
from gpu_helpers import to_cuda, u32

pytestmark = pytest.mark.gpu


def deep_tree(levels, interior, leaf_at):
    """A chain of `levels` quad nodes with three interior slots behind the next
    one, so that a ray along +x pushes three entries at each, then a node with
    `interior` interior slots and a leaf whose triangle the ray hits: in front
    of them ("near") or behind ("far"). Returns the nodes, indices and
    triangles; every other triangle is off the ray."""
    boxes, links, tris = [None], [None], []

    def pair():
        boxes.extend([None, None])
        links.extend([None, None])
        return len(boxes) - 2

    def leaf(at, x, on_ray=False):
        y = 0.0 if on_ray else 0.9
        t = np.array([[x, y - 0.05, -0.05], [x, y + 0.05, -0.05], [x, y, 0.05]], np.float32)
        boxes[at] = (t.min(0) - 0.01, t.max(0) + 0.01)
        links[at] = (1, len(tris))
        tris.append(t)

    def small(at, x):  # two leaves in a box that the ray enters at x
        boxes[at] = (np.array([x, -1.0, -1.0]), np.array([90.0, 1.0, 1.0]))
        k = pair()
        links[at] = (-1, k)
        leaf(k, x + 1.0)
        leaf(k + 1, x + 2.0)

    def wide(at):
        boxes[at] = (np.array([1.0, -1.0, -1.0]), np.array([100.0, 1.0, 1.0]))
        k = pair()
        links[at] = (-1, k)
        return k

    def quad(at):  # the four grandchildren of node `at`
        k = wide(at)
        a, b = wide(k), wide(k + 1)
        return [a, a + 1, b, b + 1]

    at = 0
    for _ in range(levels):
        slots = quad(at)
        for x, c in zip((2.0, 3.0, 4.0), slots[:3]):
            small(c, x)
        at = slots[3]
    slots = quad(at)
    leaf(slots[0], 1.5 if leaf_at == "near" else 80.0, on_ray=True)
    for x, c in zip((2.0, 3.0, 4.0)[:interior], slots[1:1 + interior]):
        small(c, x)
    for c in slots[1 + interior:]:
        leaf(c, 50.0)
    nodes = np.zeros((len(boxes), 8), np.float32)
    ints = nodes.view(np.int32)
    for k, ((lo, hi), (count, first)) in enumerate(zip(boxes, links)):
        nodes[k, :3], nodes[k, 4:7] = lo, hi
        ints[k, 3], ints[k, 7] = count, first
    return nodes, np.arange(len(tris), dtype=np.uint32), np.stack(tris)


def _structure(nodes, idx, tris):
    data = (struct.pack("<Q", len(nodes)) + nodes.tobytes() + struct.pack("<Q", len(idx)) + idx.tobytes() +
            struct.pack("<I", 1))
    g = rb.Bvh.from_bytes(data)
    g.attach_triangles(to_cuda(tris))
    return rb.Mbvh.construct(g)


@pytest.mark.parametrize("mode", [{"any_hit": True}, {"any_hit": True, "exact_nodes": True}, {"exact_nodes": True}],
                         ids=["any", "any_exact", "closest_exact"])
@pytest.mark.parametrize("leaf_at", ["far", "near"])
@pytest.mark.parametrize("levels", [20, 21])
@pytest.mark.parametrize("interior", [1, 2, 3])
def test_small_launches_stop_where_large_ones_do(levels, interior, leaf_at, mode):
    m = _structure(*deep_tree(levels, interior, leaf_at))
    ray = np.array([[0.0, 0.0, 0.0, 1.0, 1e-4, 1e-4]], np.float32)
    few, many = to_cuda(np.repeat(ray, 100, 0)), to_cuda(np.repeat(ray, 80000, 0))
    want = m.intersect(many, **mode)[0].cpu().numpy()
    want_status = m.status()
    got = m.intersect(few, **mode)[0].cpu().numpy()
    assert m.status() == want_status
    assert np.array_equal(u32(got), u32(want[:100]))
    # 3 entries per level, then a push less than interior slots
    overflows = 3 * levels + interior - 1 > 64
    hit_first = mode.get("any_hit") and leaf_at == "far"
    assert (want_status == rb.ResultCode.StackOverflow) == (overflows and not hit_first)
    assert (rb.hit_prims(got)[0] == -2) == (overflows and not hit_first)
    if overflows and leaf_at == "far":  # the leaf's t stands
        assert abs(got[0, 0] - 80.0) < 1e-3
