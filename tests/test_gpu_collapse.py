"""The MBVH collapse and the closest-hit traversal tree, one thread per BVH2
node: node counts around the block size, the smallest trees, chains (the
longest walks to a known place), and arrays with nodes no root reaches."""
import struct

import numpy as np
import pytest

import oracle
import rtbvh_gb300 as rb
from gpu_helpers import gpu_build, to_cuda, u32
from rtbvh_gb300 import scenes

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 4, 5, 6, 7, 8, 9, 16, 17, 31, 33, 64, 127, 128, 129, 255, 257, 1000, 4099]


def _half_area(n):
    d = n[4:7] - n[0:3]
    return np.float32(np.float32((d[0] + d[1]) * d[2]) + np.float32(d[0] * d[1]))


def _wide_slots(nodes, c):
    """BVH2 nodes in the four slots of node c's traversal node: its children,
    then twice the interior slot of largest half area opened."""
    ni = nodes.view(np.int32)
    inner = lambda x: ni[x, 3] < 0 and ni[x, 7] >= 0  # noqa: E731
    if not inner(c):
        return [c]
    slots = [ni[c, 7], ni[c, 7] + 1]
    while len(slots) < 4:
        best, area = -1, np.float32(-1.0)
        for i, x in enumerate(slots):
            if inner(x) and _half_area(nodes[x]) > area:
                best, area = i, _half_area(nodes[x])
        if best < 0:
            break
        x = ni[slots[best], 7]
        slots[best] = x
        slots.append(x + 1)
    return slots


def _check_wide(m, nodes):
    ex, cp = m.traversal_tree()
    ni, xi = nodes.view(np.int32), ex.view(np.int32)
    seen, stack = 0, [(0, 0)]
    while stack:
        w, c = stack.pop()
        seen += 1
        slots = _wide_slots(nodes, c)
        for i in range(4):
            x = slots[i] if i < len(slots) else slots[0]
            assert np.array_equal(u32(ex[w, [i, 8 + i, 16 + i, 4 + i, 12 + i, 20 + i]]), u32(nodes[x, [0, 1, 2, 4, 5, 6]]))
            if i >= len(slots):
                assert (xi[w, 24 + i], xi[w, 28 + i]) == (-1, -1)
            elif ni[x, 3] < 0 and ni[x, 7] >= 0:
                assert xi[w, 28 + i] == -1
                stack.append((int(xi[w, 24 + i]), int(x)))
            else:
                assert (xi[w, 24 + i], xi[w, 28 + i]) == (ni[x, 7], ni[x, 3])
    assert seen == len(ex) == len(cp)


@pytest.mark.parametrize("n", SIZES)
def test_collapse_sizes(n):
    tris = scenes.incoherent(n, seed=100 + n, median=0.05)
    for kind in ("locb", "sah"):
        g = gpu_build(tris, kind)
        m = rb.Mbvh.construct(g)
        nodes = g.nodes()
        assert np.array_equal(u32(m.quad_nodes()), u32(oracle.mbvh(nodes)))
        if kind == "locb":
            _check_wide(m, nodes)


def _chain(depth, extra):
    """A BVH2 whose left children go on `depth` levels, every right child a
    leaf, and `extra` nodes that nothing refers to."""
    n = depth + 1
    nodes = np.zeros((2 * n - 1 + extra, 8), np.float32)
    ints = nodes.view(np.int32)
    ints[:, 3], ints[:, 7] = -1, -1
    at, leaf = 0, 0
    for k in range(depth):
        nodes[at, 0:3], nodes[at, 4:7] = 0.0, float(n - k)
        ints[at, 3], ints[at, 7] = -1, 2 * k + 1
        right = 2 * k + 2
        nodes[right, 0:3], nodes[right, 4:7] = float(n - k - 1), float(n - k)
        ints[right, 3], ints[right, 7] = 1, leaf
        leaf += 1
        at = 2 * k + 1
    nodes[at, 4:7] = 1.0
    ints[at, 3], ints[at, 7] = 1, leaf
    return nodes, np.arange(n, dtype=np.uint32)


@pytest.mark.parametrize("depth,extra", [(1, 0), (2, 3), (63, 0), (700, 300)])
def test_collapse_of_a_chain(depth, extra):
    nodes, idx = _chain(depth, extra)
    data = struct.pack("<Q", len(nodes)) + nodes.tobytes() + struct.pack("<Q", len(idx)) + idx.tobytes()
    g = rb.Bvh.from_bytes(data + struct.pack("<I", 1))
    m = rb.Mbvh.construct(g)
    assert np.array_equal(u32(m.quad_nodes()), u32(oracle.mbvh(nodes)))
    tris = np.zeros((len(idx), 3, 3), np.float32)
    tris[:, :, :] = np.arange(len(idx))[::-1, None, None] + np.float32(0.25)
    tris[:, 1, 0] += np.float32(0.5)
    tris[:, 2, 1] += np.float32(0.5)
    m.attach_triangles(to_cuda(tris))
    ex, cp = m.traversal_tree()
    xi = ex.view(np.int32)
    leaves = sorted(int(xi[k, 24 + i]) for k in range(len(ex)) for i in range(4) if xi[k, 28 + i] >= 0)
    assert leaves == list(range(len(idx)))
    assert m.status() == rb.ResultCode.Ok


@pytest.mark.parametrize("sizes", [[1] * 70, [2, 1, 3, 1, 2, 300, 1], [1]])
def test_collapse_of_a_forest_of_tiny_meshes(sizes):
    off = np.concatenate([[0], np.cumsum(sizes)])
    tris = scenes.incoherent(int(off[-1]), seed=9, median=0.3)
    per = 64
    rays = np.concatenate([scenes.incoherent_rays(per, seed=20 + k)[0] for k in range(len(sizes))])
    batch = rb.Batch(to_cuda(tris), off, to_cuda(rays), np.arange(len(sizes) + 1) * per)
    hits = batch.run().cpu().numpy()
    assert batch.status() == rb.ResultCode.Ok
    for k in range(len(sizes)):
        m = rb.Mbvh.construct(gpu_build(tris[off[k]:off[k + 1]], "locb"))
        want = m.intersect(to_cuda(rays[k * per:(k + 1) * per]))[0].cpu().numpy()
        got = hits[k * per:(k + 1) * per]
        hit = rb.hit_prims(want) >= 0
        assert np.array_equal(u32(got[:, :3]), u32(want[:, :3]))
        assert np.array_equal(rb.hit_prims(got), np.where(hit, rb.hit_prims(want) + off[k], rb.hit_prims(want)))
