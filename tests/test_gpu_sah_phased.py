"""Binned-SAH builds of more than 2^21 primitives launch the phases of a level
one by one instead of in one cooperative launch: trees and leaves against the
oracle."""
import numpy as np
import pytest

import oracle
from gpu_helpers import gpu_build, oracle_build, u32
from test_gpu_sah import _leaf_sets
from test_gpu_sah_sizes import _scene

pytestmark = pytest.mark.gpu


def _check(n, kind):
    tris = _scene(n, kind)
    g = gpu_build(tris, "sah")
    on, oi = oracle_build(tris, "sah")
    nodes, idx = g.nodes(), g.indices()
    assert len(nodes) == len(on)
    assert np.array_equal(np.sort(idx), np.arange(len(tris)))
    quads, want = oracle.mbvh(nodes), oracle.mbvh(on)
    assert np.array_equal(u32(quads), u32(want))
    for a, b in zip(_leaf_sets(quads, idx), _leaf_sets(want, oi)):
        assert np.array_equal(a, b)


def test_levels_of_few_and_of_many_tasks():
    """A level of at most 1,024 tasks is numbered by one block, a larger one by
    the grid; here levels of 512, 1,013, 1,652, 942 and 127 tasks follow one
    another, so the form changes both ways."""
    _check(3300001, "soup")


@pytest.mark.parametrize("n,kind", [(2097152, "soup"), (2097153, "soup"), (2200003, "equal"), (2200001, "sphere")])
def test_both_sides_of_the_cooperative_size(n, kind):
    """The last size of one launch and the first of separate phases, and equal
    and clustered primitives above it."""
    _check(n, kind)
