"""Sorts of the sizes that one block does alone, at the edges of its rows and
items per thread, through LOCB builds: codes all different, all alike (the
order has to stay) and in a few large groups, against the oracle."""
import numpy as np
import pytest

from gpu_helpers import gpu_build, oracle_build, u32
from rtbvh_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["soup", "alike", "groups"])
@pytest.mark.parametrize("n", [2, 31, 32, 33, 64, 65, 1023, 1024, 1025, 2048, 2049, 4096, 4097, 8191, 8192, 8193])
def test_small_sorts(n, kind):
    tris = scenes.incoherent(n, seed=n)
    if kind == "alike":  # different triangles, one centre up to rounding
        tris = tris - tris.mean(axis=1, keepdims=True)
        tris[0] *= 1000.0
    elif kind == "groups":
        tris = (tris - tris.mean(axis=1, keepdims=True)) * 1e-3 + (np.arange(n) * 7919 % 5)[:, None, None]
    tris = tris.astype(np.float32)
    g = gpu_build(tris, "locb")
    on, oi = oracle_build(tris, "locb")
    assert np.array_equal(g.indices(), oi)
    assert np.array_equal(u32(g.nodes()), u32(on))
