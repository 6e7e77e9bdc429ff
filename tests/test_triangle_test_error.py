"""How far a triangle accepted by the float32 test may lie from the reported
point, against the bound the any-hit walks leave room for (kTestError in
traverse.cu): 0.17 |e1| |e2| |d| |o - v0| + 1.6e-6 |o - v0|."""
import numpy as np
import pytest

EPS = 2.0 ** -24


def _cross(a, b):
    return np.stack([a[:, 1] * b[:, 2] - b[:, 1] * a[:, 2], a[:, 2] * b[:, 0] - b[:, 2] * a[:, 0],
                     a[:, 0] * b[:, 1] - b[:, 0] * a[:, 1]], 1)


def _dot(a, b):
    return (a[:, 0] * b[:, 0] + a[:, 1] * b[:, 1]) + a[:, 2] * b[:, 2]


def _accepted(v0, e1, e2, o, d):
    """(t, u, v) and the accepting mask of the reference's test in float32."""
    with np.errstate(all="ignore"):
        h = _cross(d, e2)
        det = _dot(e1, h)
        f = np.float32(1.0) / det
        s = o - v0
        u = f * _dot(s, h)
        q = _cross(s, e1)
        v = f * _dot(d, q)
        t = f * _dot(e2, q)
        return t, u, v, (np.abs(det) >= np.float32(1e-5)) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (t > 1e-4)


@pytest.mark.parametrize("size", [0.01, 0.1, 1.0, 10.0])
@pytest.mark.parametrize("length", [0.1, 1.0, 30.0])
def test_the_accepted_point_lies_within_the_bound(size, length):
    rng = np.random.default_rng(3)
    n = 400000
    v0 = rng.uniform(-20.0, 20.0, (n, 3)).astype(np.float32)
    e1, e2 = ((size * rng.uniform(0.2, 1.0, (n, 1)) * rng.normal(size=(n, 3))).astype(np.float32) for _ in range(2))
    nrm = np.cross(e1.astype(float), e2)
    area = np.linalg.norm(nrm, axis=1, keepdims=True)
    nrm /= area
    # directions in the plane, tilted to determinants of 1e-5 to 1e-4 (or to
    # all that the triangle allows)
    a = rng.uniform(0.0, 2.0 * np.pi, (n, 1))
    e = e1 / np.linalg.norm(e1.astype(float), axis=1, keepdims=True)
    tilt = np.minimum(10.0 ** rng.uniform(-5.0, -4.0, (n, 1)) / (area * length), 3.0) * rng.choice([-1.0, 1.0], (n, 1))
    d = np.cos(a) * e + np.sin(a) * np.cross(nrm, e) + tilt * nrm
    d = (length * d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    w = rng.dirichlet((1.0, 1.0, 1.0), n)
    far = 10.0 ** rng.uniform(-4.0, 1.0, (n, 1)) * rng.choice([-1.0, 1.0], (n, 1))
    o = (v0 + w[:, :1] * e1 + w[:, 1:2] * e2 + far * d / length).astype(np.float32)
    t, u, v, ok = _accepted(v0, e1, e2, o, d)
    assert ok.sum() > 50
    v0, e1, e2, o, d, t, u, v = (x[ok].astype(np.float64) for x in (v0, e1, e2, o, d, t, u, v))
    off = np.linalg.norm(o + t[:, None] * d - v0 - u[:, None] * e1 - v[:, None] * e2, axis=1)
    s = np.linalg.norm(o - v0, axis=1)
    e1, e2, d = (np.linalg.norm(x, axis=1) for x in (e1, e2, d))
    s = np.maximum(s, 0.5 * np.maximum(e1, e2))  # the farthest corner is at least that far
    assert (off <= (0.17 * e1 * e2 * d + 1.6e-6) * s).all()
    # the constants: the sum of the roundings over the smallest determinant
    assert 27.4 * EPS / 1e-5 * 1.01 < 0.17 and 26 * EPS < 1.6e-6
