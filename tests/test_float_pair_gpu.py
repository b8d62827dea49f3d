"""The cosine lobe's sample on the device against its double evaluation in numpy, bit for bit: angles on a grid,
next to the quadrants (where the reduced angle cancels) and at the ends of the range."""
import numpy as np
import pytest

from pico_gb300.types import DIFFUSE, Material

pytestmark = pytest.mark.gpu

f = np.float32


def _normalise(v):
    d = (v[0] * v[0] + v[1] * v[1]) + v[2] * v[2]
    s = f(1.0) / np.sqrt(d)
    return [x * s for x in v]


def _angles(where, n, rng):
    if where == "grid":
        return rng.integers(0, 2**32, n).astype(f) / f(2**32)
    if where == "quadrants":
        base = rng.integers(0, 5, n) * 0.25
        return np.clip(base + rng.integers(-200, 200, n) * 2.0**-26, 0.0, 1.0).astype(f)
    ends = np.array([0.0, 1.0, 0.25, 0.5, 0.75, 2.0**-32, 1.0 - 2.0**-24], f)
    return ends[np.arange(n) % len(ends)]


@pytest.mark.parametrize("where,n", [("grid", 40000), ("quadrants", 40000), ("ends", 70)])
def test_cosine_sample_is_the_double_evaluation(ctx, where, n):
    rng = np.random.default_rng(7)
    u1, u2 = rng.integers(0, 2**32, n).astype(f) / f(2**32), _angles(where, n, rng)
    u1[:4] = [0.0, 1.0, 2.0**-32, 0.5]
    up = np.tile(np.array([[0, 0, 1]], f), (n, 1))   # V = N = z: the frame swaps x and y
    xi = np.zeros((n, 4), f)
    xi[:, 0], xi[:, 1] = u1, u2
    _, L, P, _, _ = ctx.bsdf_eval(np.full(n, DIFFUSE, np.uint32), [Material(diffuse=(0.5, 0.5, 0.5))] * n, up, up, up, xi)
    r = np.sqrt(u1)
    phi = (u2.astype(np.float64) * np.pi * 2.0).astype(f).astype(np.float64)
    x = (r.astype(np.float64) * np.cos(phi)).astype(f)
    y = (r.astype(np.float64) * np.sin(phi)).astype(f)
    z = np.sqrt(np.maximum(f(1.0) - u1, f(0.0)))
    h = _normalise([x, y, z])
    want = np.stack(_normalise([h[1], h[0], h[2]]), axis=1)
    np.testing.assert_array_equal(P, np.maximum(h[2] / f(np.pi), f(0.0)))
    np.testing.assert_array_equal(L, want)
