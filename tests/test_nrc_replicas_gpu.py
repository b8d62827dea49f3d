"""Training batches on both sides of the size from which the coarse levels' gradients gather in copies: a batch's
gradient is the mean of its parts' gradients, weighted by their records."""
import numpy as np
import pytest

import po_nrc
from pico_gb300 import RadianceCache

pytestmark = pytest.mark.gpu

LO, HI = (-1.0, -1.0, -1.0), (1.0, 1.0, 1.0)


@pytest.mark.parametrize("log2_table", [12, 14, 19])   # no, two and four levels have copies
@pytest.mark.parametrize("n", [16383, 16384, 20001])
def test_gradient_of_a_batch_is_its_parts(ctx, n, log2_table):
    cache = RadianceCache(ctx, log2_table_size=log2_table, aabb_min=LO, aabb_max=HI, seed=2)
    rng = np.random.default_rng(n)
    cache.set_params(cache.params()[0], rng.uniform(-0.5, 0.5, (16, cache.table_size, 2)).astype(np.float32))
    q = po_nrc.make_queries(n, 4, LO, HI)
    q["position"][: n // 2] *= 0.05   # half of the records share a few coarse cells
    t = rng.gamma(1.0, 1.0, (n, 3)).astype(np.float32)
    cache.train(q, t, apply=False)
    whole = cache.gradients()
    parts, at = [np.zeros_like(g, dtype=np.float64) for g in whole], 0
    for k in (n // 3, n // 3, n - 2 * (n // 3)):
        cache.train(q[at:at + k], t[at:at + k], apply=False)
        for p, g in zip(parts, cache.gradients()):
            p += g.astype(np.float64) * (k / n)
        at += k
    cache.free()
    # every record's contribution is the same but for the loss scale's rounding into bf16 (2^-9 of it, of either sign):
    # at most 2^-8 of a sum's norm, and the sums' own float rounding far below
    for g, p in zip(whole, parts):
        assert np.linalg.norm(g - p) <= 2.0**-8 * np.linalg.norm(p)
