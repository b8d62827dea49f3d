"""Radiance-cache renders whose buffers may not grow beyond what one pass, or three, takes: groups of passes shrink to
fit and give back what they had reserved before, so a render fits wherever its passes fit one at a time."""
import ctypes as C

import numpy as np
import pytest

import pico_gb300
from pico_gb300 import ESTIMATOR_RADIANCE_CACHE, RadianceCache, scenes

pytestmark = pytest.mark.gpu

W, H, DEPTH, SPP = 41, 30, 5, 20


def _group_bytes(passes, paths):
    """Path state, previous roughness, records (query, throughput and payload, target, flag, place in the order) and
    terminal queries."""
    slots, records, terms = passes * max(W * H, paths), passes * paths * DEPTH, passes * W * H
    queries = max(records, terms) if passes == 1 else records + terms
    return slots * (208 + 4) + records * (32 + 16 + 5) + queries * 64 + 2048   # and some counters


def _render(ctx, budget, paths, steps):
    ctx.lib.pico_test_cache_budget(ctx.handle, C.c_uint64(budget))
    gs = ctx.upload(scenes.cornell_box())
    cache = RadianceCache(ctx, log2_table_size=12, seed=5, train_paths=paths, max_train_steps=steps)
    cache.attach()
    try:
        image = gs.render(scenes.cornell_camera(W, H), DEPTH, SPP, seed=4, estimator=ESTIMATOR_RADIANCE_CACHE,
                          denoise=True)
        return image, cache.stats(), cache.info()
    finally:
        cache.free()
        gs.free()


@pytest.mark.parametrize("paths", [300, 5000])   # fewer than the image's pixels, and more records than queries
@pytest.mark.parametrize("passes", [1, 3])
@pytest.mark.parametrize("steps", [0, 4])
def test_groups_shrink_to_fit(ctx, passes, paths, steps):
    want = _render(ctx, 2**64 - 1, paths, steps)
    small = pico_gb300.Context(0)   # holds nothing yet
    try:
        got = _render(small, _group_bytes(passes, paths), paths, steps)
        with pytest.raises(pico_gb300.PicoError):
            _render(small, 1, 2 * paths + 5000, steps)
        again = _render(small, _group_bytes(passes, paths), paths, steps)
    finally:
        small.close()
    assert got[1:] == want[1:] == again[1:]
    for a, b, c in zip(got[0], again[0], want[0]):
        assert np.isfinite(a).all() and np.isfinite(b).all()
        if steps == 0:   # without optimiser steps the images are equal bit for bit
            np.testing.assert_array_equal(a, c)
            np.testing.assert_array_equal(b, c)
