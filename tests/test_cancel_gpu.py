"""Cancelled renders into buffers without a sample, whose mean and variance are not uploaded: pixels that took samples
hold those of the uncancelled render's first so many, the others the caller's values."""
import ctypes as C
import threading
import time

import numpy as np
import pytest

import pico_gb300
from pico_gb300 import ESTIMATOR_RADIANCE_CACHE, RadianceCache, scenes

pytestmark = pytest.mark.gpu


def _cancelled(gs, cam, spp, seed, estimator, after):
    """The buffers of a render that is cancelled `after` seconds in, and the values they began with."""
    W, H = cam.resolution
    rng = np.random.default_rng(9)
    pix, var = (rng.normal(size=(H, W, 3)).astype(np.float32) for _ in range(2))
    count = np.zeros((H, W), np.uint32)
    before, flag = (pix.copy(), var.copy()), C.c_int32(0 if after > 0 else 1)
    timer = threading.Timer(after, lambda: setattr(flag, "value", 1))
    timer.start()
    try:
        gs.render(cam, 4, spp, seed=seed, estimator=estimator, pixels=pix, sample_count=count, variance=var,
                  max_variance=-1.0, should_quit=flag)
    except pico_gb300.PicoError as e:
        assert e.status == -6
    timer.cancel()
    timer.join()
    return pix, count, var, before


def _check(gs, cam, seed, estimator, got):
    pix, count, var, before = got
    for c in np.unique(count):
        at = count == c
        want = before if c == 0 else gs.render(cam, 4, int(c), seed=seed, estimator=estimator, max_variance=-1.0)[::2]
        np.testing.assert_array_equal(pix[at], want[0][at])
        np.testing.assert_array_equal(var[at], want[1][at])


@pytest.mark.parametrize("estimator", [0, 1])
def test_some_chunks_sampled(ctx, estimator):
    """A path limit below the image renders it in chunks: some are done when the cancel is seen, others not begun."""
    gs, cam = ctx.upload(scenes.cornell_box()), scenes.cornell_camera(96, 65)
    limit, spp = 1000, 64
    try:
        ctx.set_path_limit(limit)
        gs.render(cam, 4, spp, seed=3, estimator=estimator, max_variance=-1.0)
        t = time.perf_counter()
        gs.render(cam, 4, spp, seed=3, estimator=estimator, max_variance=-1.0)
        whole = time.perf_counter() - t
        for part in (0.5, 0.4, 0.6, 0.3, 0.7):
            got = _cancelled(gs, cam, spp, 3, estimator, part * whole)
            if 0 < (got[1] > 0).sum() < got[1].size:
                break
        assert 0 < (got[1] > 0).sum() < got[1].size
        ctx.set_path_limit(0)
        _check(gs, cam, 3, estimator, got)
    finally:
        ctx.set_path_limit(0)
        gs.free()


@pytest.mark.parametrize("part", [0.0, 0.5])
def test_radiance_cache(ctx, part):
    """A cache render is cancelled between groups of passes: every pixel has the same samples, none at first."""
    gs, cam = ctx.upload(scenes.cornell_box()), scenes.cornell_camera(96, 65)
    cache = RadianceCache(ctx, log2_table_size=12, seed=5, max_train_steps=0)
    cache.attach()
    try:
        gs.render(cam, 4, 160, seed=3, estimator=ESTIMATOR_RADIANCE_CACHE)
        t = time.perf_counter()
        gs.render(cam, 4, 160, seed=3, estimator=ESTIMATOR_RADIANCE_CACHE)
        got = _cancelled(gs, cam, 160, 3, ESTIMATOR_RADIANCE_CACHE, part * (time.perf_counter() - t))
        assert len(np.unique(got[1])) == 1 and got[1].flat[0] % 16 == 0
        assert part > 0 or got[1].flat[0] == 0
        _check(gs, cam, 3, ESTIMATOR_RADIANCE_CACHE, got)
    finally:
        cache.free()
        gs.free()
