"""Radiance-cache renders whose passes are traced in groups of up to 16 against the same render one pass at a time (a
path limit of one sample per pixel), at sample counts around the group's size."""
import numpy as np
import pytest

from pico_gb300 import ESTIMATOR_RADIANCE_CACHE, RadianceCache, scenes

pytestmark = pytest.mark.gpu


def _render(ctx, gs, cam, spp, limit, **config):
    cache = RadianceCache(ctx, log2_table_size=12, seed=5, **config)
    cache.attach()
    ctx.set_path_limit(limit)
    try:
        image = gs.render(cam, 5, spp, seed=4, estimator=ESTIMATOR_RADIANCE_CACHE)
        return image, cache.stats(), cache.info()
    finally:
        ctx.set_path_limit(0)
        cache.free()


@pytest.mark.parametrize("spp", [1, 3, 16, 17, 33])
def test_frozen_cache(ctx, spp):
    """Without optimiser steps the images are equal bit for bit."""
    gs, cam = ctx.upload(scenes.cornell_box()), scenes.cornell_camera(21, 13)
    grouped = _render(ctx, gs, cam, spp, 0, max_train_steps=0)
    single = _render(ctx, gs, cam, spp, 21 * 13, max_train_steps=0)
    gs.free()
    for a, b in zip(grouped[0], single[0]):
        np.testing.assert_array_equal(a, b)
    assert grouped[1:] == single[1:] and grouped[2]["frames"] == spp


@pytest.mark.parametrize("spp,warmup", [(2, 0), (17, 0), (3, 18)])
def test_training_cache(ctx, spp, warmup):
    """With training, every pass has its own paths, records and steps, however the passes are grouped."""
    gs, cam = ctx.upload(scenes.cornell_box()), scenes.cornell_camera(21, 13)
    config = dict(train_paths=256, train_batch=512, warmup_frames=warmup)
    grouped, single = (_render(ctx, gs, cam, spp, limit, **config) for limit in (0, 21 * 13))
    gs.free()
    assert grouped[1:] == single[1:]
    assert grouped[1]["train_paths"] == 256 * (spp + warmup) and grouped[1]["train_steps"] > 0
    assert np.isfinite(grouped[0][0]).all() and (grouped[0][1] == spp).all()


@pytest.mark.parametrize("spp", [5, 17, 33])
def test_image_that_goes_on(ctx, spp):
    """Some pixels finished, some with samples, some without: grouped and single passes take the same samples."""
    gs, cam = ctx.upload(scenes.cornell_box()), scenes.cornell_camera(21, 13)
    rng = np.random.default_rng(spp)
    pix, var = (rng.random((13, 21, 3)).astype(np.float32) for _ in range(2))
    count = rng.choice(np.array([0, 3, spp], np.uint32), (13, 21))
    images = []
    for limit in (0, 256):   # without a limit in groups; below, in chunks of at most 256 pixels, pass by pass
        cache = RadianceCache(ctx, log2_table_size=12, seed=5, max_train_steps=0)
        cache.attach()
        ctx.set_path_limit(limit)
        try:
            images.append(gs.render(cam, 5, spp, seed=4, estimator=ESTIMATOR_RADIANCE_CACHE, pixels=pix.copy(),
                                    sample_count=count.copy(), variance=var.copy()) + (cache.stats()["queries"],))
        finally:
            ctx.set_path_limit(0)
            cache.free()
    gs.free()
    for a, b in zip(*images):
        np.testing.assert_array_equal(a, b)
    done = count == spp
    assert 0 < done.sum() < done.size and (images[0][0][done] == pix[done]).all() and (images[0][1][~done] > spp - 1).all()
