"""Renders into buffers without a sample yet do not read the mean and variance passed in; renders into buffers with
some do, and a cancelled render leaves the pixels that took none as they were."""
import ctypes as C

import numpy as np
import pytest

import pico_gb300
from pico_gb300 import scenes

pytestmark = pytest.mark.gpu

W, H = 24, 17


def _buffers(rng, done):
    """Arbitrary values, and `done` pixels of six samples each (all the render's samples)."""
    pix, var = (rng.normal(size=(H, W, 3)).astype(np.float32) for _ in range(2))
    count = np.zeros((H, W), np.uint32)
    count.reshape(-1)[rng.permutation(H * W)[:done]] = 6
    return pix, count, var


@pytest.mark.parametrize("done", [0, 1, H * W - 1, H * W])
def test_values_without_samples_do_not_count(ctx, done):
    rng = np.random.default_rng(done)
    gs, cam = ctx.upload(scenes.cornell_box()), scenes.cornell_camera(W, H)
    clean = gs.render(cam, 4, 6, seed=3, estimator=1)
    for batched in (False, True):
        pix, count, var = _buffers(rng, done)
        before, kept = (pix.copy(), var.copy()), count == 6
        if batched:
            ctx.render_many([{"gpu_scene": gs, "camera": cam, "max_samples": 6, "max_depth": 4, "seed": 3,
                              "estimator": 1, "pixels": pix, "sample_count": count, "variance": var}])
        else:
            gs.render(cam, 4, 6, seed=3, estimator=1, pixels=pix, sample_count=count, variance=var)
            assert ctx.render_stats()["samples"] == 6 * (H * W - done)
        assert (count == 6).all()
        for got, was, want in ((pix, before[0], clean[0]), (var, before[1], clean[2])):
            np.testing.assert_array_equal(got[kept], was[kept])
            np.testing.assert_array_equal(got[~kept], want[~kept])
    gs.free()


@pytest.mark.parametrize("estimator", [0, 1])
@pytest.mark.parametrize("done", [0, 5])
def test_cancelled_before_a_sample(ctx, estimator, done):
    pix, count, var = _buffers(np.random.default_rng(9), done)
    before = pix.copy(), count.copy(), var.copy()
    gs = ctx.upload(scenes.cornell_box())
    with pytest.raises(pico_gb300.PicoError) as e:
        gs.render(scenes.cornell_camera(W, H), 4, 6, seed=3, estimator=estimator, pixels=pix, sample_count=count,
                  variance=var, should_quit=C.c_int32(1))
    gs.free()
    assert e.value.status == -6
    for a, b in zip((pix, count, var), before):
        np.testing.assert_array_equal(a, b)
