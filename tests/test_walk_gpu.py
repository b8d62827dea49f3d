"""The near-first queue walk at the edges of its leaves and of its warps: instances that share a TLAS leaf beside
instances with a leaf of their own, and primary-ray launches of fewer pixels than a warp, a claim and a grid."""
import numpy as np
import pytest

from pico_gb300 import scenes
from pico_gb300.types import DIFFUSE, Instance

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stacked", [2, 31, 32, 33])
def test_shared_and_single_instance_leaves(ctx, oracle, stacked):
    """`stacked` concentric instances cannot be split and share one leaf (over 31: a chain of leaves)."""
    s = scenes.instance_field(n_instances=5, level=1, seed=6, extent=3.0)
    for k in range(stacked):
        s.instances.append(Instance(0, scenes.glm_storage(scenes.scale(np.full(3, 0.5 + 0.01 * k))), DIFFUSE, 0))
    rays = scenes.surface_rays(s, 3000, seed=stacked)
    gs = ctx.upload(s)
    got, want = gs.trace_closest(rays), oracle.scene(s).trace(rays)
    gs.free()
    assert (want["inst"] >= 5).any()
    for k in ("inst", "prim"):
        np.testing.assert_array_equal(got[k], want[k])
    np.testing.assert_array_equal(got["t"].view(np.uint32), want["t"].view(np.uint32))


@pytest.mark.parametrize("size", [(1, 1), (31, 1), (9, 33), (129, 65)])
def test_denoiser_inputs_of_few_pixels(ctx, oracle, size):
    scene, cam = scenes.cornell_box(), scenes.cornell_camera(*size)
    gs = ctx.upload(scene)
    got, want = gs.denoiser_inputs(cam), oracle.scene(scene).denoiser_inputs(cam)
    gs.free()
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, np.asarray(b).reshape(a.shape))


@pytest.mark.parametrize("size", [(1, 1), (7, 9), (8, 8), (17, 5), (64, 31)])
def test_tile_order_covers_ragged_images(ctx, size):
    """Every pixel of images that do not divide into 8 x 8 tiles takes its samples once, on the device's list and
    on the host-built one of batched renders, with the same result as when the whole image is one batch's chunk."""
    gs = ctx.upload(scenes.cornell_box())
    cam = scenes.cornell_camera(*size)
    whole, count, _ = gs.render(cam, 4, 6, seed=3, estimator=1)
    assert (count == 6).all()
    try:
        ctx.set_path_limit(64)
        chunked, count, _ = gs.render(cam, 4, 6, seed=3, estimator=1)
    finally:
        ctx.set_path_limit(0)
    items = [{"gpu_scene": gs, "camera": cam, "max_samples": 6, "max_depth": 4, "seed": 3, "estimator": 1}]
    ctx.render_many(items)
    gs.free()
    assert (count == 6).all() and (items[0]["sample_count"] == 6).all()
    np.testing.assert_array_equal(whole, chunked)
    np.testing.assert_array_equal(whole, items[0]["pixels"])


@pytest.mark.parametrize("n", [1, 5, 31, 33, 1000, 5471, 5472, 5473, 20000, 175104, 175105])
def test_few_rays_per_warp(ctx, oracle, n):
    """Launches of one ray per warp up to 32: every ray is walked once, whatever the warps' shares."""
    s = scenes.instance_field(n_instances=16, level=1, seed=3, extent=5.0)
    rays = scenes.surface_rays(s, n, seed=n)
    gs = ctx.upload(s)
    got, want = gs.trace_closest(rays), oracle.scene(s).trace(rays)
    gs.free()
    for k in ("inst", "prim"):
        np.testing.assert_array_equal(got[k], want[k])
    np.testing.assert_array_equal(got["t"].view(np.uint32), want["t"].view(np.uint32))
