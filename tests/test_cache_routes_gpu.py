"""Trained radiance-cache images: repeated, and with passes traced in groups against one pass at a time (a path limit of
one image).

A training step's records have fixed places, but the sums of its grid gradients are taken in the order in which atomics
arrive, and the optimiser turns a rounding difference in a gradient that nearly cancels into a whole step, so an image
may differ from its own repetition.  The two routes may differ by that much, four times, or by a hundredth of what one
training pass more or less makes, where repetitions happen to agree: a route that gave a pass other records or steps,
or its answers before them, would differ like the latter."""
import numpy as np
import pytest

from pico_gb300 import ESTIMATOR_RADIANCE_CACHE, RadianceCache, scenes

pytestmark = pytest.mark.gpu


def _distance(a, b):
    return float(np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b.astype(np.float64)))


def _images(ctx, scene, W, H, depth, spp, paths, batch):
    """A function that renders the image with its own, newly seeded cache, and returns it and the cache's counts."""
    gs = ctx.upload(scenes.cornell_box() if scene == "cornell" else scenes.lit_field(n_instances=64, level=2, seed=3))
    cam = scenes.cornell_camera(W, H) if scene == "cornell" else scenes.lit_field_camera(W, H)

    def image(limit=0, warmup=0):
        cache = RadianceCache(ctx, log2_table_size=14, seed=5, train_paths=paths, train_batch=batch,
                              warmup_frames=warmup)
        cache.attach()
        ctx.set_path_limit(limit)
        try:
            return gs.render(cam, depth, spp, seed=4, estimator=ESTIMATOR_RADIANCE_CACHE)[0], cache.stats()
        finally:
            ctx.set_path_limit(0)
            cache.free()

    return image


@pytest.mark.parametrize("paths,batch", [(2048, 4096), (256, 512), (1000, 777)])
def test_a_step_takes_the_same_records_each_time(ctx, paths, batch):
    """Where a pass's records are split over several steps, which step takes a record must not depend on when the
    record was written."""
    image = _images(ctx, "cornell", 48, 37, 5, 6, paths, batch)
    repeated, other = [image() for _ in range(6)], image(warmup=1)[0]
    assert repeated[0][1]["train_steps"] >= 12
    own = max(_distance(a[0], b[0]) for a in repeated for b in repeated)
    assert own <= min(_distance(other, r[0]) for r in repeated) / 100


@pytest.mark.parametrize("scene,W,H,depth,spp,paths,batch", [
    ("cornell", 48, 37, 5, 6, 2048, 4096), ("field", 96, 54, 8, 18, 16384, 16384), ("field", 320, 180, 6, 4, 65536, 65536)])
def test_same_training(ctx, scene, W, H, depth, spp, paths, batch):
    image = _images(ctx, scene, W, H, depth, spp, paths, batch)
    limit = max(W * H, paths)   # room for one pass
    grouped, single = [image() for _ in range(5)], [image(limit) for _ in range(5)]
    other = image(warmup=1)[0]
    assert all(s == grouped[0][1] for _, s in grouped + single)
    grouped, single = [g[0] for g in grouped], [s[0] for s in single]
    own = max(_distance(r[i], r[j]) for r in (grouped, single) for i in range(5) for j in range(i))
    between = max(_distance(a, b) for a in grouped for b in single)
    apart = min(_distance(other, b) for b in grouped + single)
    print("own %.2g, between %.2g, a pass apart %.2g" % (own, between, apart))
    assert between <= max(4 * own, apart / 100)
