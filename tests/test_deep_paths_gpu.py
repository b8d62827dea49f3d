"""Paths deeper than the ring of queue sizes (64 depths) and than its second turn: the number of paths that reach a
depth does not depend on how deep the render may go, and never grows with the depth."""
import numpy as np
import pytest

from pico_gb300 import scenes
from pico_gb300.types import DIFFUSE, LIGHT, Instance, Material, SceneData

pytestmark = pytest.mark.gpu


def _closed_box():
    s = SceneData(materials=[Material(diffuse=(0.97, 0.97, 0.97)), Material(emissive=(4.0, 4.0, 4.0))])
    s.meshes = [scenes.cube_mesh(), scenes.quad_mesh([[-0.3, 0.9, -0.3], [0.3, 0.9, -0.3], [0.3, 0.9, 0.3],
                                                      [-0.3, 0.9, 0.3]], [0, -1, 0])]
    s.instances = [Instance(0, scenes.glm_storage(scenes.scale([2.0, 2.0, 2.0])), DIFFUSE, 0),
                   Instance(1, scenes.glm_storage(np.eye(4)), LIGHT, 1)]
    return s


@pytest.mark.parametrize("batched", [False, True])
def test_reached_depths(ctx, batched):
    gs, cam = ctx.upload(_closed_box()), scenes.lit_field_camera(48, 40)
    cam.position, cam.direction = (0.1, 0.0, -0.6), (0.0, 0.0, 1.0)
    rays = {}
    for depth in (1, 2, 61, 62, 63, 64, 65, 66, 126, 127, 128, 129, 130):
        if batched:
            item = {"gpu_scene": gs, "camera": cam, "max_samples": 512, "max_depth": depth, "seed": 5, "estimator": 1}
            _, report = ctx.render_many([item])
            rays[depth], image = report["rays"], item["pixels"]
        else:
            image = gs.render(cam, depth, 512, seed=5, estimator=1)[0]
            st = ctx.render_stats()
            rays[depth] = st["camera_paths"] + st["bounce_rays"] + st["shadow_rays"]
        assert np.isfinite(image).all()
    gs.free()
    added = {d: rays[d] - rays[d - 1] for d in rays if d - 1 in rays}   # by the paths that reach depth d
    order = sorted(added)
    assert all(added[a] >= added[b] for a, b in zip(order, order[1:])), added
    assert added[66] > 100 and added[130] > 0, added
