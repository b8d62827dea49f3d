"""A ray batch on a caller's stream beside the G-buffer's launch on the context's own: each walks a queue of its own."""
import numpy as np
import pytest

from pico_gb300 import scenes
from pico_gb300.types import HIT_DTYPE

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [5000, 3_000_001])
def test_batch_beside_gbuffer(ctx, n):
    gs = ctx.upload(scenes.instance_field(n_instances=256, level=3, seed=2))
    cam = scenes.lit_field_camera(640, 360)
    g = torch.Generator("cuda").manual_seed(3)
    rays = torch.zeros(n, 8, device="cuda")
    rays[:, 0:3] = torch.rand(n, 3, generator=g, device="cuda") * 40 - 20
    rays[:, 4:7] = torch.nn.functional.normalize(torch.randn(n, 3, generator=g, device="cuda"), dim=1)
    rays[:, 3] = 1.0
    hits = torch.empty(n, HIT_DTYPE.itemsize // 4, dtype=torch.int32, device="cuda")
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    gs.trace_closest_device(rays.data_ptr(), n, hits.data_ptr(), side.cuda_stream)
    side.synchronize()
    alone, inputs = hits.cpu().numpy(), gs.denoiser_inputs(cam)
    for _ in range(5):
        hits.fill_(-7)
        torch.cuda.synchronize()
        gs.trace_closest_device(rays.data_ptr(), n, hits.data_ptr(), side.cuda_stream)
        beside = gs.denoiser_inputs(cam)
        side.synchronize()
        np.testing.assert_array_equal(hits.cpu().numpy(), alone)
        for a, b in zip(beside, inputs):
            np.testing.assert_array_equal(a, b)
    gs.free()
