"""The denoiser at the edges of its tiles, sub-lattices and luminance cells: last tiles of 1 to 17 columns and rows (on
both sides of each spacing, where a level's white points come from cells or from the footprint itself), footprints
wider than the image, and pixels without a value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(1, 300), (97, 3), (31, 33), (65, 66), (68, 67), (72, 71), (79, 80), (81, 129),
                                 (128, 64), (513, 145)])
def test_against_the_oracle(ctx, oracle, W, H):
    rng = np.random.default_rng(W * 1000 + H)
    pix = rng.gamma(1.0, 1.0, (H, W, 3)).astype(np.float32)
    pix[:: 7, :: 5] *= 40.0                       # white points differ between tiles
    pix[: H // 2, : W // 3] = 0.0
    pix[H // 3, W // 2, 1] = np.nan               # never a white point; its taps have no value
    nrm = rng.normal(size=(H, W, 3)).astype(np.float32)
    pos = (rng.normal(size=(H, W, 3)) * 3).astype(np.float32)
    dif = rng.random((H, W, 3)).astype(np.float32)
    got, want = ctx.atrous(pix, nrm, pos, dif, W, H), oracle.atrous(pix, nrm, pos, dif, W, H)
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    # 1e-4 relative, the bound of the other comparisons; an absolute 1e-6 where neighbours cancel to nothing
    np.testing.assert_allclose(got[ok], want[ok], rtol=1e-4, atol=1e-6)
