"""The denoiser where a tap's weight lies below the smallest normal float: an infinite or huge colour still counts with
it, as with the reference's exponentials."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.inf, 3e38])
@pytest.mark.parametrize("W,H", [(24, 16), (70, 66)])
def test_against_the_oracle(ctx, oracle, value, W, H):
    rng = np.random.default_rng(W)
    pix = rng.uniform(0.5, 1.0, (H, W, 3)).astype(np.float32)
    pix[H // 2, W // 2, 0] = value
    nrm = np.zeros((H, W, 3), np.float32)
    nrm[H // 2, W // 2, 0] = np.sqrt(88.5 / 4)    # exp(-4 |dn|^2) = 3.7e-39, times the table's 0.003 to 0.16
    pos = np.zeros((H, W, 3), np.float32)
    pos[..., 0] = rng.uniform(1.0, 2.0, (H, W))   # |dp| at most the range
    dif = rng.random((H, W, 3)).astype(np.float32)
    got, want = ctx.atrous(pix, nrm, pos, dif, W, H), oracle.atrous(pix, nrm, pos, dif, W, H)
    pix[H // 2, W // 2, 0] = 1.0
    without = oracle.atrous(pix, nrm, pos, dif, W, H)
    assert want[H // 2, W // 2 + 1, 0] > 1.001 * without[H // 2, W // 2 + 1, 0]   # a neighbour gets its share
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
    np.testing.assert_array_equal(np.isinf(got), np.isinf(want))
    ok = np.isfinite(want)
    # 1e-4 relative, the bound of the denoiser's other comparisons (the smallest weights here keep 10 bits and move
    # a result by less than 1e-6)
    np.testing.assert_allclose(got[ok], want[ok], rtol=1e-4)
