"""The run-length coder at the edges of its pieces (127 equal, 128 literal bytes), of the 32 bytes a warp takes at a
time and of the row, against the oracle's stbi_write_hdr."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _row(width, lengths, rng):
    """Stretches of the given lengths: equal bytes, then bytes that all differ from their neighbours, in turn."""
    out, k = [], 0
    while sum(map(len, out)) < width:
        n = lengths[k % len(lengths)]
        out.append(np.full(n, 0.25 + 0.5 * (k % 2)) if k % 2 == 0 else 0.5 + 0.003 * ((np.arange(n) * 37) % 128))
        k += 1
    return np.concatenate(out)[:width]


@pytest.mark.parametrize("width", [8, 31, 32, 33, 64, 383, 384, 1000])
@pytest.mark.parametrize("lengths", [(3, 1), (2, 2), (126, 127), (127, 128), (128, 129), (255, 257), (29, 3), (400, 5)])
def test_stretches(ctx, oracle, width, lengths):
    rng = np.random.default_rng(width)
    img = np.zeros((5, width, 3), np.float32)
    for y in range(4):
        for c in range(3):
            img[y, :, c] = np.roll(_row(width, lengths, rng), 7 * y + 11 * c)
    img[4] = rng.choice(np.array([0.25, 0.5, 0.75], np.float32), (width, 3))
    flat = img.reshape(-1, 3)
    assert ctx.encode_hdr(flat[::-1].copy(), width, 5) == oracle.hdr_file(img, width, 5)


def test_images_in_turn(ctx, oracle):
    """A smaller image after a larger one: nothing of the first stays in the second's file."""
    rng = np.random.default_rng(3)
    for h, w in ((40, 300), (3, 20), (17, 130)):
        img = rng.gamma(0.5, 2.0, (h, w, 3)).astype(np.float32)
        assert ctx.encode_hdr(img.reshape(-1, 3)[::-1].copy(), w, h) == oracle.hdr_file(img, w, h)


@pytest.mark.parametrize("width", [7, 8, 32767, 32768])
def test_widths_around_the_coded_ones(ctx, oracle, width):
    """Rows of 8 to 32,767 pixels are run-length coded, the widest from 131,068 bytes of shared memory; others are not."""
    rng = np.random.default_rng(width)
    img = rng.choice(np.array([0.25, 0.5, 0.75], np.float32), (2, width, 3))
    img[1, : width // 2] = rng.random((width // 2, 3))
    assert ctx.encode_hdr(img.reshape(-1, 3)[::-1].copy(), width, 2) == oracle.hdr_file(img, width, 2)
