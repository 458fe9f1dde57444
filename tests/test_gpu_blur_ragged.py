"""The tensor-core ring passes on images whose rows are not whole 16-byte
units: every pair of side residues mod 4, sides around a band (32 lines) and a
tile (64 positions), segments that end mid-tile, every radius residue, split
and exact weights, colours outside -- bytes equal to the oracle's (integer
sums: no tolerance)."""
import numpy as np
import pytest

import pixie_gb300 as px
from oracle import pxo
from pixie_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _init():
    px.lib().pxg_init(0)
    pxo.set_golden_mode(False)
    px.blur_config(3)
    yield


CASES = [(4 + i, 4 + j, 9 + i + 4 * j) for i in range(4) for j in range(4)]
CASES += [(w, h, r) for (w, h) in [(31, 65), (33, 63), (65, 33), (129, 31), (1237, 101), (101, 1237), (5, 300),
                                   (300, 5), (255, 258), (2051, 67), (64, 65), (65, 64)] for r in (9, 18, 64, 127)]


@pytest.mark.parametrize("w,h,r", CASES)
def test_ragged_blur(w, h, r):
    img = wl.premultiplied_image(w * 7 + h * 3 + r, w, h)
    oob = (0.2, 0.5, 0.9, 0.6) if (w + h + r) % 2 else (0, 0, 0, 0)
    ref = img.copy()
    pxo.blur(ref, r, pxo.color_to_rgbx(oob))
    g = px.Image.from_numpy(img)
    g.blur(r, oob)
    assert np.array_equal(g.to_numpy(), ref)


# radii 6..8 on either side of the sizes from which the ring takes them
@pytest.mark.parametrize("w,h,r", [(2196, 2204, 6), (2200, 2200, 6), (1905, 1904, 8), (2048, 2024, 7), (2049, 2350, 8),
                                   (2333, 2333, 7), (2331, 2327, 7), (2501, 2504, 6)])
def test_small_radius_of_large_images(w, h, r):
    img = wl.premultiplied_image(w + h + r, w, h)
    ref = img.copy()
    pxo.blur(ref, r, pxo.color_to_rgbx((0.9, 0.1, 0.3, 0.5)))
    for exported in (False, True):
        g = px.Image.from_numpy(img)
        if exported:
            assert g.device_ptr
        g.blur(r, (0.9, 0.1, 0.3, 0.5))
        assert np.array_equal(g.to_numpy(), ref)
