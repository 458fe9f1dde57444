"""The one-launch small-radius blur at every number of rows a tile may have:
heights around one and several tiles, widths around a tile and not a multiple
of 4, each radius -- bytes equal to the oracle's (integer sums: no
tolerance)."""
import numpy as np
import pytest

import pixie_gb300 as px
from oracle import pxo
from pixie_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r", range(1, 9))
@pytest.mark.parametrize("w,h", [(1, 1), (127, 7), (129, 9), (640, 640), (641, 643), (1001, 999), (1237, 1001),
                                 (1920, 1080), (2000, 1711), (64, 1300)])
def test_tile_rows(w, h, r):
    px.lib().pxg_init(0)
    img = wl.premultiplied_image(w + h + r, w, h)
    oob = (0.2, 0.5, 0.9, 0.6)
    ref = img.copy()
    pxo.blur(ref, r, pxo.color_to_rgbx(oob))
    g = px.Image.from_numpy(img)
    g.blur(r, oob)
    assert px.last_blur_kernel() == 5
    assert np.array_equal(g.to_numpy(), ref)
