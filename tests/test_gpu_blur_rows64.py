"""The one-launch small-radius blur on images whose tiles have 64 rows, which is
an instance of its own: rows of whole 16-byte units and others, the last tile
short, each radius -- the oracle's bytes (integer sums: no tolerance)."""
import numpy as np
import pytest

import pixie_gb300 as px
from oracle import pxo
from pixie_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r", (3, 5, 6))
@pytest.mark.parametrize("w,h", [(5000, 700), (3733, 1285)])
def test_rows_64(w, h, r):
    px.lib().pxg_init(0)
    img = wl.premultiplied_image(w + r, w, h)
    oob = (0.2, 0.5, 0.9, 0.6)
    ref = img.copy()
    pxo.blur(ref, r, pxo.color_to_rgbx(oob))
    g = px.Image.from_numpy(img)
    g.blur(r, oob)
    assert px.last_blur_kernel() == 5
    assert np.array_equal(g.to_numpy(), ref)
