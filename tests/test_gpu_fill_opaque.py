"""Fills whose colour replaces what it is drawn on: pixels of full coverage are
written without being read, partly covered ones blended as before, at every
alignment of a row, byte for byte against the oracle."""
import numpy as np
import pytest

import pixie_gb300 as px
from oracle import pxo
from pixie_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,alpha", [(17, 1.0), (17, 0.4), (17, 0.0), (0, 1.0), (0, 0.998), (0, 0.5)])
@pytest.mark.parametrize("w,h", [(1, 5), (3, 9), (4, 4), (5, 33), (67, 40), (130, 31), (1029, 17), (2050, 9)])
def test_replacing_fills(w, h, mode, alpha):
    px.lib().pxg_init(0)
    pxo.set_golden_mode(False)
    color = [0.9, 0.3, 0.6, alpha]
    rect = [1, 0, 0, 2, w, 0, 2, w, h, 2, 0, h, 0]
    inner = [1, 1, 1, 2, w - 2, 1, 2, w - 2, h - 1, 2, 1, h - 1, 0]
    slanted = [1, 0.3, 0.2, 2, w * 0.9, 0.1 * h, 2, w - 0.4, h * 0.8, 2, w * 0.1, h - 0.3, 0]
    back = wl.premultiplied_image(w * 7 + h, w, h)
    for cmds in (rect, inner, slanted, list(wl.plain_path(3, n_cubics=5, size=float(min(w, h))))):
        cmds = np.asarray(cmds, np.float32)
        ref = back.copy()
        pxo.fill_path(ref, cmds, color, 1.0, mode, None, 0)
        img = px.Image.from_numpy(back)
        img.fill_path(cmds, px.Paint(color=color, blend_mode=px.BlendMode(mode)))
        assert np.array_equal(img.to_numpy(), ref)
