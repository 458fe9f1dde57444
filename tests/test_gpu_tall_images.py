"""Paths with few of a tall image's rows: the row kernel's items are shared out
over the path's rows, whatever their number, byte for byte against the oracle."""
import numpy as np
import pytest

import pixie_gb300 as px
from oracle import pxo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [6100, 12200, 20000])  # one, two and four rows per item by the image's rows
@pytest.mark.parametrize("rows", [0.5, 1, 2, 5, 0.5003, 64, 3001, -1])  # -1: all of them
@pytest.mark.parametrize("at", [0.0, 0.25, 4096.75])
def test_rows_of_the_path(h, rows, at):
    px.lib().pxg_init(0)
    pxo.set_golden_mode(False)
    w = 21
    top, end = (at, at + rows) if rows > 0 else (-3.0, h + 5.0)
    cmds = np.asarray([1, 2.25, top, 2, 18.5, top + (end - top) * 0.125, 2, 11.75, end, 2, 9.5, top + (end - top) * 0.5,
                       0], np.float32)
    ref = pxo.new_image(w, h)
    pxo.fill_path(ref, cmds, [0.1, 0.7, 0.4, 0.8], 1.0, 0, None, 0)
    img = px.Image(w, h)
    img.fill_path(cmds, px.Paint(color=(0.1, 0.7, 0.4, 0.8)))
    assert np.array_equal(img.to_numpy(), ref)
