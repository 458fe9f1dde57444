"""Paths of about 64 primitives, from which on launches of few rows take a CTA per
row, and of as many rows as still do: the oracle's bytes on both sides."""
import numpy as np
import pytest

import pixie_gb300 as px
from oracle import pxo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edges", (62, 63, 64, 65, 200))
@pytest.mark.parametrize("w,h", [(34, 5), (257, 40), (1400, 33), (60, 5000)])
def test_edges(edges, w, h):
    px.lib().pxg_init(0)
    pxo.set_golden_mode(False)
    rs = np.random.RandomState(edges + w)
    x, y = rs.rand(edges) * w * 1.1 - 0.05 * w, rs.rand(edges) * h * 1.1 - 0.05 * h
    cmds = [1.0, x[0], y[0]]
    for k in range(1, edges):
        cmds += [2.0, x[k], y[k]]
    cmds = np.asarray(cmds + [0.0], np.float32)
    for winding in (0, 1):
        ref = pxo.new_image(w, h)
        pxo.fill_path(ref, cmds, [0.3, 0.8, 0.1, 0.7], 1.0, 0, None, winding)
        img = px.Image(w, h)
        img.fill_path(cmds, px.Paint(color=[0.3, 0.8, 0.1, 0.7]), None, winding)
        assert np.array_equal(img.to_numpy(), ref)
