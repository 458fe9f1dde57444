"""Batches of masks of one size whose outlines are light and heavy, in turn: the
row kernel's configuration is chosen for each kind, the bytes are the oracle's."""
import numpy as np
import pytest

import pixie_gb300 as px
from oracle import pxo
from pixie_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


def test_light_and_heavy_outlines():
    px.lib().pxg_init(0)
    pxo.set_golden_mode(False)
    w, h, count = 190, 150, 5
    for rounds in range(2):
        for cubics in (3, 64):  # counting 72 and 1536 lines
            m = px.Masks()
            paths = []
            for k in range(count):
                cmds = wl.plain_path(10 * cubics + k, n_cubics=cubics, size=150.0)
                paths.append(cmds)
                m.add_path(cmds, w, h)
            for _ in range(3):
                m.render()
                for k, cmds in enumerate(paths):
                    ref = pxo.new_image(w, h)
                    pxo.fill_path(ref, cmds, [1, 1, 1, 1], 1.0, 0, None, 0)
                    assert np.array_equal(m.mask(k), ref[..., 3])
    classes = [ln for ln in px.autotune_report().splitlines() if "side<=256,count<=8" in ln]
    assert any("heavy" in ln for ln in classes) and any("heavy" not in ln for ln in classes)
